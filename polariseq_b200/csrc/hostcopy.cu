// Copies between pageable host arrays and the device.
//
// NumPy arrays are pageable, and a copy of pageable memory goes through the
// driver's own staging on the calling thread (3-8 GB/s here, with the page
// faults of a fresh result array in the same thread: 24 searched samples
// returned 600 MB in 250 ms while their kernels took 28).  Copies of STAGE_MIN
// bytes or more go through the context's pinned ring instead: a few threads
// move slices between the array and the ring (and take its page faults side by
// side) while the copy engine works on the other buffers.  Pinned arrays and
// small copies take cudaMemcpyAsync as they are.  Measured on whole calls from
// NumPy arrays (16 host cores): the 24 samples 306 -> 72 ms, connectivities of a
// million cells 100 -> 22.6 ms, the E4M3 build of 600,011 x 40 107 -> 82 ms.
//
// The ring (RING x CHUNK bytes) and its events belong to the context, are made
// on first use and freed with it; the threads live for one copy.
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

#include "ctx.cuh"
#include "hostcopy.cuh"

namespace pq {

constexpr size_t CHUNK = size_t(4) << 20;
constexpr int RING = 6;
constexpr size_t STAGE_MIN = size_t(8) << 20;
constexpr unsigned MAX_THREADS = 8;

struct HostStage {
    uint8_t* buf[RING] = {};
    cudaEvent_t ev[RING] = {};  // the last device copy of each buffer
};

void host_stage_free(HostStage* s) {
    if (!s) return;
    for (int i = 0; i < RING; ++i) {
        if (s->ev[i]) {
            cudaEventSynchronize(s->ev[i]);
            cudaEventDestroy(s->ev[i]);
        }
        if (s->buf[i]) cudaFreeHost(s->buf[i]);
    }
    delete s;
}

namespace {

// The context's ring with no copy in flight; null when it cannot be had.
HostStage* stage_of(pq_ctx* c) {
    if (!c->stage) {
        HostStage* s = new HostStage();
        for (int i = 0; i < RING; ++i)
            if (cudaMallocHost(reinterpret_cast<void**>(&s->buf[i]), CHUNK) != cudaSuccess ||
                cudaEventCreateWithFlags(&s->ev[i], cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                host_stage_free(s);
                return nullptr;
            }
        c->stage = s;
    }
    for (int i = 0; i < RING; ++i) cudaEventSynchronize(c->stage->ev[i]);
    return c->stage;
}

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

template <class F>
void until(F&& done) {
    for (int i = 0; !done(); ++i)
        if (i > 64) std::this_thread::yield();
}

// Runs `work(thread, threads)` on a few threads beside `lead()` on this one;
// `lead` gets the number of threads (at least one) first.  False when no thread
// could be started (nothing has run).
template <class W, class L>
bool with_threads(W&& work, L&& lead) {
    const unsigned hw = std::thread::hardware_concurrency();
    const unsigned want = std::max(1u, std::min(MAX_THREADS, hw / 2));
    std::atomic<int> go{0};  // the thread count, once they are all started
    std::vector<std::thread> ts;
    try {
        ts.reserve(want);
        for (unsigned t = 0; t < want; ++t)
            ts.emplace_back([&, t] {
                until([&] { return go.load(std::memory_order_acquire) != 0; });
                const int n = go.load(std::memory_order_acquire);
                if (n > 0) work(int(t), n);
            });
    } catch (const std::exception&) {
    }
    const int n = int(ts.size());
    if (n > 0) {
        go.store(n, std::memory_order_release);
        lead(n);
    }
    for (std::thread& t : ts) t.join();
    return n > 0;
}

// Slice t of T of chunk i: [lo, hi) within the chunk, whole pages.
void slice(size_t len, int t, int T, size_t& lo, size_t& hi) {
    const size_t per = ((len + size_t(T) - 1) / size_t(T) + 4095) & ~size_t(4095);
    lo = std::min(len, per * size_t(t));
    hi = std::min(len, lo + per);
}

}  // namespace

void copy_to_device(pq_ctx* c, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    HostStage* s = bytes >= STAGE_MIN && pageable(src) ? stage_of(c) : nullptr;
    cudaError_t err = cudaSuccess;
    if (s) {
        const int n = int((bytes + CHUNK - 1) / CHUNK);
        std::vector<std::atomic<int>> done(n);
        for (auto& d : done) d.store(0);
        std::atomic<int> avail{0};  // chunks whose buffer is free; -1: stop
        const bool ran = with_threads(
            [&](int t, int T) {
                for (int i = 0; i < n; ++i) {
                    until([&] { return avail.load(std::memory_order_acquire) > i ||
                                       avail.load(std::memory_order_acquire) < 0; });
                    if (avail.load(std::memory_order_acquire) < 0) return;
                    const size_t off = size_t(i) * CHUNK;
                    size_t lo, hi;
                    slice(std::min(CHUNK, bytes - off), t, T, lo, hi);
                    std::memcpy(s->buf[i % RING] + lo, static_cast<const uint8_t*>(src) + off + lo,
                                hi - lo);
                    done[i].fetch_add(1, std::memory_order_acq_rel);
                }
            },
            [&](int T) {
                for (int i = 0; i < n && err == cudaSuccess; ++i) {
                    // three chunks ahead; their buffers' last copies are RING - 3 behind
                    const int a = std::min(n, i + 3);
                    for (int x = avail.load(std::memory_order_relaxed); x < a; ++x) {
                        if (x >= RING) cudaEventSynchronize(s->ev[x % RING]);
                        avail.store(x + 1, std::memory_order_release);
                    }
                    until([&] { return done[i].load(std::memory_order_acquire) == T; });
                    const size_t off = size_t(i) * CHUNK;
                    err = cudaMemcpyAsync(static_cast<uint8_t*>(dst) + off, s->buf[i % RING],
                                          std::min(CHUNK, bytes - off), cudaMemcpyHostToDevice, st);
                    if (err == cudaSuccess) err = cudaEventRecord(s->ev[i % RING], st);
                }
                if (err != cudaSuccess) avail.store(-1, std::memory_order_release);
            });
        if (ran) {
            pqh::ck(err, "h2d");
            return;
        }
    }
    pqh::ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st), "h2d");
}

void copy_to_host(pq_ctx* c, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    HostStage* s = bytes >= STAGE_MIN && pageable(dst) ? stage_of(c) : nullptr;
    cudaError_t err = cudaSuccess;
    if (s) {
        const int n = int((bytes + CHUNK - 1) / CHUNK);
        std::vector<std::atomic<int>> done(n);
        for (auto& d : done) d.store(0);
        std::atomic<int> arrived{0};  // chunks in their buffer; -1: stop
        const bool ran = with_threads(
            [&](int t, int T) {
                for (int i = 0; i < n; ++i) {
                    until([&] { return arrived.load(std::memory_order_acquire) > i ||
                                       arrived.load(std::memory_order_acquire) < 0; });
                    if (arrived.load(std::memory_order_acquire) < 0) return;
                    const size_t off = size_t(i) * CHUNK;
                    size_t lo, hi;
                    slice(std::min(CHUNK, bytes - off), t, T, lo, hi);
                    std::memcpy(static_cast<uint8_t*>(dst) + off + lo, s->buf[i % RING] + lo,
                                hi - lo);
                    done[i].fetch_add(1, std::memory_order_acq_rel);
                }
            },
            [&](int T) {
                auto issue = [&](int i) {
                    if (i >= RING)  // the buffer's last chunk has been taken
                        until([&] { return done[i - RING].load(std::memory_order_acquire) == T; });
                    const size_t off = size_t(i) * CHUNK;
                    err = cudaMemcpyAsync(s->buf[i % RING], static_cast<const uint8_t*>(src) + off,
                                          std::min(CHUNK, bytes - off), cudaMemcpyDeviceToHost, st);
                    if (err == cudaSuccess) err = cudaEventRecord(s->ev[i % RING], st);
                };
                int sent = 0;
                for (; sent < std::min(n, 3) && err == cudaSuccess; ++sent) issue(sent);
                for (int i = 0; i < n && err == cudaSuccess; ++i) {
                    err = cudaEventSynchronize(s->ev[i % RING]);
                    if (err != cudaSuccess) break;
                    arrived.store(i + 1, std::memory_order_release);
                    if (sent < n) {
                        issue(sent);
                        ++sent;
                    }
                }
                if (err != cudaSuccess) arrived.store(-1, std::memory_order_release);
            });
        if (ran) {
            pqh::ck(err, "d2h");
            return;
        }
    }
    pqh::ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st), "d2h");
    pqh::ck(cudaStreamSynchronize(st), "d2h");
}

}  // namespace pq
