// Copies between pageable host arrays and the device (hostcopy.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

struct pq_ctx;

namespace pq {

struct HostStage;  // a context's pinned staging buffers

// Copies `bytes` on stream st.  On return the host array has been read
// (to_device: the device copy is ordered on st) or written (to_host: everything
// queued on st before has finished).  Throws pqh::DeviceError.
void copy_to_device(pq_ctx* c, void* dst, const void* src, size_t bytes, cudaStream_t st);
void copy_to_host(pq_ctx* c, void* dst, const void* src, size_t bytes, cudaStream_t st);
void host_stage_free(HostStage* s);

}  // namespace pq
