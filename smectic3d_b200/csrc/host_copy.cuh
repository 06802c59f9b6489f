// Copies between pageable host arrays and the device.
//
// cudaMemcpyAsync moves a pageable array through one staging buffer with one host
// thread, 8 GB/s here; the two copies of a 128^3 run took longer than its steps.
// Large copies are cut into chunks that a few threads move through pinned buffers of
// their own while the copy engine works on the chunks before.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace shb {

// Same contract as cudaMemcpyAsync on a pageable array followed, for device to
// host, by a synchronisation of ``stream``: on return the host array has been read
// (or written) completely.  Small copies and pinned arrays take cudaMemcpyAsync.
cudaError_t copy_to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream);
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream);

// Every handle holds the pinned buffers (6 MB, one set per process) while it lives;
// host_copy.cu says when they are made and given back.
void host_copy_retain();
void host_copy_release();

}  // namespace shb
