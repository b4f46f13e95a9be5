// ss_stage.h -- large copies between pageable host memory and the device.
//
// A pageable cudaMemcpyAsync goes through the driver's own staging buffer on
// one host thread (about 9 GB/s up; down into freshly mapped pages about 4
// GB/s, since that thread also takes the page faults).  These copies cut the
// range over several host threads, each moving 1 MiB pieces through two
// page-locked buffers of its own, so the host side runs at memory speed and the
// link stays busy.  Small copies take the plain call.
//
// The pieces' buffers come from the library's pool of page-locked blocks
// (host_block_take: bounded, shared by all threads, handed back on return);
// nothing else outlives the call.  Down returns when the host range is filled,
// up when it is free to reuse, unless it is page-locked and small enough for the
// plain call (then, as with that call, when the stream has got there); the
// device side is ordered on the stream.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace ssb {

cudaError_t stage_upload(void *dst, const void *src, size_t bytes, cudaStream_t s);
cudaError_t stage_download(void *dst, const void *src, size_t bytes, cudaStream_t s);

}  // namespace ssb
