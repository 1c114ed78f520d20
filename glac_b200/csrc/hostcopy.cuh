// Copies between pageable host memory and the device by several host threads.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace glac {

// Both order themselves after the work already on `st`.  copy_to_host returns
// when `host` may be read; after copy_to_device `host` may be changed once `st`
// has been synchronised.
cudaError_t copy_to_device(void *dev, const void *host, size_t bytes, int device, cudaStream_t st);
cudaError_t copy_to_host(void *host, const void *dev, size_t bytes, int device, cudaStream_t st);

// The pinned staging memory (16 MB a process, once copies pay for it) lives while at least one holder does.
void hostcopy_hold();
void hostcopy_drop();

}  // namespace glac
