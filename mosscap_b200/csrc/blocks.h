// Device memory blocks kept from one adjoint to the next.
//
// A differentiable run creates and destroys an mc_adjoint for every forward /
// backward pass, and cudaMalloc / cudaFree of its states, checkpoints and segment
// took 6 of the 20 ms of a 20-step pass on 512^2. Freed blocks are kept here, at most
// kKeptBytes over the process, and handed out again for the same size on the same
// device.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace mc {

constexpr size_t kKeptBytes = size_t(512) << 20;

// cudaMalloc on the current device, or a kept block of that size. When the
// device has no room, the kept blocks are given back first.
cudaError_t block_alloc(void** p, size_t bytes);
// Take a block back (null: nothing). No work that uses it may be pending: the
// caller has synchronised its device. Past kKeptBytes the oldest blocks go back to the
// device.
void block_free(void* p, size_t bytes, int device);
// Give every kept block back to its device.
void blocks_release();
// cudaMalloc; when the device has no room, once more after blocks_release.
cudaError_t device_alloc(void** p, size_t bytes);

} // namespace mc
