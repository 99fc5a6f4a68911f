// sp_stage.h -- copies between the caller's host memory and the device.
//
// Same meaning as cudaMemcpyAsync from or to pageable memory: sp_copy_in returns
// when the source has been read (the device copy may still run on the stream),
// sp_copy_out when the destination holds the data.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <functional>

// `enqueued`, when given, is called with the number of bytes whose copies are on
// the stream, each time it grows and at last with `bytes`.
cudaError_t sp_copy_in(void *dev, const void *host, size_t bytes, cudaStream_t s,
                       const std::function<cudaError_t(size_t)> &enqueued = nullptr);
cudaError_t sp_copy_out(void *host, const void *dev, size_t bytes, cudaStream_t s);

// A little host memory that the device can write, from a pool of the process; null
// when none is left or `bytes` is more than a slot's. Give it back when nothing on
// the device can still write it.
void *sp_mail_take(size_t bytes);
void sp_mail_give(void *slot);
