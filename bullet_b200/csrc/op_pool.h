// The memory pool behind b200_op_ft_forward's scratch (op_ft_forward.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace b200 {
int op_pool_alloc(int device, cudaStream_t stream, size_t bytes, int** out);  // 0, or a B200_ERR_* with the message set
void op_pool_trim(int device);  // gives back what the pool keeps between calls
}  // namespace b200
