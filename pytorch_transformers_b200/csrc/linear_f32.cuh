// The two forms of the float32 linear layer (linear_f32.cu: CUDA cores, linear_f32_tc.cu: tensor cores).
#pragma once
#include <cuda_runtime.h>

// arguments as ptb_linear_f32 takes them; rows of w at whole 16-byte words
int linear_f32_tensor(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, int ldx, int act,
                      int* error_flag, cudaStream_t stream);
