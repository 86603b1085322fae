// prim.cuh -- device-wide primitives of libsexgpu (see prim.cu).
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace sx {
size_t scan_temp_ints(long long n);
int exclusive_scan(const int *in, int *out, long long n, int *total, int *tmp, cudaStream_t st,
                   const int *n_dev = nullptr);
int exclusive_scan2(const int *in0, int *out0, int *total0, const int *in1, int *out1, int *total1, long long n,
                    int *tmp, cudaStream_t st);
}  // namespace sx
