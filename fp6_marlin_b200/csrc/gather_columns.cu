// Columns of a row-major fp16 matrix in another order, with an optional bias: y[m, f] = c[m, src[f]] + bias[f].
// W46Linear puts the output features back into the model's order with it (the reference leaves that to its caller;
// an attempt inside its binding is commented out, fp6_marlin_cuda.cpp:93-122).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fp6m.h"

namespace {

constexpr int kThreads = 128, kRows = 4;

// Thread = eight neighbouring output columns of four rows: indices and bias are loaded once for the rows, the features of
// one region keep their order, so a warp's two-byte reads fall into few lines, and the result leaves as 16-byte stores.
// Latency-bound at the sizes of a decode step or a short prompt (3 x 67 rows of 4096 features: 3.3 MB): one launch, started
// while the kernel in front of it finishes, in place of an index_select and an addition: that W46Linear call with a bias
// takes 49 us with the GEMM (two launches) at 44, and took 60 with the two torch operations and the GEMM at 46.
__global__ void __launch_bounds__(kThreads) gather_columns_kernel(const half* __restrict__ c, half* __restrict__ y, const long long* __restrict__ src,
                                                                  const half* __restrict__ bias, int M, int N) {
  const int col = (blockIdx.x * kThreads + threadIdx.x) * 8;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (col >= N) return;
  long long at[8];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const longlong2 two = *reinterpret_cast<const longlong2*>(src + col + i);
    at[i] = two.x;
    at[i + 1] = two.y;
  }
  uint4 b = make_uint4(0, 0, 0, 0);
  if (bias) b = *reinterpret_cast<const uint4*>(bias + col);
  const half* add = reinterpret_cast<const half*>(&b);
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const int row = blockIdx.y * kRows + r;
    if (row >= M) return;
    uint4 out;
    half* v = reinterpret_cast<half*>(&out);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // an index outside the matrix (a damaged buffer) reads nothing and shows as NaN
      v[i] = (unsigned long long)at[i] < (unsigned long long)N ? c[(size_t)row * N + at[i]] : __ushort_as_half(0x7FFF);
      if (bias) v[i] = __hadd(v[i], add[i]);
    }
    *reinterpret_cast<uint4*>(y + (size_t)row * N + col) = out;
  }
}

}  // namespace

extern "C" int fp6m_gather_columns(const void* c, void* y, const void* src, const void* bias, int M, int N, int dev, void* stream) {
  if (M < 0 || N < 0 || N % 8) return FP6M_ERR_BAD_ARG;
  if (M == 0 || N == 0) return FP6M_OK;
  if (!c || !y || !src) return FP6M_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(c) & 1) || ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(bias)) & 15))
    return FP6M_ERR_BAD_ARG;
  int before = -1;
  if (cudaGetDevice(&before) != cudaSuccess) return FP6M_ERR_CUDA;
  if (before != dev && cudaSetDevice(dev) != cudaSuccess) return FP6M_ERR_CUDA;
  cudaError_t e = cudaSuccess;
  constexpr int kMaxRows = 65535 * kRows;               // of one launch
  for (int m0 = 0; m0 < M && e == cudaSuccess; m0 += kMaxRows) {
    const int rows = M - m0 < kMaxRows ? M - m0 : kMaxRows;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((N / 8 + kThreads - 1) / kThreads, (rows + kRows - 1) / kRows);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, gather_columns_kernel, static_cast<const half*>(c) + (size_t)m0 * N, static_cast<half*>(y) + (size_t)m0 * N,
                           static_cast<const long long*>(src), static_cast<const half*>(bias), rows, N);
    if (M - m0 <= kMaxRows) break;                      // (m0 + kMaxRows could pass INT_MAX)
  }
  if (before != dev) cudaSetDevice(before);
  return e == cudaSuccess ? FP6M_OK : FP6M_ERR_CUDA;
}
