// GPU half of the C ABI (include/fp6m.h): argument validation that mirrors the reference's host
// dispatcher, the stripe schedule, and the kernel launches.  No allocation, no synchronisation.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>

#include "../../include/fp6m.h"
#include "fp6m_layout.h"
#include "gemm_params.h"

namespace {

using namespace fp6m;

thread_local char g_cuda_error[256] = "";

int cuda_fail(cudaError_t e, const char* where) {
  std::snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s", where, cudaGetErrorString(e));
  return FP6M_ERR_CUDA;
}

int sm_count(int dev) {
  static std::atomic<int> cached[64] = {};
  if (dev < 0 || dev >= 64) return 0;
  int n = cached[dev];
  if (!n) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cached[dev] = n;
  }
  return n;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) switched = cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceGuard() { if (switched) cudaSetDevice(prev); }
};

// How a GEMM of M rows is cut into launches: kernel, tile of rows, rows per launch, grid.
struct LaunchPlan {
  bool wide;        // the kernel with scaled operands and tiles of 256 rows
  int tile;         // (most) rows of A per MMA tile
  int rows;         // rows of A per launch
  int ctas;         // grid of the first (largest) launch
  int row_ctas;     // CTAs that the device offers (for the number of row tiles)
};

// `sms` <= 0: the largest grid any device can get (an upper bound for sizing buffers).
LaunchPlan plan_launches(int M, const Geometry& geo, int sms, int two_launches = -1, bool fewest_tiles = false) {
  LaunchPlan lp;
  // 129 to 256 rows on a layer with INT4 group scales and up to 48 blocks per CTA: two launches of the kernels for up to 128 rows.
  // It multiplies the fp32 sums by the group scales; the other kernel rounds every scaled weight to fp16 first, which costs
  // bits (INT4 columns against 64-bit sums, K = 1024 to 11008: relative error 2.07e-4 here, 2.67e-4 there; with the rounding
  // of the result alone 2.07e-4).  One launch of the other kernel is faster and is the plan of layers without group scales, on
  // which the errors of both kernels agree to five digits (us at 129 / 201 / 256 rows, two launches -> one: 4096 x 4096
  // 33 / 44 / 44 -> 24 / 27 / 27, 4096 x 12288 41 / 52 / 52 -> 31 / 36 / 39, K = N = 8192 47 / 59 / 59 -> 39 / 45 / 49, 11008 x 4096
  // 43 / 56 / 56 -> 40 / 42 / 43, 1024 x 4096 26 / 35 / 36 -> 17, 4096 x 22016 56 / 69 / 74 -> 43 / 49 / 54), and of larger layers,
  // where two launches take longer even than one with 256-row tiles (K = N = 16384, 111 blocks per CTA, 4 %).
  // `two_launches`: -1 decides here, 0 / 1 force (sizing a buffer for either).
  bool two = false;
  if (M > kTc5MaxRows && M <= 2 * kTc5MaxRows) {
    const long long blocks = (long long)(geo.strips4 + geo.strips6) * geo.k128;
    const bool group_scales = geo.groups > 1 && geo.strips4 > 0;
    two = two_launches < 0 ? group_scales && blocks <= 48ll * (sms > 0 ? sms : 148) : two_launches != 0;
  }
  lp.wide = M > kTc5MaxRows && !two;
  lp.tile = lp.wide ? kWideTileRows : tc5_tile_rows(M < kTc5MaxRows ? M : kTc5MaxRows);
  // CTAs own contiguous ranges of (tile, strip) pairs, so the tiles of a launch are all in flight at once:
  // keep their activations (tile x K halves each) within half of L2
  // (measured at K = 16384: 64 MB of activations per launch are as fast as 32 MB on a full layer and 23 % faster
  // on a shard of 2048 columns, whose 16 strips need eight row tiles to give every CTA a strip; 96 MB are slower)
  int max_tiles = (int)((64ll << 20) / ((long long)lp.tile * geo.K * 2));
  if (max_tiles < 1) max_tiles = 1;
  if (max_tiles > kMaxRowTiles) max_tiles = kMaxRowTiles;
  lp.rows = lp.wide ? lp.tile * max_tiles : lp.tile;
  const int launch_rows = M < lp.rows ? M : lp.rows;
  const int cap = lp.wide ? kMaxWideCtas : kMaxCtas;
  long long want = sms > 0 ? (long long)sms * (lp.wide ? 1 : tc5_ctas_per_sm(launch_rows)) : cap;
  int ctas = want < cap ? (int)want : cap;
  lp.row_ctas = fewest_tiles ? 0 : ctas;            // 0: no tile beyond those that hold the rows
  const int row_tiles = lp.wide ? wide_row_tiles(launch_rows, geo, lp.row_ctas) : 1;     // (more with a larger grid: without a device an upper bound)
  // at least ~16 units per CTA, also when that leaves SMs idle: a small GEMM split over every SM spends
  // its time in the split-K reduction (16 contributors per strip for N = 1024), not in streaming
  const long long total_units = (long long)row_tiles * (geo.strips4 + geo.strips6) * units_per_strip(geo);
#ifndef FP6M_MIN_UNITS_PER_CTA
#define FP6M_MIN_UNITS_PER_CTA 16
#endif
  long long by_work = total_units / FP6M_MIN_UNITS_PER_CTA;
  if (by_work < 1) by_work = 1;
  if (ctas > by_work) ctas = (int)by_work;
  if (ctas < 1) ctas = 1;
  lp.ctas = ctas;
  return lp;
}

size_t scratch_bytes_of(const LaunchPlan& lp) {
  const size_t b = lp.wide ? wide_scratch_bytes(lp.ctas) : tc5_scratch_bytes(lp.ctas, lp.tile);
  return (b + 255) & ~(size_t)255;
}

}  // namespace

extern "C" {

size_t fp6m_mul_scratch_bytes(int M, int N, int K, int quant_cols, int sms) {
  if (M <= 0 || N <= 0 || K <= 0) {
    // no shape given: the bound over every configuration (the largest grid with the largest partial tile)
    size_t b = tc5_scratch_bytes(kMaxCtas, kTc5MaxRows);
    const size_t w = wide_scratch_bytes(kMaxWideCtas);
    if (w > b) b = w;
    return (b + 255) & ~(size_t)255;
  }
  const int qc = quant_cols < 0 ? 0 : (quant_cols > N ? N : quant_cols);
  const Geometry geo = make_geometry(K, N, qc, 128);
  if (M > kTc5MaxRows && M <= 2 * kTc5MaxRows) {
    // neither the group size is given here nor always a device: enough for either way of cutting 129 to 256 rows into launches
    const size_t a = scratch_bytes_of(plan_launches(M, geo, sms, 0)), b = scratch_bytes_of(plan_launches(M, geo, sms, 1));
    return a > b ? a : b;
  }
  return scratch_bytes_of(plan_launches(M, geo, sms));
}

int fp6m_mul_launches(int M, int N, int K, int quant_cols, int sms, int* many_rows_kernel) {
  if (many_rows_kernel) *many_rows_kernel = 0;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int qc = quant_cols < 0 ? 0 : (quant_cols > N ? N : quant_cols);
  const LaunchPlan lp = plan_launches(M, make_geometry(K, N, qc, 128), sms);
  if (many_rows_kernel) *many_rows_kernel = lp.wide ? 1 : 0;
  return (M + lp.rows - 1) / lp.rows;
}

}  // extern "C"

namespace {

int mul_impl(const void* A, const void* B, void* C, const void* s, int M, int N, int K,
             void* workspace, size_t workspace_bytes, void* scratch, size_t scratch_bytes,
             int dev, void* stream, int thread_k, int thread_n, int sms, int max_par,
             int quant_cols, int group_size, int layout, int* status_dev, const OutputMap& out,
             int epilogue = kEpilogueNone, const void* residual = nullptr) {
  // --- the checks of the reference dispatcher, in its order (fp6_marlin_cuda_kernel.cu:885-907)
  if (M < 0 || N < 0 || K < 0) return FP6M_ERR_BAD_ARG;
  if (thread_k == -1 || thread_n == -1) {
    if (M <= 16) { thread_k = 128; thread_n = 128; } else { thread_k = 64; thread_n = 256; }
  }
  if (thread_k <= 0 || thread_n <= 0) return FP6M_ERR_KERN_SHAPE;
  if (N % thread_n != 0 || K % thread_k != 0) return FP6M_ERR_PROB_SHAPE;
  if (M == 0 || N == 0 || K == 0) return FP6M_OK;
  // the reference has kernels for 128x128 tiles with at most 16 rows and for 64x256 tiles (:933-942)
  const bool shape_ok = (thread_k == 128 && thread_n == 128 && M <= 16) || (thread_k == 64 && thread_n == 256);
  if (!shape_ok) return FP6M_ERR_KERN_SHAPE;

  // --- checks of this implementation
  if (max_par < 1) max_par = 1;
  if (workspace_bytes < (size_t)(N / 128) * max_par * 4) return FP6M_ERR_WORKSPACE;  // fp6_marlin_cuda.cpp:62-63
  if (layout != FP6M_LAYOUT_B200) return FP6M_ERR_BAD_ARG;
  if (!(group_size == 128 || group_size <= 0)) return FP6M_ERR_BAD_ARG;
  const int qc = quant_cols < 0 ? 0 : quant_cols;
  if (qc > N || qc % 8 || (N - qc) % 8 || K % 8) return FP6M_ERR_PROB_SHAPE;
  if (group_size == 128 && K % 128) return FP6M_ERR_PROB_SHAPE;
  if (!A || !B || (!C && out.n_out == 0) || !s || !workspace || !scratch) return FP6M_ERR_BAD_ARG;
  if (!aligned16(A) || !aligned16(B) || !aligned16(C) || !aligned16(s) || !aligned16(scratch)) return FP6M_ERR_BAD_ARG;
  if (epilogue != kEpilogueNone && epilogue != kEpilogueSiluMul && epilogue != kEpilogueResidual) return FP6M_ERR_BAD_ARG;
  if (epilogue != kEpilogueNone && out.n_out != 0) return FP6M_ERR_BAD_ARG;       // not together with the scattered output
  if (epilogue == kEpilogueResidual && (!residual || (reinterpret_cast<uintptr_t>(residual) & 1))) return FP6M_ERR_BAD_ARG;

  DeviceGuard guard(dev);
  if (sms <= 0) sms = sm_count(dev);
  if (sms <= 0) return cuda_fail(cudaGetLastError(), "cudaDeviceGetAttribute");
  MulParams p;
  p.geo = make_geometry(K, N, qc, group_size);
  if ((long long)kMaxRowTiles * (p.geo.strips4 + p.geo.strips6) * units_per_strip(p.geo) > 0x3fffffff) return FP6M_ERR_PROB_SHAPE;
  // up to kTc5MaxRows rows (up to twice as many on some layers, in two launches): the kernel with fp32 group scaling;
  // more: the wide kernel, tiles of up to 256 rows, up to kMaxRowTiles tiles per launch
  LaunchPlan lp = plan_launches(M, p.geo, sms);
  // a caller's fixed scratch (fp6m_mul_static_scratch) may hold the partials of the fewest tiles only
  if (scratch_bytes < scratch_bytes_of(lp)) lp = plan_launches(M, p.geo, sms, -1, true);
  const bool wide = lp.wide;
  const int rows = lp.rows, ctas = lp.ctas;
  if (scratch_bytes < scratch_bytes_of(lp)) return FP6M_ERR_SCRATCH;
  p.B = static_cast<const uint8_t*>(B);
  p.S = static_cast<const half*>(s);
  p.N = N; p.K = K;
  p.epochs = static_cast<unsigned int*>(scratch);
  p.partials = reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(scratch) + kEpochWords * sizeof(unsigned int));
  p.status = status_dev;
  p.out = out;
  p.epilogue = epilogue;
  p.R = nullptr;
  {
    // 16-byte stores of finished rows need every row start and both column bases on 16-byte boundaries
    const int ld = out.n_out ? out.ld : N;
    const int base4 = out.n_out ? out.col4 : 0, base6 = out.n_out ? out.col6 : N - qc;
    bool ok = epilogue == kEpilogueNone && ld % 8 == 0 && base4 % 8 == 0 && base6 % 8 == 0;
    for (int q = 0; q < out.n_out; ++q) ok = ok && aligned16(out.peer[q]);
    p.vec_rows = ok ? 1 : 0;
  }
  p.weights_early = tc5_get_overlap() ? 1 : 0;
  const long long blocks = (long long)(p.geo.strips4 + p.geo.strips6) * p.geo.k128;

  for (int m0 = 0; m0 < M; m0 += rows) {
    p.A = static_cast<const half*>(A) + (size_t)m0 * K;
    // with the gate / up epilogue C has N / 2 columns
    p.C = C ? static_cast<half*>(C) + (size_t)m0 * (epilogue == kEpilogueSiluMul ? N / 2 : N) : nullptr;
    p.R = epilogue == kEpilogueResidual ? static_cast<const half*>(residual) + (size_t)m0 * N : nullptr;
    for (int q = 0; q < out.n_out; ++q) p.out.peer[q] = out.peer[q] + (size_t)m0 * out.ld;
    p.M = (M - m0) < rows ? (M - m0) : rows;
    // The last of several launches may be left with so few rows that a kernel for up to 128 rows is the faster one;
    // its partials fit (half as many rows, two slots per CTA).
    const bool launch_wide = wide && p.M > kTc5MaxRows;
    const int launch_ctas = wide && !launch_wide ? std::min(ctas, plan_launches(p.M, p.geo, sms).ctas) : ctas;
    p.row_tiles = launch_wide ? wide_row_tiles(p.M, p.geo, lp.row_ctas) : 1;
    p.tile_rows = launch_wide ? wide_tile_rows(p.M, p.row_tiles) : 0;
    make_schedule(p.geo, launch_ctas, &p.sched, p.row_tiles, !launch_wide && p.M <= kTeamMaxRows ? 0 : kReducerPenalty);
    align_schedule_to_blocks(&p.sched);
    // The kernels for 9 to 128 rows may also expand their first segments before the grid dependency resolves: above 32 rows always
    // (measured -2 to -3 % on a chain of launches), up to 32 rows with at most 20 blocks per CTA: us at 16 / 32 rows 4096 x 4096 (8 blocks) 7.73 /
    // 9.38 -> 6.97 / 8.57, 4096 x 1024 7.33 / 8.74 -> 6.88 / 8.14, 11008 x 4096 (19) 11.2 / 12.8 -> 11.1 / 12.6, but K = N = 8192 (28) 12.77 / 14.4
    // -> 12.70 / 14.3 and 8192 x 28672 (97) 32.5 / 35.3 -> 32.2 / 35.6: there the next launch's CTAs get their SMs too late for it.
    p.expand_early = (p.weights_early && !wide && (p.M > kTeamMaxRows || blocks <= 20ll * launch_ctas)) ? 1 : 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the lines between the kernels: measured at 5, 8, 16 and 32 rows, see the heads of gemm_few.cu and gemm_team.cu
    cudaError_t e = launch_wide ? launch_gemm_wide(p, st)
                    : p.M <= kFewMaxRows ? launch_gemm_few(p, st) : p.M <= kTeamMaxRows ? launch_gemm_team(p, st) : launch_gemm_tc5(p, st);
    if (e != cudaSuccess) return cuda_fail(e, launch_wide ? "w46_gemm_wide launch" : p.M <= kFewMaxRows ? "w46_gemm_few launch" : p.M <= kTeamMaxRows ? "w46_gemm_team launch" : "w46_gemm_tc5 launch");
  }
  return FP6M_OK;
}

}  // namespace

extern "C" {

int fp6m_mul(const void* A, const void* B, void* C, const void* s, int M, int N, int K,
             void* workspace, size_t workspace_bytes, void* scratch, size_t scratch_bytes,
             int dev, void* stream, int thread_k, int thread_n, int sms, int max_par,
             int quant_cols, int group_size, int layout, int* status_dev) {
  OutputMap out = {};
  return mul_impl(A, B, C, s, M, N, K, workspace, workspace_bytes, scratch, scratch_bytes, dev, stream, thread_k, thread_n,
                  sms, max_par, quant_cols, group_size, layout, status_dev, out);
}

int fp6m_mul_fused(const void* A, const void* B, void* C, const void* s, int M, int N, int K,
                   void* workspace, size_t workspace_bytes, void* scratch, size_t scratch_bytes,
                   int dev, void* stream, int thread_k, int thread_n, int sms, int max_par,
                   int quant_cols, int group_size, int layout, int* status_dev, int epilogue, const void* residual) {
  OutputMap out = {};
  return mul_impl(A, B, C, s, M, N, K, workspace, workspace_bytes, scratch, scratch_bytes, dev, stream, thread_k, thread_n,
                  sms, max_par, quant_cols, group_size, layout, status_dev, out, epilogue, residual);
}

int fp6m_mul_scatter(const void* A, const void* B, void* const* outputs, int n_outputs, int ld_out, int col4_base, int col6_base,
                     const void* s, int M, int N, int K, void* workspace, size_t workspace_bytes, void* scratch,
                     size_t scratch_bytes, int dev, void* stream, int thread_k, int thread_n, int sms, int max_par,
                     int quant_cols, int group_size, int layout, int* status_dev) {
  if (!outputs || n_outputs < 1 || n_outputs > 8 || ld_out < N || col4_base < 0 || col6_base < 0) return FP6M_ERR_BAD_ARG;
  {
    // both column ranges must lie inside a row of the outputs: the stores go to peer memory unchecked
    const int qc = quant_cols < 0 ? 0 : quant_cols;
    if (qc > N || (long long)col4_base + (N - qc) > ld_out || (long long)col6_base + qc > ld_out) return FP6M_ERR_BAD_ARG;
  }
  OutputMap out = {};
  out.n_out = n_outputs;
  out.ld = ld_out;
  out.col4 = col4_base;
  out.col6 = col6_base;
  for (int q = 0; q < n_outputs; ++q) {
    if (!outputs[q] || (reinterpret_cast<uintptr_t>(outputs[q]) & 1)) return FP6M_ERR_BAD_ARG;
    out.peer[q] = static_cast<half*>(outputs[q]);
  }
  return mul_impl(A, B, nullptr, s, M, N, K, workspace, workspace_bytes, scratch, scratch_bytes, dev, stream, thread_k,
                  thread_n, sms, max_par, quant_cols, group_size, layout, status_dev, out);
}

// Scratch of fp6m_mul_static_scratch.  In host code this name is only a handle: the device address
// comes from cudaGetSymbolAddress, once per device.
static __device__ __align__(256) unsigned char g_static_scratch[FP6M_STATIC_SCRATCH_BYTES];

int fp6m_mul_static_scratch(const void* A, const void* B, void* C, const void* s, int M, int N, int K,
                            void* workspace, size_t workspace_bytes, int dev, void* stream,
                            int thread_k, int thread_n, int sms, int max_par,
                            int quant_cols, int group_size, int layout, int* status_dev) {
  static std::atomic<void*> scratch_of_device[64] = {};
  if (dev < 0 || dev >= 64) return FP6M_ERR_BAD_ARG;
  if (!scratch_of_device[dev]) {
    DeviceGuard guard(dev);                 // the symbol has one instance per device: ask with `dev` current
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || !ptr) return cuda_fail(e, "cudaGetSymbolAddress(static scratch)");
    scratch_of_device[dev] = ptr;
  }
  // fp6m_mul checks the size it needs against what it is given and returns FP6M_ERR_SCRATCH if it is short
  return fp6m_mul(A, B, C, s, M, N, K, workspace, workspace_bytes, scratch_of_device[dev],
                  (size_t)FP6M_STATIC_SCRATCH_BYTES, dev, stream, thread_k, thread_n, sms, max_par,
                  quant_cols, group_size, layout, status_dev);
}

int fp6m_dump_operands(const void* B, const void* s, void* W_out, int N, int K, int quant_cols,
                       int group_size, int dev, void* stream) {
  if (!B || !s || !W_out || N <= 0 || K <= 0) return FP6M_ERR_BAD_ARG;
  if (!(group_size == 128 || group_size <= 0)) return FP6M_ERR_BAD_ARG;
  const int qc = quant_cols < 0 ? 0 : quant_cols;
  if (qc > N) return FP6M_ERR_BAD_ARG;
  DeviceGuard guard(dev);
  cudaError_t e = launch_dump_operands(static_cast<const uint8_t*>(B), static_cast<const half*>(s),
                                       static_cast<half*>(W_out), make_geometry(K, N, qc, group_size),
                                       static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? FP6M_OK : cuda_fail(e, "dump_operands launch");
}

int fp6m_set_launch_overlap(int enable) {
  const int before = tc5_get_overlap() ? 1 : 0;
  if (enable >= 0) tc5_set_overlap(enable != 0);
  return before;
}

int fp6m_set_ordered_sums(int enable) {
  const int before = tc5_get_ordered_sums() ? 1 : 0;
  if (enable >= 0) tc5_set_ordered_sums(enable != 0);
  return before;
}

const char* fp6m_last_cuda_error(void) { return g_cuda_error; }

const char* fp6m_version(void) { return "fp6m-b200 0.1 (sm_100a)"; }

}  // extern "C"
