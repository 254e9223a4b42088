// Device-side weight preparation: the truncating fp16 -> FP6 E3M2 cast and the packing of logical
// INT4 / FP6 codes and scales into the b200 layout, bit for bit what the host functions of
// host_pack.cpp produce.  The reference prepares weights in single-threaded host loops
// (fp6_marlin/weight_quant.cpp:106-124, fp6_marlin/weight_prepacking.cpp:123-177); for 70B-scale
// layers that takes seconds per layer, here it is a few memory-bound kernels.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fp6m.h"
#include "fp6m_layout.h"

namespace fp6m {

namespace {

// fp16 bits -> code `s eee mm`, mantissa truncated, FP6 subnormals by shifting the mantissa with its
// implicit one (weight_quant.cpp:27-91); values outside {0} U [0.0625, 28] are reported and coded 0.
__device__ __forceinline__ uint8_t encode_fp6(uint16_t h, int* status) {
  const int sign = h >> 15, exp = (h >> 10) & 0x1F, man = h & 0x3FF;
  const uint16_t mag = h & 0x7FFF;
  uint8_t code = 0;
  if ((mag != 0 && mag < 0x2C00) || mag > 0x4F00) {
    if (status) atomicExch(status, FP6M_ERR_VALUE_RANGE);
  } else {
    int e6 = 0, m6 = 0;
    if (exp != 0) {
      const int unbiased = exp - 15;
      m6 = man >> 8;
      if (unbiased < -2) {
        m6 = (m6 | 4) >> (-2 - unbiased);
      } else {
        e6 = unbiased + 3;
      }
    }
    code = (uint8_t)((sign << 5) | (e6 << 2) | m6);
  }
  return code;
}

__global__ void encode_fp6_kernel(const uint16_t* __restrict__ w, uint8_t* __restrict__ codes, size_t count, int* status) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) codes[i] = encode_fp6(w[i], status);
}

// one thread per (strip, unit, column): the column's eight words of the unit
__global__ void pack_int4_kernel(const uint8_t* __restrict__ q4, Geometry geo, uint8_t* __restrict__ B_out) {
  const int ups = units_per_strip(geo);
  const int c = threadIdx.x;                          // column inside the strip
  const int unit = blockIdx.x % ups, strip = blockIdx.x / ups;
  const int nq = strip_quads(geo.n4, strip);
  if (c >= kQuadCols * nq) return;
  uint8_t* base = B_out + int4_unit_offset(geo, strip, unit);
  const int col = strip * kStripCols + c;
  for (int w8 = 0; w8 < 8; ++w8) {
    uint32_t word = 0;
    for (int i = 0; i < 8; ++i) {
      const int row = unit * kUnitRows + 8 * w8 + i;
      uint32_t q = 8;                                 // padding dequantises to zero
      if (row < geo.K && col < geo.n4) q = q4[(size_t)row * geo.n4 + col] & 15u;
      word |= q << (4 * int4_nibble_pos(i));
    }
    *reinterpret_cast<uint32_t*>(base + word_offset(c, w8)) = word;
  }
}

__global__ void pack_fp6_kernel(const uint8_t* __restrict__ c6, Geometry geo, uint8_t* __restrict__ B_out) {
  const int ups = units_per_strip(geo);
  const int c = threadIdx.x;
  const int unit = blockIdx.x % ups, strip = blockIdx.x / ups;
  const int nq = strip_quads(geo.n6, strip);
  if (c >= kQuadCols * nq) return;
  uint8_t* base = B_out + fp6_unit_offset(geo, strip, unit);
  uint8_t* base2 = base + (size_t)nq * kInt4UnitQuadBytes;
  const int col = strip * kStripCols + c;
  uint32_t two[4] = {0, 0, 0, 0};
  for (int w8 = 0; w8 < 8; ++w8) {
    uint32_t four = 0;
    for (int i = 0; i < 8; ++i) {
      const int row = unit * kUnitRows + 8 * w8 + i;
      uint32_t code = 0;
      if (row < geo.K && col < geo.n6) code = c6[(size_t)row * geo.n6 + col] & 63u;
      const int b = i & 3, js = 2 * (w8 & 1) + (i >> 2);
      four |= (code & 15u) << (8 * b + 4 * (i >> 2));
      two[w8 >> 1] |= ((code >> 5) & 1u) << ((8 * b + 7 - 2 * js + 32) & 31);
      two[w8 >> 1] |= ((code >> 4) & 1u) << ((8 * b + 4 - 2 * js + 32) & 31);
    }
    *reinterpret_cast<uint32_t*>(base + word_offset(c, w8)) = four;
  }
  *reinterpret_cast<uint4*>(base2 + c * 16) = make_uint4(two[0], two[1], two[2], two[3]);
}

// scales in plain column order per strip (and per group); padding columns get 1.0
__global__ void pack_scales_kernel(const uint16_t* __restrict__ s4, const uint16_t* __restrict__ s6, Geometry geo,
                                   uint16_t* __restrict__ s_out) {
  const int c = threadIdx.x;
  const int rows4 = geo.strips4 * geo.groups;
  const int b = blockIdx.x;
  if (b < rows4) {
    const int strip = b / geo.groups, grp = b % geo.groups;
    if (c >= kQuadCols * strip_quads(geo.n4, strip)) return;
    const int col = strip * kStripCols + c;
    s_out[int4_scale_offset(geo, strip, grp) + c] = col < geo.n4 ? s4[(size_t)grp * geo.n4 + col] : (uint16_t)0x3C00;
  } else {
    const int strip = b - rows4;
    if (c >= kQuadCols * strip_quads(geo.n6, strip)) return;
    const int col = strip * kStripCols + c;
    s_out[fp6_scale_offset(geo, strip) + c] = col < geo.n6 ? s6[col] : (uint16_t)0x3C00;
  }
}

// ---- quantise and pack in one go -------------------------------------------------------------------
// fp16 W[k, n] -> packed words and scales, bit for bit what the quantisers of quant.py (torch operations on the
// GPU) followed by the packing kernels above give; W is read once (the columns whose scale spans all of K: twice)
// and nothing but the result is written.  One 4096 x 11008 layer: 1283 us a call through the separate operations (a
// dozen passes over half, float, int32 and byte matrices) -> 81 us, of which the packing kernel is 44 (116 MB, 2.6 TB/s;
// it is bound by its conversions and fused multiply-adds, about eight instructions per value) and the synchronising check
// of the FP6 columns most of the rest.
// Rows that start off a 4-byte boundary, or an odd width, take the forms without pair loads (timed alone: 97 us -> 110 / 119).

// Two neighbouring columns of a row, zero where `c0` / `c1` say that there is no such column.  kPair: the address is
// 4-byte aligned and the columns exist or are missing together.
template <bool kPair>
__device__ __forceinline__ half2 load_pair(const half* __restrict__ w, size_t at, bool c0, bool c1) {
  const half z = __ushort_as_half(0);
  if constexpr (kPair) return c1 ? *reinterpret_cast<const half2*>(w + at) : __half2half2(z);
  return __halves2half2(c0 ? w[at] : z, c1 ? w[at + 1] : z);
}

// Scales of the columns that have one for all of K (FP6: max|w| / 28, INT4 without groups: max|w| * 2/15), straight into
// the packed scale order; padding columns get 1.0.  One CTA = 16 columns (one 32-byte sector per row) and all rows: no
// atomics, no second pass.  Also clears the status word that the packing kernel may set.
constexpr int kMaxCols = 16, kMaxThreads = 1024;
template <bool kPair>
__global__ void __launch_bounds__(kMaxThreads) column_scales_kernel(const half* __restrict__ w, Geometry geo, int ctas4, uint16_t* __restrict__ s_out, int* status) {
  const bool is6 = (int)blockIdx.x >= ctas4;
  const int col0 = ((int)blockIdx.x - (is6 ? ctas4 : 0)) * kMaxCols;         // inside the region
  const int ncols = is6 ? geo.n6 : geo.n4;
  const int pair = threadIdx.x & 7, warp = threadIdx.x >> 5;
  const int c = col0 + 2 * pair;
  const bool c0 = c < ncols, c1 = c + 1 < ncols;
  if (blockIdx.x == 0 && threadIdx.x == 0 && status) *status = 0;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");       // the packing kernel's INT4 blocks need nothing from here
  half2 m = __half2half2(__ushort_as_half(0));
  const half* src = w + (is6 ? geo.n4 : 0) + c;
  constexpr int kStep = kMaxThreads / 8, kBatch = 16;                   // loads in flight per thread: the latency is the time
  for (int row0 = threadIdx.x >> 3; row0 < geo.K; row0 += kStep * kBatch) {
    half2 v[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int row = row0 + i * kStep;
      v[i] = load_pair<kPair>(src, (size_t)row * geo.N, c0 && row < geo.K, c1 && row < geo.K);
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) m = __hmax2_nan(m, __habs2(v[i]));
  }
  for (int d = 8; d < 32; d *= 2) m = __hmax2_nan(m, __shfl_xor_sync(0xffffffffu, m, d));
  __shared__ half2 part[kMaxThreads / 32][8];
  if ((threadIdx.x & 31) < 8) part[warp][pair] = m;
  __syncthreads();
  if (threadIdx.x < 8) {
    for (int i = 1; i < kMaxThreads / 32; ++i) m = __hmax2_nan(m, part[i][pair]);
    const int strip = c / kStripCols, in_strip = c % kStripCols;
    uint16_t* dst = s_out + (is6 ? fp6_scale_offset(geo, strip) : int4_scale_offset(geo, strip, 0)) + in_strip;
    const float factor = is6 ? (float)(1.0 / 28.0) : (float)(2.0 / 15.0);
    dst[0] = c0 ? __half_as_ushort(__float2half_rn(__low2float(m) * factor)) : (uint16_t)0x3C00;
    dst[1] = c1 ? __half_as_ushort(__float2half_rn(__high2float(m) * factor)) : (uint16_t)0x3C00;
  }
}

// w / s in fp32, correctly rounded, for finite w and finite s > 0 with r = 1 / s correctly rounded: Markstein's division (IBM J. Res.
// Dev. 34, 1990) - quotient, exact remainder, correction.  Both come from halves, so nothing over- or underflows; the
// plain operator, which has to care, was three quarters of this kernel's 102 us.
__device__ __forceinline__ float quotient(float w, float s, float r) {
  const float q = w * r;
  return fmaf(fmaf(-q, s, w), r, q);
}
// INT4 codes where that does not hold (scale zero, infinite or NaN), as the int32 tensors of the torch rule give them.
__device__ __noinline__ uint32_t quantize_int4_special(float w, float s, bool group) {
  const int r = __float2int_rz(rintf(__half2float(__float2half_rn(w / s))));
  if (group) return (uint32_t)(min(max(r, -8), 7) + 8);
  return (uint32_t)min(max((int)((unsigned)r + 8u), 0), 15);        // r may be INT_MAX: the sum wraps
}
__device__ __forceinline__ uint32_t quantize_fp6(half w, float s, int* status) {
  half x = __float2half_rn(__half2float(w) / s);
  if (__half2float(__habs(x)) < 0.0625f) x = __ushort_as_half(0);
  if (__half2float(x) > 28.f) x = __ushort_as_half(0x4F00);
  if (__half2float(x) < -28.f) x = __ushort_as_half(0xCF00);
  return encode_fp6(__half_as_ushort(x), status);
}

// One CTA = one 128-row block of one strip (INT4 strips first).  Thread = two neighbouring columns x 32 rows, so a warp
// reads whole 128-byte lines and a thread finishes 16 of the 32 bytes of each of its columns' words of a unit; the four
// row quarters meet in shared memory for the group maximum.
template <bool kPair>
__global__ void __launch_bounds__(256, 4) quantize_pack_kernel(const half* __restrict__ w, Geometry geo, bool group_scales, uint8_t* __restrict__ B_out,
                                                            uint16_t* s_out, int* status) {
  const bool is6 = (int)blockIdx.x >= geo.strips4 * geo.k128;
  const int at = (int)blockIdx.x - (is6 ? geo.strips4 * geo.k128 : 0);
  const int strip = at / geo.k128, block = at % geo.k128;
  const int region_cols = is6 ? geo.n6 : geo.n4;
  const int nq = strip_quads(region_cols, strip);
  const int warp = threadIdx.x >> 5, quarter = warp >> 1;
  const int pair = (warp & 1) * 32 + (threadIdx.x & 31), c = 2 * pair;      // columns c, c + 1 of the strip
  const int col = strip * kStripCols + c;
  const bool c0 = col < region_cols, c1 = col + 1 < region_cols;
  const int row0 = block * kBlockRows + quarter * 32;
  const half* src = w + (is6 ? geo.n4 : 0) + col;

  const int unit = 2 * block + (quarter >> 1), w8_0 = 4 * (quarter & 1);    // this thread's words of the unit: w8_0 .. w8_0 + 3

  if (is6) {
    // the scales come from column_scales_kernel, during which this kernel may have been started
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (c >= kQuadCols * nq) return;
    const uint16_t* sp = s_out + fp6_scale_offset(geo, strip) + c;
    const float s0 = __half2float(__ushort_as_half(sp[0])), s1 = __half2float(__ushort_as_half(sp[1]));
    uint8_t* base = B_out + fp6_unit_offset(geo, strip, unit);
    uint32_t* four0 = reinterpret_cast<uint32_t*>(base + word_offset(c, w8_0));
    uint32_t* four1 = reinterpret_cast<uint32_t*>(base + word_offset(c + 1, w8_0));
    uint32_t* two = reinterpret_cast<uint32_t*>(base + (size_t)nq * kInt4UnitQuadBytes + c * 16 + (quarter & 1) * 8);
#pragma unroll 1
    for (int j = 0; j < 4; j += 2) {                    // two words of each column and the two-bit word that goes with them
      half2 x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int row = row0 + 8 * j + i;
        x[i] = load_pair<kPair>(src, (size_t)row * geo.N, c0 && row < geo.K, c1 && row < geo.K);
      }
      uint32_t f0[2] = {0, 0}, f1[2] = {0, 0}, t0 = 0, t1 = 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const bool here = row0 + 8 * j + i < geo.K;
        const uint32_t code0 = here && c0 ? quantize_fp6(__low2half(x[i]), s0, status) : 0u;
        const uint32_t code1 = here && c1 ? quantize_fp6(__high2half(x[i]), s1, status) : 0u;
        const int b = i & 3, js = i >> 2, four_shift = 8 * b + (js & 1) * 4;
        f0[i >> 3] |= (code0 & 15u) << four_shift;
        f1[i >> 3] |= (code1 & 15u) << four_shift;
        t0 |= (((code0 >> 5) & 1u) << ((8 * b + 7 - 2 * js + 32) & 31)) | (((code0 >> 4) & 1u) << ((8 * b + 4 - 2 * js + 32) & 31));
        t1 |= (((code1 >> 5) & 1u) << ((8 * b + 7 - 2 * js + 32) & 31)) | (((code1 >> 4) & 1u) << ((8 * b + 4 - 2 * js + 32) & 31));
      }
      *reinterpret_cast<uint2*>(four0 + j) = make_uint2(f0[0], f0[1]);
      *reinterpret_cast<uint2*>(four1 + j) = make_uint2(f1[0], f1[1]);
      two[j >> 1] = t0;
      two[4 + (j >> 1)] = t1;
    }
    return;
  }

  half2 v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = load_pair<kPair>(src, (size_t)(row0 + i) * geo.N, c0 && row0 + i < geo.K, c1 && row0 + i < geo.K);

  float s0, s1;
  if (group_scales) {
    __shared__ half2 part[4][64];
    half2 m = __habs2(v[0]);
#pragma unroll
    for (int i = 1; i < 32; ++i) m = __hmax2_nan(m, __habs2(v[i]));
    part[quarter][pair] = m;
    __syncthreads();
    m = __hmax2_nan(__hmax2_nan(part[0][pair], part[1][pair]), __hmax2_nan(part[2][pair], part[3][pair]));
    // torch divides a tensor by a number as a product with its fp32 reciprocal
    half h0 = __float2half_rn(__low2float(m) * (1.0f / 7.0f)), h1 = __float2half_rn(__high2float(m) * (1.0f / 7.0f));
    if (__half2float(h0) == 0.f) h0 = __ushort_as_half(0x3C00);
    if (__half2float(h1) == 0.f) h1 = __ushort_as_half(0x3C00);
    if (quarter == 0 && c < kQuadCols * nq) {
      uint16_t* dst = s_out + int4_scale_offset(geo, strip, block) + c;
      dst[0] = c0 ? __half_as_ushort(h0) : (uint16_t)0x3C00;
      dst[1] = c1 ? __half_as_ushort(h1) : (uint16_t)0x3C00;
    }
    s0 = __half2float(h0);
    s1 = __half2float(h1);
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (c >= kQuadCols * nq) return;
    const uint16_t* sp = s_out + int4_scale_offset(geo, strip, 0) + c;
    s0 = __half2float(__ushort_as_half(sp[0]));
    s1 = __half2float(__ushort_as_half(sp[1]));
  }
  if (c >= kQuadCols * nq) return;

  uint8_t* base = B_out + int4_unit_offset(geo, strip, unit);
  uint32_t words[2][4];
  if (s0 > 0.f && s0 < INFINITY && s1 > 0.f && s1 < INFINITY) {
    // both columns at once: fp16(w / s) clamped to [-8, 7], and the sum with 1544 = 1536 + 8, whose unit in the last
    // place is 1, rounds it to the nearest integer (ties to even, 1544 is even) and leaves the code in the low nibble
    const float r0 = 1.f / s0, r1 = 1.f / s1;
    const half2 lowest = __float2half2_rn(-8.f), highest = __float2half2_rn(7.f), offset = __float2half2_rn(1544.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t low = 0, high = 0;                     // nibbles 0..3 and 4..7 of both columns' words
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 x = __half22float2(v[8 * j + i]);
        half2 q = __floats2half2_rn(quotient(x.x, s0, r0), quotient(x.y, s1, r1));
        q = __hadd2_rn(__hmax2(__hmin2(q, highest), lowest), offset);
        const uint32_t code = *reinterpret_cast<const uint32_t*>(&q) & 0x000F000Fu;
        if (i & 1) high |= code << (4 * (i >> 1)); else low |= code << (4 * (i >> 1));
      }
      words[0][j] = __byte_perm(low, high, 0x5410);
      words[1][j] = __byte_perm(low, high, 0x7632);
    }
  } else {
    // rare: value by value, read again (keeping the 32 pairs alive for this would cost the other path its registers)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      words[0][j] = words[1][j] = 0;
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        const int row = row0 + 8 * j + i;
        const half2 x = load_pair<kPair>(src, (size_t)row * geo.N, c0 && row < geo.K, c1 && row < geo.K);
        words[0][j] |= quantize_int4_special(__low2float(x), s0, group_scales) << (4 * int4_nibble_pos(i));
        words[1][j] |= quantize_int4_special(__high2float(x), s1, group_scales) << (4 * int4_nibble_pos(i));
      }
    }
  }
  // rows and columns that do not exist carry the code of zero
#pragma unroll
  for (int side = 0; side < 2; ++side)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rows = (side ? c1 : c0) ? geo.K - (row0 + 8 * j) : 0;      // of this word that exist
      if (rows < 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i >= rows) words[side][j] = (words[side][j] & ~(15u << (4 * int4_nibble_pos(i)))) | (8u << (4 * int4_nibble_pos(i)));
      }
    }
#pragma unroll
  for (int side = 0; side < 2; ++side)
    *reinterpret_cast<uint4*>(base + word_offset(c + side, w8_0)) = make_uint4(words[side][0], words[side][1], words[side][2], words[side][3]);
}

struct Guard {
  int prev = -1;
  explicit Guard(int dev) {
    cudaGetDevice(&prev);
    if (dev >= 0 && dev != prev) cudaSetDevice(dev);
  }
  ~Guard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

}  // namespace
}  // namespace fp6m

using namespace fp6m;

extern "C" {

int fp6m_encode_fp6_device(const void* w, void* codes, size_t count, int dev, void* stream, int* status_dev) {
  if (!w || !codes) return FP6M_ERR_BAD_ARG;
  if (count == 0) return FP6M_OK;
  Guard guard(dev);
  const int threads = 256;
  const size_t blocks = (count + threads - 1) / threads;
  if (blocks > 0x7fffffffu) return FP6M_ERR_BAD_ARG;
  encode_fp6_kernel<<<(unsigned)blocks, threads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint16_t*>(w), static_cast<uint8_t*>(codes), count, status_dev);
  return cudaGetLastError() == cudaSuccess ? FP6M_OK : FP6M_ERR_CUDA;
}

int fp6m_pack_b200_device(const void* q4, const void* c6, const void* s4, const void* s6, int K, int N, int qc, int group_size,
                          void* B_out, void* s_out, int dev, void* stream) {
  if (K <= 0 || N <= 0 || qc > N || !B_out || !s_out) return FP6M_ERR_BAD_ARG;
  if (!(group_size == 128 || group_size <= 0)) return FP6M_ERR_BAD_ARG;
  const Geometry geo = make_geometry(K, N, qc, group_size);
  if ((geo.n4 > 0 && (!q4 || !s4)) || (geo.n6 > 0 && (!c6 || !s6))) return FP6M_ERR_BAD_ARG;
  Guard guard(dev);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int ups = units_per_strip(geo);
  if (geo.strips4 > 0)
    pack_int4_kernel<<<geo.strips4 * ups, kStripCols, 0, st>>>(static_cast<const uint8_t*>(q4), geo, static_cast<uint8_t*>(B_out));
  if (geo.strips6 > 0)
    pack_fp6_kernel<<<geo.strips6 * ups, kStripCols, 0, st>>>(static_cast<const uint8_t*>(c6), geo, static_cast<uint8_t*>(B_out));
  pack_scales_kernel<<<geo.strips4 * geo.groups + geo.strips6, kStripCols, 0, st>>>(
      static_cast<const uint16_t*>(s4), static_cast<const uint16_t*>(s6), geo, static_cast<uint16_t*>(s_out));
  return cudaGetLastError() == cudaSuccess ? FP6M_OK : FP6M_ERR_CUDA;
}

int fp6m_quantize_pack_b200_device(const void* w, int K, int N, int qc, int group_size, void* B_out, void* s_out,
                                   int dev, void* stream, int* status_dev) {
  if (K <= 0 || N <= 0 || qc > N || !w || !B_out || !s_out) return FP6M_ERR_BAD_ARG;
  if (!(group_size == 128 || group_size <= 0)) return FP6M_ERR_BAD_ARG;
  if (group_size == 128 && K % kBlockRows) return FP6M_ERR_PROB_SHAPE;
  if ((reinterpret_cast<uintptr_t>(w) & 1) || (reinterpret_cast<uintptr_t>(B_out) & 15) || (reinterpret_cast<uintptr_t>(s_out) & 1)) return FP6M_ERR_BAD_ARG;
  const Geometry geo = make_geometry(K, N, qc, group_size);
  if ((int64_t)(geo.strips4 + geo.strips6) * geo.k128 > 0x7fffffff) return FP6M_ERR_BAD_ARG;
  Guard guard(dev);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const half* src = static_cast<const half*>(w);
  uint8_t* B = static_cast<uint8_t*>(B_out);
  uint16_t* s = static_cast<uint16_t*>(s_out);
  // pairs of columns by 4-byte loads: rows and the first FP6 column start on 4-byte boundaries
  const bool pairs = (reinterpret_cast<uintptr_t>(w) & 3) == 0 && N % 2 == 0 && geo.n4 % 2 == 0;
  const int ctas4 = group_size > 0 ? 0 : ceil_div(geo.n4, kQuadCols) * (kQuadCols / kMaxCols);
  const int ctas6 = ceil_div(geo.n6, kQuadCols) * (kQuadCols / kMaxCols);
  if (ctas4 + ctas6 > 0) {
    if (pairs) column_scales_kernel<true><<<ctas4 + ctas6, kMaxThreads, 0, st>>>(src, geo, ctas4, s, status_dev);
    else column_scales_kernel<false><<<ctas4 + ctas6, kMaxThreads, 0, st>>>(src, geo, ctas4, s, status_dev);
  }
  const unsigned blocks = (unsigned)((geo.strips4 + geo.strips6) * geo.k128);
  // INT4 blocks with group scales run beside column_scales_kernel (which was launched after everything before it had
  // finished); the blocks that need its scales wait for it
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas4 + ctas6 > 0 ? 1 : 0;
  if (pairs) cudaLaunchKernelEx(&cfg, quantize_pack_kernel<true>, src, geo, group_size > 0, B, s, status_dev);
  else cudaLaunchKernelEx(&cfg, quantize_pack_kernel<false>, src, geo, group_size > 0, B, s, status_dev);
  return cudaGetLastError() == cudaSuccess ? FP6M_OK : FP6M_ERR_CUDA;
}

}  // extern "C"
