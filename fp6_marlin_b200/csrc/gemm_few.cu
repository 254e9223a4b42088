// W(4&6)A16 GEMM for up to 8 rows of A (token generation), on mma.sync with the weights expanded in registers.
//
// Why not tcgen05 here: a call of a few rows is a few microseconds, most of it set-up, first data and tails, and with tensor
// memory a CTA allocates 512 columns and passes operands, sums and slots between roles through mbarriers.
// Here a consumer warp keeps a tile to itself: packed words -> registers -> mma.sync
// m16n8k16 -> registers, one barrier wait per segment.
// What bounds it: an m16n8k16 takes 7.4 cycles of an SM quarter's issue, the other instructions about one each (micro-benchmarks),
// so the inner loop of a segment needs 320 cycles of issue with one tile of eight rows and 450 with two, against 350 that HBM needs for its
// 8 KB; from 9 rows on the kernel of gemm_team.cu, whose MMAs cost no issue slots, is the faster one.  In a launch a segment costs 530
// cycles (from 4096 x 22016 to 8192 x 57344 at 8 rows), so waits between the roles add to that; K = N = 8192 has 43 % of the issue
// slots busy, and set-up, first data and tail are a third of a CTA's life.
// Measured, us per GEMM in a chain of launches (256 FP6 columns, group scales, weights larger than L2), against the tcgen05 kernel that served
// these sizes before, without / with launch overlap:
//   4096 x 4096 at 1 row 8.7 / 7.7 -> 6.3 / 6.2, 4096 x 12288 at 5 rows 12.85 / 12.35 -> 9.85 / 9.45, 4096 x 22016 at 5 rows 17.9 / 17.6 -> 14.9 /
//   14.4, 11008 x 4096 at 5 rows 12.8 / 12.85 -> 9.8 / 9.5, K = N = 8192 at 8 rows 14.45 / 14.05 -> 11.75 / 11.4, 8192 x 57344 at 5 rows
//   66.0 / 65.6 -> 56.4 / 56.2, 16384 x 1024 at 8 rows 12.2 / 10.9 -> 9.1 / 8.9;
//   with two tiles, at 16 rows with overlap: K = N = 8192 13.8 -> 15.3, 8192 x 57344 62 -> 74 (hence the line at 8 rows).
//
// The product is computed transposed, as in the other kernels: W is the 16-row operand (16 weight columns x 16 rows of K), A the
// 8-column one.  The order of K inside a fragment is free as long as both operands agree, so a thread (g = lane / 4,
// t = lane % 4) takes the packed words 2 t and 2 t + 1 of a 64-row unit of its columns - 16 consecutive rows of K - and the two
// 16-byte chunks of its row of A with the same numbers: no shuffles, and both come as wide conflict-free loads.
// Roles (12 warps): eight consumers - two sets of four, a set takes every second segment, a warp 32 of its columns; two
// weights producers (every second segment each); one activations producer (cp.async, 16 bytes a lane, so that no tensor
// map is encoded on the host); one warp for the launch epoch.
// The group scale is applied in fp32 to the sums of a segment.  At the end of a slice (the CTA's blocks of a strip) the sets pool
// their sums through shared memory in a fixed order, turned round so that lane = column.  Sums are always added in one
// order: results repeat bit for bit.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <type_traits>

#include "device_utils.cuh"
#include "fp6m_layout.h"
#include "gemm_params.h"
#include "tc5_common.cuh"

namespace fp6m {

namespace {

constexpr int kStages = 8;
constexpr int kRows = kFewMaxRows;                   // one mma tile of eight rows of A
constexpr int kSets = 2;                             // sets of four consumer warps; a set takes every second segment
constexpr int kConsumers = 4 * kSets;
constexpr int kThreads = 32 * (kConsumers + 4);
static_assert(kStages % kSets == 0, "a stage always belongs to the same set");
static_assert(kStages % 2 == 0 && kStages <= 32, "and to the same producer; the first round of copies is issued by one lane per stage");
constexpr int kActBytes = kRows * 256;
constexpr int kStageBytes = kStageW + kActBytes;
constexpr int kXchPitch = 36;                        // words per row of the exchange buffer: 2 rows = 72 words, 8 banks apart
constexpr int kXchQuad = kRows * kXchPitch * 4;      // one quad of 32 columns
constexpr int kNumBars = 2 * kStages + 1;
constexpr int kSmemBytes = kStages * kStageBytes + 4 * kXchQuad + kNumBars * 8 + 16 + 128;
constexpr int kOutRows = kRows / kSets;              // finished rows per consumer thread

__device__ __forceinline__ float lds_half(uint32_t addr) { return __half2float(__ushort_as_half((unsigned short)lds_u16(addr))); }

// D (16 columns of W x 8 rows of A) += W fragment x A fragment; `first` starts from zero
__device__ __forceinline__ void mma_tile(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, bool first) {
  if (first) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

__global__ void __launch_bounds__(kThreads, 1) w46_gemm_few_kernel(const __grid_constant__ MulParams p) {
  constexpr int S = kStages;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint32_t xch0 = smem0 + S * kStageBytes;
  const uint32_t full = xch0 + 4 * kXchQuad, empty = full + 8 * S, epoch_bar = empty + 8 * S;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_raw + (epoch_bar + 8 - smem_u32(smem_raw)));    // [0] launch epoch

  const int tid = threadIdx.x, warp = uniform_warp_index(), lane = tid & 31;
  // ranges are handed out from the last to the first, see add_partials
  const int cta = gridDim.x - 1 - blockIdx.x;
  const Geometry& geo = p.geo;
  const int kb = geo.k128;                       // blocks (segments) per strip
  const int B0 = p.sched.bound[cta] >> 1, B1 = p.sched.bound[cta + 1] >> 1;
  const int nseg = B1 - B0;
  launch_dependents();
  if (nseg <= 0) {                     // no work: still counted, see read_epoch_and_count
    if (tid == 0) {
      grid_dependency_wait();
      read_epoch_and_count(p.epochs, gridDim.x);
    }
    return;
  }
  WaitState ws;
  const int s_first = B0 / kb, blk_first = B0 - s_first * kb;
  const uint64_t policy = make_evict_first_policy();

  // ---- set-up: lane i of the first producer prepares stage i and issues its first copy
  if (warp == kConsumers) {
    if (lane < S) {
      mbar_init(full + 8 * lane, 1 + 32);          // expect_tx arrival of the weights producer, 32 lanes of the activations producer
      mbar_init(empty + 8 * lane, 4);              // one lane of each warp of the set
      if (lane == 0) mbar_init(epoch_bar, 1);
      mbar_fence_init();
      if (lane < nseg) {
        int s = s_first, blk = blk_first + lane;
        while (blk >= kb) { blk -= kb; ++s; }
        const uint32_t bytes = segment_bytes(geo, s), sbytes = segment_scale_bytes(geo, s);
        const uint8_t* src = p.B + segment_offset(geo, s, blk);
        const half* ssrc = p.S + (sbytes ? int4_scale_offset(geo, s, blk) : 0);
        if (!p.weights_early) {
          // the kernel before this one may be writing the weights: bring the lines into L2 while it finishes, read them after it
          tma_prefetch_l2(src, bytes, policy);
          if (sbytes) tma_prefetch_l2(ssrc, sbytes, policy);
          grid_dependency_wait();
        }
        mbar_arrive_expect_tx(full + 8 * lane, bytes + sbytes);
        tma_load_1d_stream(smem0 + lane * kStageBytes, src, bytes, full + 8 * lane, policy);
        if (sbytes) tma_load_1d_stream(smem0 + lane * kStageBytes + kStageScaleOff, ssrc, sbytes, full + 8 * lane, policy);
      }
    }
    __syncwarp();
  } else if (p.M < kRows) {
    // rows of the activation tiles that A does not have stay zero
    const int t = warp < kConsumers ? tid : tid - 32;
    const int vecs = (kRows - p.M) * 8;                  // 16-byte vectors per unit and stage
    for (int i = t; i < S * 2 * vecs; i += kThreads - 32) {
      const int tile = i / vecs, v = i - tile * vecs;    // tile = stage * 2 + unit
      const uint32_t at = smem0 + (tile >> 1) * kStageBytes + kStageW + (tile & 1) * (kRows * 128) + p.M * 128 + v * 16;
      asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0) : "memory");
    }
  }
  __syncthreads();
  grid_dependency_wait();

  if (warp >= kConsumers && warp < kConsumers + 2) {
    // ================================================================== weights producers: every other segment each
    int n = S + (warp - kConsumers);
    if (n < nseg) {
      int s = s_first, blk = blk_first + n;
      while (blk >= kb) { blk -= kb; ++s; }
      const uint8_t* src = p.B + segment_offset(geo, s, blk);
      uint32_t bytes = segment_bytes(geo, s), sbytes = segment_scale_bytes(geo, s);
      const uint8_t* ssrc = reinterpret_cast<const uint8_t*>(p.S + (sbytes ? int4_scale_offset(geo, s, blk) : 0));
      int stage = n - S;
      uint32_t phase = 0;                      // parity of the stage's previous use
      for (; n < nseg; n += 2) {
        mbar_wait<32>(empty + 8 * stage, phase, ws);
        if (elect_one()) {
          mbar_arrive_expect_tx(full + 8 * stage, bytes + sbytes);
          tma_load_1d_stream(smem0 + stage * kStageBytes, src, bytes, full + 8 * stage, policy);
          if (sbytes) tma_load_1d_stream(smem0 + stage * kStageBytes + kStageScaleOff, ssrc, sbytes, full + 8 * stage, policy);
        }
        __syncwarp();
        src += 2 * bytes;                      // blocks of a strip, and their groups, follow one another without gaps
        ssrc += 2 * sbytes;
        blk += 2;
        if (blk >= kb) {
          while (blk >= kb) { blk -= kb; ++s; }
          if (n + 2 < nseg) {
            src = p.B + segment_offset(geo, s, blk);
            bytes = segment_bytes(geo, s);
            sbytes = segment_scale_bytes(geo, s);
            if (sbytes) ssrc = reinterpret_cast<const uint8_t*>(p.S + int4_scale_offset(geo, s, blk));
          }
        }
        stage += 2;
        if (stage >= S) { stage -= S; phase ^= 1; }
      }
    }
  } else if (warp == kConsumers + 2) {
    // ================================================================== activations producer
    // lane: 16-byte chunk w of the rows r0, r0 + 2, ...  (Unrolled, with the addresses prepared: computing eight of them per
    // segment in a loop made this warp the bottleneck, 8192 x 57344 at 16 rows 83 instead of 77 us.)
    const int w = lane & 15, r0 = lane >> 4;
    const uint32_t dst0 = smem0 + kStageW + (w >> 3) * (kRows * 128) + r0 * 128;
    const uint32_t swz = ((w & 7) ^ r0) << 4;                // (chunk ^ row % 8) * 16 without the row's upper bits
    const size_t two_rows = 2 * (size_t)p.K;
    const half* row_base = p.A + (size_t)(r0 < p.M ? r0 : 0) * p.K + w * 8;
    int stage = 0, blk = blk_first;
    uint32_t phase = 1;                        // a fresh barrier passes parity 1
    for (int n = 0; n < nseg; ++n) {
      const bool inside = blk * kBlockRows + w * 8 < p.K;    // the last block may be half a block: zeros
      const half* src = inside ? row_base + blk * kBlockRows : p.A;
      const size_t step = inside ? two_rows : 0;
      const int bytes = inside ? 16 : 0;
      const uint32_t dst = dst0 + stage * kStageBytes;
      mbar_wait<64>(empty + 8 * stage, phase, ws);
#pragma unroll
      for (int i = 0; i < kRows / 2; ++i) {
        if (2 * i + r0 < p.M)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 256 + (swz ^ ((2 * i & 7) << 4))), "l"(src), "r"(bytes) : "memory");
        src += step;
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full + 8 * stage) : "memory");
      if (++blk == kb) blk = 0;
      if (++stage == S) { stage = 0; phase ^= 1; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == kConsumers + 3) {
    // ================================================================== launch epoch
    if (lane == 0) {
      misc[0] = read_epoch_and_count(p.epochs, gridDim.x);
      mbar_arrive(epoch_bar);
    }
  } else {
    // ================================================================== consumers
    const int set = warp >> 2, q = warp & 3;
    const int g = lane >> 2, t = lane & 3;
    // this thread's packed words of a unit: words 2 t and 2 t + 1 of the columns 32 q + 8 o + g (o = 0..3)
    const uint32_t w_off = q * 1024 + g * 32 + ((((t >> 1) ^ (g >> 2)) & 1) << 4) + ((t & 1) << 3);
    const uint32_t two_off = q * 512 + g * 16 + t * 4;
    // its chunks 2 t and 2 t + 1 of activation row g
    const uint32_t b_off0 = kStageW + g * 128 + (((2 * t) ^ g) << 4), b_off1 = kStageW + g * 128 + (((2 * t + 1) ^ g) << 4);
    const uint32_t sc_off = kStageScaleOff + 2 * (32 * q + g);
    const int c = 32 * q + lane;                 // column inside the strip, for finished values
    const int row0 = set * kOutRows;             // first finished row of this thread
    const uint32_t xch = xch0 + q * kXchQuad;

    float acc[2][4];                             // [tile of 16 columns][column g / g + 8, row 2 t / 2 t + 1]
    int n = set, stage = set;
    uint32_t phase = 0;

    auto segments = [&](auto six, int n_end, uint32_t unit_bytes, uint32_t two_base, bool scaled, bool live) {
      constexpr bool IS6 = decltype(six)::value;
#pragma unroll 1
      for (; n < n_end; n += kSets) {
        mbar_wait<20>(full + 8 * stage, phase, ws);
        const uint32_t st = smem0 + stage * kStageBytes;
        if (live) {
          float d[2][2][4];                      // two accumulators per tile, used in turn
          float sc[2][2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint2 w[4];
            uint32_t two[4];
#pragma unroll
            for (int o = 0; o < 4; ++o) w[o] = lds64(st + u * unit_bytes + w_off + o * 256);
            if constexpr (IS6) {
#pragma unroll
              for (int o = 0; o < 4; ++o) two[o] = lds_u32(st + u * unit_bytes + two_base + two_off + o * 128);
            }
            const uint4 b[2] = {lds128(st + b_off0 + u * (kRows * 128)), lds128(st + b_off1 + u * (kRows * 128))};
            if (u == 1) {
#pragma unroll
              for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) sc[mt][h] = (!IS6 && scaled) ? lds_half(st + sc_off + 32 * mt + 16 * h) : 1.f;
              __syncwarp();
              if (lane == 0) mbar_arrive(empty + 8 * stage);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint32_t e0[2][4], e1[2][4];
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) {
                const uint32_t w0 = j ? w[2 * mt].y : w[2 * mt].x, w1 = j ? w[2 * mt + 1].y : w[2 * mt + 1].x;
                if constexpr (IS6) {
                  expand_fp6(w0, two[2 * mt], 4 * j, e0[mt]);
                  expand_fp6(w1, two[2 * mt + 1], 4 * j, e1[mt]);
                } else {
                  expand_int4(w0, e0[mt]);
                  expand_int4(w1, e1[mt]);
                }
              }
              const bool first = u == 0 && j == 0;
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) mma_tile(d[0][mt], e0[mt][0], e1[mt][0], e0[mt][1], e1[mt][1], b[j].x, b[j].y, first);
#pragma unroll
              for (int mt = 0; mt < 2; ++mt) mma_tile(d[1][mt], e0[mt][2], e1[mt][2], e0[mt][3], e1[mt][3], b[j].z, b[j].w, first);
            }
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[mt][v] = fmaf(sc[mt][v >> 1], d[0][mt][v] + d[1][mt][v], acc[mt][v]);
        } else {
          __syncwarp();
          if (lane == 0) mbar_arrive(empty + 8 * stage);
        }
        stage += kSets;
        if (stage >= S) { stage -= S; phase ^= 1; }
      }
    };

    int n_first = 0;
    for (int s = s_first; n_first < nseg; ++s) {
      const bool is6 = s >= geo.strips4;
      const int strip = is6 ? s - geo.strips4 : s;
      const int region = is6 ? geo.n6 : geo.n4;
      const int nq = strip_quads(region, strip);
      const int b0 = s == s_first ? blk_first : 0;
      const int n_end = min(nseg, (s + 1) * kb - B0);
      const int b1 = b0 + (n_end - n_first);
      const bool group = !is6 && geo.groups > 1;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[mt][v] = 0.f;
      if (is6) segments(std::true_type{}, n_end, nq * kFp6UnitQuadBytes, nq * kInt4UnitQuadBytes, false, q < nq);
      else segments(std::false_type{}, n_end, nq * kInt4UnitQuadBytes, 0, group, q < nq);
      n_first = n_end;
      if (q >= nq) continue;                   // a quad that a ragged strip does not have (the quad's warps of both sets)
      // ---- the sets' sums of the slice, pooled through shared memory in the order of the sets and turned round so that
      // lane = column: a thread of set e gets the rows e * kOutRows ... of its column
      auto at = [&](int mt, int v) { return xch + (((2 * t + (v & 1)) * kXchPitch) + 16 * mt + 8 * (v >> 1) + g) * 4; };
      named_bar_sync(1 + q, 32 * kSets);       // the buffer of the slice before has been read
      if (set == 1) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int v = 0; v < 4; ++v) sts_f32(at(mt, v), acc[mt][v]);
      }
      named_bar_sync(1 + q, 32 * kSets);
      if (set == 0) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int v = 0; v < 4; ++v) sts_f32(at(mt, v), acc[mt][v] + lds_f32(at(mt, v)));
      }
      named_bar_sync(1 + q, 32 * kSets);
      float out[kOutRows];
#pragma unroll
      for (int m = 0; m < kOutRows; ++m) out[m] = lds_f32(xch + ((row0 + m) * kXchPitch + lane) * 4);

      uint32_t tag = 0;
      if (b0 > 0 || b1 < kb) {
        mbar_wait(epoch_bar, 0, ws);
        tag = misc[0] + 1;                       // launch epoch + 1
      }
      if (b0 > 0) {
        store_partial<kOutRows>(p, cta, kRows, row0, c, tag, out);
        continue;
      }
      if (b1 < kb) add_partials<kOutRows>(p, cta, (s + 1) * kb, kRows, row0, c, tag, out, ws);
      const bool writes = c < strip_cols(region, strip);
      const float col_scale = strip_column_scale(p, is6, strip, c, writes);
#pragma unroll
      for (int m = 0; m < kOutRows; ++m) out[m] *= col_scale;
      store_column_rows<kOutRows>(p, row0, is6, strip * kStripCols + c, out, writes);
    }
  }
  report_waits(ws, p.status);
}

// One CTA per SM and eight stages.  Measured and not kept: six stages and 91 KB of shared memory, so that the next launch's CTA is
// resident beside this one - in a chain of different layers an SM without a CTA of a small layer then takes two of the next one
// and others none (the four GEMMs of a Llama-2-7B block at 5 rows 58 us, 4096 x 4096 at 1 row 6.4 -> 7.5; a chain of one layer
// gains 1 to 2 %); twelve stages (K = N = 8192 at 8 rows 11.4 -> 11.7); twelve stages and four sets (12.3; only 8192 x 57344
// gains, 55 -> 51).
}  // namespace

// Runs the GEMM for rows [0, p.M) with p.M <= kFewMaxRows.  The schedule's unit boundaries must be even (whole blocks).
cudaError_t launch_gemm_few(const MulParams& p, cudaStream_t stream) {
  static std::atomic<bool> configured[64] = {};       // threads that find it false set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(w46_gemm_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.sched.ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, w46_gemm_few_kernel, p);
}

}  // namespace fp6m
