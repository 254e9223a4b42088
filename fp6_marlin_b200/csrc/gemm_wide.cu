// W(4&6)A16 GEMM on tcgen05 + TMEM for more than 128 rows of A (up to 128 rows, and on layers with group scales up to 256:
// gemm_tc5.cu).
//
// As in the kernel for up to 128 rows (gemm_tc5.cu) the product is computed transposed: the 128 weight
// columns of a strip are the M dimension of tcgen05.mma (one TMEM lane per column), the rows of A its
// N dimension (a tile's height), the dequantised weights the A operand in TENSOR MEMORY.  Differences:
//   * The INT4 group scale is multiplied into the operand - fp16(q - 8) * s_g with one fp16 rounding,
//     bit for bit the dequantised weight of the reference's rule (test.py:98) - so ONE accumulator
//     tile collects a whole slice of K and is read back once per slice, not once per scale group.
//     Per-channel INT4 scales and FP6 scales (times 4096) are applied to the fp32 sums, as before.
//   * The activations come by tiled TMA: one copy per 64-row unit brings a tile's rows x 64 halves (128-byte
//     rows, 128-byte swizzle) - the K-major swizzled operand layout of tcgen05 with 1024 bytes between
//     8-row groups; a K step of 16 advances the descriptor by 32 bytes.  Rows beyond M are zero-filled
//     by the copy engine.
//   * Segments are whole 128-row blocks (two units); one thread issues all their MMAs.
//   * The rows of a launch are cut into tiles of one height, a multiple of 16 from 48 to 256 (wide_row_tiles): the time of an
//     MMA and of an activations copy goes with the rows (264 rows as 2 x 144 instead of 2 x 256: 4096 x 4096 40.2 -> 30.3 us,
//     K = N = 8192 78.8 -> 56.0, 4096 x 22016 85.3 -> 73.5; 777 rows as 4 x 208: 4096 x 22016 173 -> 167).
// One CTA per SM: warp 0 weights producer, warp 1 activations producer, warp 2 MMA issuer (and owner of TMEM), warp 3
// reads the launch epoch, then four dequantiser warps per team; teams take the segments in turn.
//
// What bounds it: the tensor pipe needs 1024 cycles per segment and 256-row tile, and the L2 -> shared memory path the 64 KB
// of activations in that time.  Cycle counts inside the kernel (K = N = 16384, M = 1024) showed 1741 cycles per segment,
// all but 190 of them the issuer's own: 764 for eight MMAs, the rest bookkeeping, three commits and three waits.  With
// whole blocks, counters in place of a walk and two commits per segment, and with the slices written out only when
// the operands of the next slice already wait in tensor memory (before, the pipe drained at every strip's end):
// K = N = 16384 at M = 4096 2201 -> 1888 us in that comparison (1915 to 1950 in later runs on other GPUs), 4096 x 22016 at
// M = 777 208 -> 179 us.  The MMAs themselves are issued behind elect.sync with operands that are uniform to the compiler: four of
// them and a commit then take 52 cycles of the issuing warp beside eight warps of arithmetic, behind `lane == 0` they took 694,
// more than the 512 of the tensor pipe (K = N = 16384 at M = 1024 462 -> 412 us, 4096 x 22016 at M = 777 139 -> 133, GEMMs back to back).
// Split-K between CTAs uses tagged words as in gemm_tc5.cu, but the CTA in which a strip STARTS sums it: the slice is that CTA's
// last, so its own sums never leave the chip and the next CTA's partial has long been stored.  (When the CTA in which
// the strip ends did it, after its last segment, the reduction took 32,000 cycles, a tenth of the kernel at 4096 x 22016 and
// M = 1024.)  Measured: 4096 x 4096 at M = 512 / 1024 45.9 -> 40.3 / 59.9 -> 44.0 us, 11008 x 4096 at M = 1024 94.2 -> 81.8,
// 4096 x 22016 at M = 777 179 -> 173.
//
// Replaces the reference's large-tile path (thread_m_blocks 2..4 and its `parallel` batches,
// fp6_marlin/fp6_marlin_cuda_kernel.cu:864-951).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "device_utils.cuh"
#include "fp6m_layout.h"
#include "gemm_params.h"
#include "tc5_common.cuh"

namespace fp6m {

namespace {

template <int NT_, int TEAMS_, int STAGES_, int RING_>
struct WideCfg {
  static constexpr int NT = NT_;                       // most rows of A per tile = N of the MMA
  static constexpr int kTeams = TEAMS_;
  static constexpr int kStages = STAGES_;              // weight stages (one segment each)
  static constexpr int kActStages = 4;                 // activation stages (one unit each): two segments
  static constexpr int kRing = RING_;                  // TMEM operand slots (one segment each)
  static constexpr int kDeqBase = 4;
  static constexpr int kThreads = 32 * (kDeqBase + 4 * kTeams);
  static constexpr int kActUnitBytes = NT * 128;       // NT rows x 64 halves, 1024-byte aligned stages
  static constexpr int kNumBars = 2 * kStages + kActStages + 2 + 2 * kRing + 3;
  static constexpr int kOutStageBytes = 2 * 16 * kStripCols * 2;  // per team: two buffers of 16 finished rows of a strip in fp16
  static constexpr int kSmemBytes = kStages * kStageW + kActStages * kActUnitBytes + kTeams * kOutStageBytes + kNumBars * 8 + 64 + 1024;
  static constexpr int kTmemD = 0, kTmemA = NT;        // the accumulator tile, then operand slots of 64 columns
  static constexpr int kTmemUsed = kTmemA + kRing * 64;
  static constexpr int kTmemCols = kTmemUsed <= 128 ? 128 : (kTmemUsed <= 256 ? 256 : 512);
  static constexpr int kSlotWords = NT * kStripCols;
  static constexpr int kChunk = 16;                    // rows read back per tcgen05.ld
  // a stage and an operand slot always belong to the same team, so every waiter of their barriers sees each phase
  static_assert(kTmemUsed <= 512 && kTeams == 2 && NT % 32 == 0 && kStages % kTeams == 0 && kRing % kTeams == 0 && kRing >= 2, "configuration");
};

// coordinates {k0, row0}: k0 is a multiple of 64 halves = 128 bytes, so the copy starts on a 16-byte boundary
__device__ __forceinline__ void tma_load_act_rows(uint32_t dst, const CUtensorMap* map, int k0, int row0, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(k0), "r"(row0), "r"(bar) : "memory");
}

// Tensor maps of the outputs (C, or every rank's full-width output) for the asynchronous row stores; box = 128
// columns x 16 rows.  Only read when p.vec_rows == 2.
struct OutMaps {
  CUtensorMap m[8];
};

// 16 rows x 128 columns of fp16 from shared memory (row-major, 256 bytes per row) to the output behind `map` at
// column x (a multiple of 8), row y; rows beyond the output's last row are clipped by the copy engine.
__device__ __forceinline__ void tma_store_rows(const CUtensorMap* map, uint32_t src_smem, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(x), "r"(y), "r"(src_smem) : "memory");
}

template <class C>
__global__ void __launch_bounds__(C::kThreads, 1)
w46_gemm_wide_kernel(const __grid_constant__ MulParams p, const __grid_constant__ CUtensorMap amap, const __grid_constant__ OutMaps omaps) {
  constexpr int NT = C::NT, S = C::kStages, RA = C::kActStages, R = C::kRing, T = C::kTeams;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* act_base = smem + S * kStageW;
  uint8_t* out_stage = act_base + RA * C::kActUnitBytes;            // [team][16 rows][128 columns] fp16
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + T * C::kOutStageBytes);
  uint32_t* misc = reinterpret_cast<uint32_t*>(bars + C::kNumBars);   // [0] TMEM base, [1] launch epoch
  const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * S;
  const uint32_t a_full = w_empty + 8 * S, a_empty = a_full + 8 * RA;    // a_empty: only the two stages of unit 0
  const uint32_t ready = a_empty + 8 * 2, done = ready + 8 * R;
  const uint32_t slice_done = done + 8 * R, d_read = slice_done + 8, epoch_bar = d_read + 8;

  const int tid = threadIdx.x, warp = uniform_warp_index(), lane = tid & 31;
  // Ranges are handed out from the last to the first: a CTA that has to wait for the partials of higher ranges waits for
  // CTAs that were dispatched before it.
  const int cta = gridDim.x - 1 - blockIdx.x;
  const Geometry& geo = p.geo;
  const int kb = geo.k128;                       // blocks (segments) per strip
  const int nstrips = geo.strips4 + geo.strips6;
  // the CTA's range of blocks of the virtual strips (row tile x strip); the host rounds the boundaries to whole blocks
  const int B0 = p.sched.bound[cta] >> 1, B1 = p.sched.bound[cta + 1] >> 1;
  const int nseg = B1 - B0;
  const int nt = p.tile_rows;                    // rows of this launch's tiles, a multiple of 16
  launch_dependents();
  if (nseg <= 0) {                     // no work: still counted, see read_epoch_and_count
    if (tid == 0) {
      grid_dependency_wait();
      read_epoch_and_count(p.epochs, gridDim.x);
    }
    return;
  }

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(w_full + 8 * s, 1);      // the expect_tx arrival of the weights producer
      mbar_init(w_empty + 8 * s, 4);     // the team that read the stage has its words in registers
    }
    for (int s = 0; s < RA; ++s) mbar_init(a_full + 8 * s, 1);      // the expect_tx arrival of the activations producer
    for (int s = 0; s < 2; ++s) mbar_init(a_empty + 8 * s, 1);      // tcgen05.commit: unit 0's MMAs have read the stage
    for (int r = 0; r < R; ++r) {
      mbar_init(ready + 8 * r, 4);       // the segment's team stored the operands into TMEM
      mbar_init(done + 8 * r, 1);        // tcgen05.commit: the segment's MMAs have finished
    }
    mbar_init(slice_done, 1);            // tcgen05.commit: the accumulator tile holds the whole slice
    mbar_init(d_read, 4 * T);            // every dequantiser warp has read its part of the tile back
    mbar_init(epoch_bar, 1);
    mbar_fence_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(misc)), "r"(C::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, misc[0], 0);      // uniform to the compiler
  bool dead = false;

  if (warp == 0) {
    // ================================================================== weights producer
    {
      const uint64_t policy = make_evict_first_policy();
      int v = B0 / kb, blk = B0 - v * kb;
      int strip = v % nstrips;                         // the strip of the virtual strip
      const uint8_t* wsrc = nullptr;
      uint32_t bytes = 0;
      auto open_strip = [&]() {
        if (strip < geo.strips4) {
          bytes = 2 * strip_quads(geo.n4, strip) * kInt4UnitQuadBytes;
          wsrc = p.B + int4_unit_offset(geo, strip, 2 * blk);
        } else {
          bytes = 2 * strip_quads(geo.n6, strip - geo.strips4) * kFp6UnitQuadBytes;
          wsrc = p.B + fp6_unit_offset(geo, strip - geo.strips4, 2 * blk);
        }
      };
      open_strip();
      int stage = 0;
      uint32_t phase = 0;
      for (int n = 0; n < nseg; ++n) {
        if (n == S) grid_dependency_wait();            // the first S copies need nobody; from here on the teams must have made room
        mbar_wait_bounded<200>(w_empty + 8 * stage, phase ^ 1, p.status, dead);
        if (elect_one()) {
          mbar_arrive_expect_tx(w_full + 8 * stage, bytes);
          tma_load_1d_stream(smem_u32(smem) + stage * kStageW, wsrc, bytes, w_full + 8 * stage, policy);
        }
        __syncwarp();
        wsrc += bytes;                                 // blocks of a strip are contiguous in HBM
        if (++stage == S) { stage = 0; phase ^= 1; }
        if (++blk == kb) {
          blk = 0;
          if (++strip == nstrips) strip = 0;
          open_strip();
        }
      }
    }
  } else if (warp == 1) {
    // ================================================================== activations producer
    // Segment n's units go to the stages 2 (n % 2) and 2 (n % 2) + 1.  Unit 0's stage is free again when a_empty says that
    // the MMAs of segment n - 2 have read it, unit 1's when that segment is done altogether.
    {
      int v = B0 / kb, blk = B0 - v * kb;
      grid_dependency_wait();                           // A may come from the previous kernel
      for (int n = 0; n < nseg; ++n) {
        const int sa = 2 * (n & 1);
        const int row0 = (v / nstrips) * nt;
        const uint32_t dst = smem_u32(act_base) + sa * C::kActUnitBytes;
        if (n >= 2) mbar_wait_bounded<100>(a_empty + 8 * (n & 1), ((n - 2) >> 1) & 1, p.status, dead);
        if (elect_one()) {
          mbar_arrive_expect_tx(a_full + 8 * sa, nt * 128);
          tma_load_act_rows(dst, &amap, 2 * blk * kUnitRows, row0, a_full + 8 * sa);
        }
        __syncwarp();
        if (n >= 2) mbar_wait_bounded<100>(done + 8 * ((n - 2) % R), ((n - 2) / R) & 1, p.status, dead);
        if (elect_one()) {
          mbar_arrive_expect_tx(a_full + 8 * (sa + 1), nt * 128);
          tma_load_act_rows(dst + C::kActUnitBytes, &amap, (2 * blk + 1) * kUnitRows, row0, a_full + 8 * (sa + 1));
        }
        __syncwarp();
        if (++blk == kb) { blk = 0; ++v; }
      }
    }
  } else if (warp == 2) {
    // ================================================================== MMA issuer
    // One thread, so that the commits track its MMAs; the warp stays together around it (elect_one), with as little between
    // the MMAs as possible: this warp was the kernel's serial chain (1741 cycles per segment at K = N = 16384, of which the
    // tensor pipe needs 1024).
    {
      // every bounded wait below depends on the activations, which the previous kernel of the stream may still be
      // writing: start them only when it has completed
      grid_dependency_wait();
      constexpr uint32_t kStepDesc = 32 >> 4;          // 16 halves along a 128-byte row
      const uint64_t desc0 = wide_act_desc(smem_u32(act_base));
      const uint32_t d_tmem = tmem + C::kTmemD;
      const uint32_t idesc = (1u << 4) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      int blk = B0 % kb, r = 0;
      uint32_t rphase = 0, accumulate = 0, slices = 0;
      for (int n = 0; n < nseg; ++n) {
        const int sa = 2 * (n & 1);
        const uint32_t aphase = (n >> 1) & 1;
        mbar_wait_bounded<20>(ready + 8 * r, rphase, p.status, dead);
        if (!accumulate && slices > 0) mbar_wait_bounded<20>(d_read, (slices - 1) & 1, p.status, dead);   // previous slice was read back
        mbar_wait_bounded<20>(a_full + 8 * sa, aphase, p.status, dead);
        tc_fence_after();
        // the descriptor's low 14 bits hold the address / 16: adding an offset never carries out of them
        const uint64_t desc = desc0 + (uint64_t)(sa * (C::kActUnitBytes >> 4));
        const uint32_t a_tmem = tmem + C::kTmemA + r * 64;
        if (elect_one()) {
          tc_mma_unit<kStepDesc>(d_tmem, a_tmem, desc, idesc, accumulate);
          tc_commit(a_empty + 8 * (n & 1));             // unit 0's stage may be refilled when these MMAs are done
        }
        __syncwarp();
        mbar_wait_bounded<20>(a_full + 8 * (sa + 1), aphase, p.status, dead);
        tc_fence_after();
        const bool slice_ends = ++blk == kb || n + 1 == nseg;
        if (elect_one()) {
          tc_mma_unit<kStepDesc>(d_tmem, a_tmem + 32, desc + (uint64_t)(C::kActUnitBytes >> 4), idesc, 1u);
          tc_commit(done + 8 * r);                      // unit 1's stage and the operand slot are free then
          if (slice_ends) tc_commit(slice_done);
        }
        __syncwarp();
        accumulate = 1;
        if (slice_ends) {
          blk = 0;
          accumulate = 0;
          ++slices;
        }
        if (++r == R) { r = 0; rphase ^= 1; }
      }
    }
  } else if (warp == 3) {
    // ================================================================== launch epoch
    if (lane == 0) {
      // the tag of this launch's split-K partials is epoch + 1
      grid_dependency_wait();
      misc[1] = read_epoch_and_count(p.epochs, gridDim.x);
      mbar_arrive(epoch_bar);
    }
  } else if (warp >= C::kDeqBase) {
    // ================================================================== dequantisers (warps kDeqBase..)
    // thread = weight column = TMEM lane; team t expands the segments n = t, t + T, ... of the CTA
    // and writes out its half (in multiples of 16 rows) of every slice's accumulator tile
    constexpr int CH = C::kChunk;
    const int team = (warp - C::kDeqBase) >> 2;
    const int quarter = warp & 3;                    // the TMEM lanes this warp may touch
    const int c = quarter * 32 + lane;               // weight column inside the strip
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    grid_dependency_wait();                          // the waits below depend, through the MMAs, on the previous kernel's output
    const uint32_t a_base = lane_base + C::kTmemA;
    const uint32_t lds_lo = c * 32 + 16 * ((c >> 2) & 1);          // words 0..3 of the column; words 4..7 at ^ 16
    const int strip_first = B0 / kb;
    const int team0_rows = (nt / 2 + CH - 1) / CH * CH;
    const int row0 = team == 0 ? 0 : team0_rows, team_rows = team == 0 ? team0_rows : nt - team0_rows;     // both > 0: nt >= 48
    const uint32_t d_base = lane_base + C::kTmemD + row0;

    struct Slice {
      int strip_lin, strip, tile_row0;      // strip_lin: the VIRTUAL strip (row tile x strip)
      bool is6, group;
    };
    auto open_slice = [&](int strip_lin) {
      Slice sl;
      const int real = strip_lin % nstrips;
      sl.strip_lin = strip_lin;
      sl.tile_row0 = (strip_lin / nstrips) * nt;
      sl.is6 = real >= geo.strips4;
      sl.strip = sl.is6 ? real - geo.strips4 : real;
      sl.group = !sl.is6 && geo.groups > 1;
      return sl;
    };
    auto column_scale = [&](const Slice& sl, bool writes) {
      float col_scale = 1.f;      // per-channel INT4: s; FP6: s * 4096; group INT4: already in the operands
      if (writes && !sl.group) {
        const half* sp = p.S + (sl.is6 ? fp6_scale_offset(geo, sl.strip) : int4_scale_offset(geo, sl.strip, 0));
        col_scale = __half2float(__ldg(sp + c)) * (sl.is6 ? 4096.f : 1.f);
      }
      return col_scale;
    };
    // Only the first slice of a CTA can start inside a strip, so a CTA has one partial.
    auto slot_of = [&](int cc) { return p.partials + (size_t)cc * C::kSlotWords + row0 * kStripCols + c; };
    // CH finished rows of this thread's column.  Plain path: one 2-byte store per value (a warp writes 64
    // bytes of a row).  With p.vec_rows the team turns the CH x 128 block round through shared memory and
    // every thread stores 16 bytes of a row - to C, or to every rank's output over NVLink, where the size of
    // a write matters most.  All 128 threads of the team call this together.
    const uint32_t my_stage = smem_u32(out_stage) + team * C::kOutStageBytes;
    const int team_tid = (warp - C::kDeqBase - 4 * team) * 32 + lane;
    int stage_turn = 0;                                // which of the team's two buffers the next block of rows uses
    auto store_rows = [&](const Slice& sl, int m0, const float (&v)[CH], float col_scale, bool writes) {
      float out[CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) out[i] = v[i] * col_scale;
      if (!p.vec_rows) {
        store_column_rows<CH>(p, sl.tile_row0 + row0 + m0, sl.is6, sl.strip * kStripCols + c, out, writes);
        return;
      }
      const int row_first = sl.tile_row0 + row0 + m0;
      if (row_first >= p.M) return;                    // nothing of the block exists (uniform over the team): it takes no turn
      const uint32_t buf = my_stage + (uint32_t)(stage_turn & 1) * (16 * kStripCols * 2);
      ++stage_turn;
      // The copy engine has read the rows this buffer held two turns ago: team thread 0 commits exactly one group per turn,
      // empty when the rows leave by ordinary stores, so all groups but the latest include that turn's.
      if (team_tid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      named_bar_sync(1 + team, 128);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const unsigned short hbits = __half_as_ushort(__float2half_rn(out[i]));
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(buf + (uint32_t)(i * kStripCols + c) * 2), "h"(hbits) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the copy engine reads what this thread wrote
      named_bar_sync(1 + team, 128);
      const int ncols = strip_cols(sl.is6 ? geo.n6 : geo.n4, sl.strip);
      const int col_strip = (p.out.n_out == 0 ? (sl.is6 ? geo.n4 : 0) : (sl.is6 ? p.out.col6 : p.out.col4)) + sl.strip * kStripCols;
      // a full strip: one asynchronous tensor store per output; the team goes on at once
      const bool tensor_store = p.vec_rows == 2 && ncols == kStripCols;
      if (team_tid == 0) {
        if (tensor_store) {
          const int n_maps = p.out.n_out == 0 ? 1 : p.out.n_out;
#pragma unroll 1
          for (int q = 0; q < n_maps; ++q) tma_store_rows(&omaps.m[q], buf, col_strip, row_first);
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      if (tensor_store) return;
      const int g = team_tid & 15;                     // eight columns of the strip
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int i = (team_tid >> 4) + 8 * rr;
        const int row = row_first + i;
        if (row < p.M && g * 8 < ncols) {
          uint4 val;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w)
                       : "r"(buf + (uint32_t)(i * kStripCols + g * 8) * 2));
          if (p.out.n_out == 0) {
            *reinterpret_cast<uint4*>(p.C + (size_t)row * p.N + col_strip + g * 8) = val;
          } else {
            const size_t at = (size_t)row * p.out.ld + col_strip + g * 8;
#pragma unroll 1
            for (int q = 0; q < p.out.n_out; ++q) *reinterpret_cast<uint4*>(p.out.peer[q] + at) = val;
          }
        }
      }
      // (the buffer is not written again before the barrier at the top of the next turn)
    };
    // before the team leaves: its asynchronous stores have been performed
    auto drain_stores = [&]() {
      if (team_tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    };

    // Writes out the slice of virtual strip `v` (this team's rows).  A slice that starts inside its strip leaves as a tagged
    // partial.  The CTA in which a strip starts sums it: that slice is its last one, its own sums come straight from the
    // accumulator tile, and the CTA behind it has normally stored its partial long ago (its first slice).
    auto finish_slice = [&](int v, int slices) {
      const Slice sl = open_slice(v);
      mbar_wait_bounded(slice_done, slices & 1, p.status, dead);
      tc_fence_after();
      const bool starts = v * kb >= B0;
      const bool writes = c < strip_cols(sl.is6 ? geo.n6 : geo.n4, sl.strip);
      const float col_scale = starts ? column_scale(sl, writes) : 1.f;
      uint32_t tag = 0;
      if (!starts || (v + 1) * kb > B1) {
        mbar_wait_bounded(epoch_bar, 0, p.status, dead);   // completed long ago: orders the read of misc[1]
        tag = misc[1] + 1;
      }
      unsigned long long* slot = slot_of(cta);
#pragma unroll 1
      for (int m0 = 0; m0 < team_rows; m0 += CH) {
        float t[CH];
        tc_ld16(d_base + m0, t);
        if (m0 + CH == team_rows) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(d_read);          // this warp has read its part: with the others', the issuer may start the next slice
        }
        if (!starts) {
#pragma unroll
          for (int i = 0; i < CH; ++i)
            st_relaxed_u64(slot + (m0 + i) * kStripCols, ((unsigned long long)tag << 32) | __float_as_uint(t[i]));
          continue;
        }
        // the partials of the CTAs behind this one, two per round trip to L2 (32 tagged words in flight per thread), added
        // in the order of the ranges
#pragma unroll 1
        for (int cc = cta + 1; cc < (int)gridDim.x && (p.sched.bound[cc] >> 1) < (v + 1) * kb; cc += 2) {
          // a CTA without work stored nothing; at least one of the two did store, and stands in for the other
          const int next = cc + 1 < (int)gridDim.x ? cc + 1 : cc;
          const bool live0 = p.sched.bound[cc] < p.sched.bound[cc + 1];
          const bool live1 = next != cc && p.sched.bound[next] < p.sched.bound[next + 1] && (p.sched.bound[next] >> 1) < (v + 1) * kb;
          if (!live0 && !live1) continue;
          const unsigned long long* src0 = slot_of(live0 ? cc : next) + m0 * kStripCols;
          const unsigned long long* src1 = slot_of(live1 ? next : cc) + m0 * kStripCols;
          unsigned long long v0[CH], v1[CH];
          bool all_here = false;
#pragma unroll 1
          for (int spin = 0; spin < (1 << 20) && !all_here; ++spin) {
#pragma unroll
            for (int i = 0; i < CH; ++i) v0[i] = ld_relaxed_u64(src0 + i * kStripCols);
            if (live0 && live1) {
#pragma unroll
              for (int i = 0; i < CH; ++i) v1[i] = ld_relaxed_u64(src1 + i * kStripCols);
            } else {
#pragma unroll
              for (int i = 0; i < CH; ++i) v1[i] = v0[i];
            }
            all_here = true;
#pragma unroll
            for (int i = 0; i < CH; ++i)
              all_here = all_here && (uint32_t)(v0[i] >> 32) == tag && (uint32_t)(v1[i] >> 32) == tag;
            if (dead) break;
          }
          if (!all_here && !dead) {
            dead = true;
            if (p.status) atomicExch(p.status, kStatusTimeout);
          }
#pragma unroll
          for (int i = 0; i < CH; ++i) {
            t[i] += __uint_as_float((uint32_t)v0[i]);
            t[i] += live0 && live1 ? __uint_as_float((uint32_t)v1[i]) : 0.f;
          }
        }
        store_rows(sl, m0, t, col_scale, writes);
      }
    };

    // The team expands its segments n = team, team + T, ... and writes the finished slices out.  A slice is not written out
    // when its last segment has been expanded - its MMAs are up to R segments behind - but when the team needs an operand
    // slot that only MMAs of the next slice can free, which wait for the accumulator tile: by then the slice has
    // normally been summed, and the operands of the next slice's first R segments wait in tensor memory.
    struct Strip {
      int n_begin, n_end;            // its segments (of the CTA): [n_begin, n_end), its first block's segment (may be negative)
      bool is6, group, scaled;
      uint32_t unit_bytes, two_off;
      int scale_stride;
      const half* scale0;            // this column's scale of the strip's first block
    };
    auto open_strip = [&](int v) {
      Strip sp;
      const Slice sl = open_slice(v);
      const int nq = strip_quads(sl.is6 ? geo.n6 : geo.n4, sl.strip);
      sp.n_begin = v * kb - B0;
      sp.n_end = min(nseg, sp.n_begin + kb);
      sp.is6 = sl.is6;
      sp.group = sl.group;
      sp.unit_bytes = nq * (sl.is6 ? kFp6UnitQuadBytes : kInt4UnitQuadBytes);
      sp.two_off = nq * kInt4UnitQuadBytes + c * 16;
      sp.scale_stride = nq * kQuadCols;
      sp.scaled = sl.group && c < nq * kQuadCols;      // padded quads of a ragged strip hold no data
      sp.scale0 = p.S + (sl.group ? int4_scale_offset(geo, sl.strip, 0) + c : 0);
      return sp;
    };
    auto block_scale = [&](const Strip& sp, int n) {
      return sp.scaled ? __ldg(sp.scale0 + (size_t)(n - sp.n_begin) * sp.scale_stride) : __float2half(1.f);
    };

    int v = strip_first;                             // the virtual strip of segment n
    Strip sp = open_strip(v);
    int fin_v = v, fin_end = sp.n_end, slices = 0;   // the first slice that has not been written out, its last segment + 1
    auto finish_next = [&]() {
      finish_slice(fin_v, slices);
      ++slices;
      ++fin_v;
      fin_end = min(nseg, fin_end + kb);
    };
    int stage = team, r = team;
    uint32_t wphase = 0, rphase = 0;
    while (team >= sp.n_end && sp.n_end < nseg) sp = open_strip(++v);
    half next_scale = team < nseg ? block_scale(sp, team) : __float2half(1.f);
#pragma unroll 1
    for (int n = team; n < nseg; n += T) {
      while (fin_end + R <= n) finish_next();
      const half2 s2 = __half2half2(next_scale);
      const bool is6 = sp.is6, group = sp.group;
      const uint32_t unit_bytes = sp.unit_bytes, two_off = sp.two_off;
      if (n + T < nseg) {                              // the next segment's strip and scale, used one iteration later
        while (n + T >= sp.n_end) sp = open_strip(++v);
        next_scale = block_scale(sp, n + T);
      }
      mbar_wait_bounded(w_full + 8 * stage, wphase, p.status, dead);
      const uint8_t* st = smem + stage * kStageW;
      // the MMAs that read this operand slot R segments ago have finished
      mbar_wait_bounded(done + 8 * r, rphase ^ 1, p.status, dead);
      tc_fence_after();
      const uint32_t a_tmem = a_base + r * 64;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        // Columns of padded quads read stale bytes of the stage and produce values nobody stores.
        const uint8_t* su = st + h * unit_bytes;
        const uint4 lo = *reinterpret_cast<const uint4*>(su + lds_lo);          // words 0..3
        const uint4 hi = *reinterpret_cast<const uint4*>(su + (lds_lo ^ 16));   // words 4..7
        uint4 two = make_uint4(0, 0, 0, 0);
        if (is6) two = *reinterpret_cast<const uint4*>(su + two_off);
        const uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        const uint32_t twos[4] = {two.x, two.y, two.z, two.w};
#pragma unroll
        for (int step = 0; step < 4; ++step) {
          uint32_t regs[8];
          if (is6) {
            expand_fp6(words[2 * step], twos[step], 0, regs);
            expand_fp6(words[2 * step + 1], twos[step], 4, regs + 4);
          } else if (group) {
            expand_int4_scaled(words[2 * step], s2, regs);
            expand_int4_scaled(words[2 * step + 1], s2, regs + 4);
          } else {
            expand_int4(words[2 * step], regs);
            expand_int4(words[2 * step + 1], regs + 4);
          }
          tc_st8(a_tmem + h * 32 + step * 8, regs);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(w_empty + 8 * stage);          // the stage's words are in registers
      tc_wait_st();
      tc_fence_before();
      if (lane == 0) mbar_arrive(ready + 8 * r);
      stage += T;
      if (stage >= S) { stage -= S; wphase ^= 1; }
      r += T;
      if (r >= R) { r -= R; rphase ^= 1; }
    }
    const int slices_all = (B1 - 1) / kb - strip_first + 1;
    while (slices < slices_all) finish_next();

    drain_stores();
  }

  // ---- all roles are done with tensor memory: give it back
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kTmemCols) : "memory");
  }
}

using Wide256 = WideCfg<kWideTileRows, 2, 4, 4>;    // 256 + 4 x 64 = 512 TMEM columns

template <class C>
cudaError_t launch_wide(const MulParams& p_in, cudaStream_t stream, bool overlap) {
  alignas(64) CUtensorMap amap;
  cudaError_t me = encode_activation_map(p_in.A, p_in.M, p_in.K, p_in.tile_rows, &amap);
  if (me != cudaSuccess) return me;
  MulParams p = p_in;
  alignas(64) OutMaps omaps = {};
  if (p.vec_rows) {
    // asynchronous tensor stores of the finished rows: one map per output; without them the 16-byte stores stay
    bool ok = true;
    if (p.out.n_out == 0) {
      ok = encode_output_map(p.C, p.M, p.N, &omaps.m[0]) == cudaSuccess;
    } else {
      for (int q = 0; q < p.out.n_out && ok; ++q) ok = encode_output_map(p.out.peer[q], p.M, p.out.ld, &omaps.m[q]) == cudaSuccess;
    }
    if (ok) p.vec_rows = 2;
  }

  static std::atomic<bool> configured[64] = {};       // threads that find it false set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(w46_gemm_wide_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.sched.ctas);
  cfg.blockDim = dim3(C::kThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, w46_gemm_wide_kernel<C>, p, amap, omaps);
}

}  // namespace

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up once through the runtime (no link against libcuda).  Several threads may make
// the first call: the others wait for the one that looks it up.
static EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &res) != cudaSuccess || res != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(sym);
  }();
  return fn;
}

// A map of fp16 data whose elements outside read as zero.  The encoder is a driver call and needs a current context, which a
// thread that has made no other CUDA call does not have: cudaGetDevice binds none, so the first attempt fails there.
static cudaError_t encode_f16(CUtensorMap* map, int rank, const half* base, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                              CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return cudaErrorNotSupported;
  const cuuint32_t elem[3] = {1, 1, 1};
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, const_cast<half*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
      return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaSetDevice(dev);       // binds the device's primary context to the thread
    if (e != cudaSuccess) return e;
  }
  return cudaErrorInvalidValue;
}

// The last few tensor maps of the calling thread: a decode loop calls with the same activation buffer again
// and again, and encoding a map costs a driver call.  (A map depends on the pointer and the shape only.)
namespace {
struct MapKey {
  const void* A;
  int M, K, box_rows, dims;
};
struct MapCache {
  static constexpr int kEntries = 96;      // a GEMM of many launches onto eight outputs has 64 output maps
  MapKey key[kEntries] = {};
  CUtensorMap map[kEntries];
  int next = 0;
  bool find(const MapKey& k, CUtensorMap* out) const {
    for (int i = 0; i < kEntries; ++i)
      if (key[i].A == k.A && key[i].M == k.M && key[i].K == k.K && key[i].box_rows == k.box_rows && key[i].dims == k.dims) {
        *out = map[i];
        return true;
      }
    return false;
  }
  void put(const MapKey& k, const CUtensorMap& m) {
    key[next] = k;
    map[next] = m;
    next = (next + 1) % kEntries;
  }
};
thread_local MapCache g_map_cache;
}  // namespace

// A as a K x M tensor (K contiguous): one box = 64 halves x `box_rows` rows = the activations of one
// 64-row unit, written to shared memory with the 128-byte swizzle; rows beyond M read as zero.
cudaError_t encode_activation_map(const half* A, int M, int K, int box_rows, CUtensorMap* map) {
  const MapKey mk = {A, M, K, box_rows, 2};
  if (g_map_cache.find(mk, map)) return cudaSuccess;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cudaError_t e = encode_f16(map, 2, A, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  if (e == cudaSuccess) g_map_cache.put(mk, *map);
  return e;
}

// An output (C, or a rank's full-width output) as an `ld` x `rows` fp16 tensor; one box = 128 columns x 16 rows,
// row-major in shared memory (no swizzle).  Stores beyond the last row are clipped.
cudaError_t encode_output_map(const half* base, int rows, int ld, CUtensorMap* map) {
  const MapKey mk = {base, rows, ld, 16, 4};
  if (g_map_cache.find(mk, map)) return cudaSuccess;
  const cuuint64_t dims[2] = {(cuuint64_t)ld, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kStripCols, 16};
  const cudaError_t e = encode_f16(map, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
  if (e == cudaSuccess) g_map_cache.put(mk, *map);
  return e;
}

// A as a 64 x M x K/64 tensor (K a multiple of 64): one box = 64 halves x `box_rows` rows x 2 units = the
// activations of one 128-row block as two swizzled tiles, one behind the other; units beyond K and rows
// beyond M read as zero.
cudaError_t encode_activation_segment_map(const half* A, int M, int K, int box_rows, CUtensorMap* map) {
  const MapKey mk = {A, M, K, box_rows, 3};
  if (g_map_cache.find(mk, map)) return cudaSuccess;
  const cuuint64_t dims[3] = {64, (cuuint64_t)M, (cuuint64_t)(K / 64)};
  const cuuint64_t strides[2] = {(cuuint64_t)K * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 2};
  const cudaError_t e = encode_f16(map, 3, A, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  if (e == cudaSuccess) g_map_cache.put(mk, *map);
  return e;
}

static int tile_height(int rows, int tiles) { return ((rows + tiles - 1) / tiles + 15) / 16 * 16; }

// `rows` (> 128) rows of A go into tiles of one height, a multiple of 16: as few as hold them, and more where strips
// would otherwise be shared by several of the `ctas` CTAs.  Another tile dequantises all weights once more, but leaves
// fewer and lower partial tiles to exchange.  It pays up to 14 blocks per CTA, or up to 38 when the tiles stay high enough
// (112 rows) for the MMAs to cover the dequantisers; measured on layers with one scale per column, us with n / n + 1 / n + 2 / n + 3
// tiles, n the fewest: 1024 x 4096 (1.7 blocks per CTA and tile) 256 rows 29 / 21 / 19 / 17, 512 rows 29 / 25 / 21 / 21; 4096 x 4096 (6.9) 129
// rows 29 / 24 / 25 / 29, 256 rows 42 / 27 / 28 / 29, 512 rows 40 / 35 / 33 / 39, 777 rows 39 / 43; 8192 x 4096 and 4096 x 8192 (13.8) 201 rows
// 54 / 41 / 43 and 39 / 33 / 41, 300 rows 42 / 49 and 400 rows 39 / 47; 11008 x 4096 (18.6) 201 rows 50 / 42 / 49, 256 rows 56 / 43 / 49, 300 rows
// 46 / 51; K = N = 8192 (28) 256 rows 52 / 50, 300 rows 53 / 68; 4096 x 22016 (37) 200 rows 50 / 66; 4096 x 12288, more than one strip per
// CTA with two tiles, 256 rows 42 / 45.
int wide_row_tiles(int rows, const Geometry& geo, int ctas) {
  const int strips = geo.strips4 + geo.strips6;
  int tiles = (rows + kWideTileRows - 1) / kWideTileRows;
  while (true) {
    const int more = tiles + 1, height = tile_height(rows, more);
    const long long blocks = (long long)more * strips * geo.k128;
    const bool pays = blocks <= 14ll * ctas || (height >= 112 && blocks <= 38ll * ctas);
    if (more > kMaxRowTiles || (long long)more * strips > ctas || height < 48 || !pays) return tiles;     // (both teams need rows)
    tiles = more;
  }
}
int wide_tile_rows(int rows, int tiles) { return tile_height(rows, tiles); }

size_t wide_scratch_bytes(int ctas) {
  return kEpochWords * sizeof(unsigned int) + (size_t)ctas * kWideTileRows * kStripCols * sizeof(unsigned long long);
}

// Runs the GEMM for rows [0, p.M) in p.row_tiles tiles of p.tile_rows rows; the host dispatcher loops over larger M.
cudaError_t launch_gemm_wide(const MulParams& p, cudaStream_t stream) {
  const bool overlap = tc5_get_overlap();
  return launch_wide<Wide256>(p, stream, overlap);
}

}  // namespace fp6m
