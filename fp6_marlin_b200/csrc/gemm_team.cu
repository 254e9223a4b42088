// W(4&6)A16 GEMM for 9 to 32 rows of A on tcgen05: every dequantiser team reads back and sums its own segments.
//
// Same product and operands as gemm_tc5.cu (128 weight columns of a strip = M of the MMA and one TMEM lane each, the rows of A =
// N, the expanded weights are read from tensor memory), with fewer hand-overs.  A team of four warps takes every third segment:
// it expands a 64-row unit into its half of an operand slot, publishes it, expands the other unit, and while the team's issuer
// runs the eight MMAs of this segment it reads the sums of its segment before back from the other one of its two accumulator
// tiles, times the group scale in fp32, into registers.  So there are no epilogue warps, no ring of scales, no tiles to zero
// and no barrier between accumulator and team: program order does it.  One thread issues all MMAs of a tile, hence sums
// in one order and results that repeat bit for bit.
// What bounds it: the teams' instructions (expansion 144 per warp and segment, at half rate) and the waits between them: a segment costs 510
// cycles (from 4096 x 22016 to 8192 x 57344 at 16 rows), HBM needs 350 for it, the tensor pipe 75, the issuers 100.  Before the issuers used elect.sync (see elect_one) they needed 1400.
// Measured, us per GEMM in a chain of launches (256 FP6 columns, group scales, weights larger than L2), against the kernel with epilogue warps
// that served these sizes before, without / with launch overlap:
//   at 16 rows 4096 x 4096 8.85 / 7.7 -> 7.55 / 6.7, 4096 x 22016 17.9 / 17.7 -> 15.9 / 15.3, 11008 x 4096 12.9 / 12.8 -> 11.4 / 10.7, K = N = 8192
//   14.6 / 14.15 -> 13.2 / 12.6, 8192 x 57344 66.5 / 66.4 -> 56.7 / 56.4, 16384 x 1024 12.2 / 10.7 -> 10.5 / 9.6;
//   at 32 rows 4096 x 4096 10.3 / 9.2 -> 9.1 / 8.4, K = N = 8192 16.9 / 16.5 -> 14.85 / 14.5, 8192 x 57344 74.5 -> 61.8, 16384 x 1024 15.9 / 14.8 -> 14.3 / 13.3.
//   Four teams instead of three, on another GPU: 4096 x 4096 8.2 instead of 7.5, K = N = 8192 13.5 instead of 12.4, 8192 x 57344 59.1 instead of 54.4.
//
// A slice (the CTA's blocks of one strip) is finished when a team has expanded its first segment of the next one, so its last
// MMAs are done by then; the teams pool their sums through shared memory, and two of them write the rows out or leave them as a partial.  The
// CTA's last slice, if its strip goes on in other CTAs, is summed by two or four groups of warps (kSumGroups).  Roles: warps 0 and 1 weights (every second segment
// each), warp 2 tensor memory, activations and launch epoch, then one MMA issuer per team, then the teams.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "device_utils.cuh"
#include "fp6m_layout.h"
#include "gemm_params.h"
#include "tc5_common.cuh"

namespace fp6m {

namespace {

template <int NT_, int STAGES_, int TEAMS_, int SUM_GROUPS_>
struct TeamCfg {
  static constexpr int NT = NT_;                       // rows of A = N of the MMA
  static constexpr int T = TEAMS_;
  static constexpr int kStages = STAGES_;
  static_assert(kStages % T == 0, "a stage always belongs to the same team");
  // The two weights producers take every second segment, so with an odd number of stages a stage changes producer on each use, and
  // a producer waits for every second phase of w_empty only.  Its parity wait for segment n - S must not pass on the phase before,
  // so segment n - 2 S must have been read by then.  It has: this producer has waited for segment n - 2 T - S, which the same
  // team reads, in order, and which is not before n - 2 S.
  static_assert(2 * T <= kStages, "a weights producer's waits bound the phase of a stage");
  static_assert(kStages <= 32, "the first round of weight copies is issued by one lane per stage");
  static constexpr int kIssueBase = 3;                 // warps 0, 1: weights; 2: activations, TMEM, epoch; then one MMA issuer per team
  static constexpr int kTeamBase = (kIssueBase + T + 3) & ~3;
  static constexpr int kThreads = 32 * (kTeamBase + 4 * T);
  static constexpr int kTeamThreads = 128 * T;
  static constexpr int kActRing = 2 * T;               // activation tiles: two per team
  static constexpr int kActUnitBytes = NT * 128;
  static constexpr int kActBytes = 2 * kActUnitBytes;
  static constexpr int kPoolBytes = T * NT * kStripCols * 4;
  static constexpr int kNumBars = 2 * kStages + 2 * kActRing + 4 * T + 1;
  static constexpr int kSmemBytes = kStages * kStageW + kActRing * kActBytes + kPoolBytes + kNumBars * 8 + 64 + 1024;
  static constexpr int kTmemD = 0, kTmemA = 2 * T * NT;          // two accumulator tiles per team, then one operand slot of 64 columns per team
  static constexpr int kTmemUsed = kTmemA + T * 64;
  static constexpr int kTmemCols = kTmemUsed <= 256 ? 256 : 512;
  static_assert(kTmemUsed <= 512, "tensor memory has 512 columns");
  static constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  static constexpr int kOutTeams = T < 4 ? 2 : 4;      // teams that write finished rows
  static constexpr int kOutRows = NT / kOutTeams;
  // Groups of four warps that sum a strip which goes on in other CTAs, with their shares of the rows: 2 = the output teams, 4 = all teams
  // and the four warps before them (issuers that are done).  More groups mean fewer rows a thread and so more contributors in flight
  // per round trip to L2 (add_partials): with 16 rows four instead of two, with 32 rows two instead of one.  (Two with the sixteen rows a
  // thread of two groups spill: 8192 x 2048 at 32 rows 13.7 us, K = N = 8192 17.3 instead of 15.2.)  launch_gemm_team says which is when faster.
  static constexpr int kSumGroups = SUM_GROUPS_;
  static constexpr int kSumRows = NT / kSumGroups;
  static constexpr bool kSumHelpers = kSumGroups > T;
  static_assert(kSumGroups <= T + 1 && kTeamBase - 4 >= kIssueBase, "one group of helpers, and none of them a producer");
};

// the sums of the teams for the rows row0 ... of column c
template <class C, int RR>
__device__ __forceinline__ void pooled_sums(uint32_t pool, int row0, int c, float (&out)[RR]) {
#pragma unroll
  for (int m = 0; m < RR; ++m) {
    out[m] = 0.f;
#pragma unroll
    for (int e = 0; e < C::T; ++e) out[m] += lds_f32(pool + ((e * C::NT + row0 + m) * kStripCols + c) * 4);
  }
}

template <class C, bool EARLY>
__global__ void __launch_bounds__(C::kThreads, 1) w46_gemm_team_kernel(const __grid_constant__ MulParams p, const __grid_constant__ CUtensorMap amap) {
  constexpr int NT = C::NT, S = C::kStages, T = C::T;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;       // activation tiles first: 1024-byte boundaries
  const uint32_t act_base = smem0, w_base = act_base + C::kActRing * C::kActBytes;
  const uint32_t pool = w_base + S * kStageW;
  const uint32_t bars0 = pool + C::kPoolBytes;
  const uint32_t w_full = bars0, w_empty = w_full + 8 * S;
  const uint32_t act_full = w_empty + 8 * S, act_done = act_full + 8 * C::kActRing;
  const uint32_t ready = act_done + 8 * C::kActRing;          // [team][unit]: the unit's operands are in tensor memory
  const uint32_t freed = ready + 8 * 2 * T;                   // [team][unit]: its MMAs are done
  const uint32_t epoch_bar = freed + 8 * 2 * T;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_raw + (epoch_bar + 8 - smem_u32(smem_raw)));   // [0] TMEM base, [1] launch epoch

  const int tid = threadIdx.x, warp = uniform_warp_index(), lane = tid & 31;
  const int cta = gridDim.x - 1 - blockIdx.x;
  const Geometry& geo = p.geo;
  const int kb = geo.k128;
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

  // ---- set-up
  if (warp == 0) {
    if (lane < S) {
      mbar_init(w_full + 8 * lane, 1);
      mbar_init(w_empty + 8 * lane, 4);            // one lane of each warp of the team
      mbar_fence_init();
      if (lane < nseg) {
        int s = s_first, blk = blk_first + lane;
        while (blk >= kb) { blk -= kb; ++s; }
        const uint32_t bytes = segment_bytes(geo, s), sbytes = segment_scale_bytes(geo, s);
        const uint8_t* src = p.B + segment_offset(geo, s, blk);
        const half* ssrc = p.S + (sbytes ? int4_scale_offset(geo, s, blk) : 0);
        if (!p.weights_early) {
          tma_prefetch_l2(src, bytes, policy);
          if (sbytes) tma_prefetch_l2(ssrc, sbytes, policy);
          grid_dependency_wait();
        }
        mbar_arrive_expect_tx(w_full + 8 * lane, bytes + sbytes);
        tma_load_1d_stream(w_base + lane * kStageW, src, bytes, w_full + 8 * lane, policy);
        if (sbytes) tma_load_1d_stream(w_base + lane * kStageW + kStageScaleOff, ssrc, sbytes, w_full + 8 * lane, policy);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane < C::kActRing) {
      mbar_init(act_full + 8 * lane, 1);
      mbar_init(act_done + 8 * lane, 1);
    }
    if (lane < 2 * T) {
      mbar_init(ready + 8 * lane, 4);              // one lane of each warp of the team
      mbar_init(freed + 8 * lane, 1);
    }
    if (lane == 0) mbar_init(epoch_bar, 1);
    mbar_fence_init();
    __syncwarp();
  } else if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(misc))), "r"(C::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, misc[0], 0);      // uniform to the compiler
  // With EARLY (p.expand_early) the teams go on: their first segments need the weights only.  An instance of its own, because as a
  // condition it costs the calls without it 0.03 us.
  if (!EARLY || warp < C::kTeamBase) grid_dependency_wait();

  if (warp < 2) {
    // ================================================================== weights producers: every other segment each
    int n = S + warp;
    if (n < nseg) {
      int s = s_first, blk = blk_first + n;
      while (blk >= kb) { blk -= kb; ++s; }
      const uint8_t* src = p.B + segment_offset(geo, s, blk);
      uint32_t bytes = segment_bytes(geo, s), sbytes = segment_scale_bytes(geo, s);
      const uint8_t* ssrc = reinterpret_cast<const uint8_t*>(p.S + (sbytes ? int4_scale_offset(geo, s, blk) : 0));
      int stage = n - S;
      uint32_t phase = 0;                      // parity of the stage's previous use
      for (; n < nseg; n += 2) {
        mbar_wait<200>(w_empty + 8 * stage, phase, ws);
        if (elect_one()) {
          mbar_arrive_expect_tx(w_full + 8 * stage, bytes + sbytes);
          tma_load_1d_stream(w_base + stage * kStageW, src, bytes, w_full + 8 * stage, policy);
          if (sbytes) tma_load_1d_stream(w_base + stage * kStageW + kStageScaleOff, ssrc, sbytes, w_full + 8 * stage, policy);
        }
        __syncwarp();
        src += 2 * bytes;
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
  } else if (warp == 2) {
    // ================================================================== activations producer; launch epoch
    // The host encoded the three-dimensional map.  (It does for every K that mul_impl lets through, multiples of 64; without the
    // other branch the 16-row instance measures slower: 8192 x 28672 at 9 rows 33.7 -> 34.2 us, 16384 x 1024 12.3 -> 12.45.)
    const bool act3d = (p.K & 63) == 0;
    int blk = blk_first, r = 0;
    uint32_t phase = 1;                        // a fresh barrier passes parity 1
    for (int n = 0; n < nseg; ++n) {
      mbar_wait<100>(act_done + 8 * r, phase, ws);       // the MMAs that read this tile are done
      if (elect_one()) {
        const uint32_t dst = act_base + r * C::kActBytes;
        mbar_arrive_expect_tx(act_full + 8 * r, C::kActBytes);
        if (act3d) {
          tma_load_act_segment(dst, &amap, 2 * blk, act_full + 8 * r);
        } else {
          tma_load_act(dst, &amap, 2 * blk * kUnitRows, act_full + 8 * r);
          tma_load_act(dst + C::kActUnitBytes, &amap, (2 * blk + 1) * kUnitRows, act_full + 8 * r);
        }
        if (n == min(nseg, C::kActRing) - 1) {
          misc[1] = read_epoch_and_count(p.epochs, gridDim.x);
          mbar_arrive(epoch_bar);
        }
      }
      __syncwarp();
      if (++blk == kb) blk = 0;
      if (++r == C::kActRing) { r = 0; phase ^= 1; }
    }
  } else if (warp >= C::kIssueBase && warp < C::kIssueBase + T) {
    // ================================================================== MMA issuers: the segments of one team each
    const int team = warp - C::kIssueBase;
    const uint32_t rd = ready + 16 * team, fr = freed + 16 * team;
    const uint32_t a_tmem = tmem + C::kTmemA + team * 64;
    const uint32_t d0 = tmem + C::kTmemD + team * 2 * NT;
    const uint64_t desc0 = wide_act_desc(act_base + team * C::kActBytes);
    constexpr uint64_t kTileStep = (uint64_t)(T * C::kActBytes) >> 4;       // from the team's first activation tile to its second
    constexpr uint32_t kStepDesc = 32 >> 4;            // 16 halves along a 128-byte row
    uint32_t i = 0;
    for (int n = team; n < nseg; n += T, ++i) {
      const uint32_t tile = i & 1;
      const int r = team + (tile ? T : 0);
      const uint64_t desc = desc0 + (tile ? kTileStep : 0);
      const uint32_t d = d0 + tile * NT;
      mbar_wait<32>(act_full + 8 * r, (i >> 1) & 1, ws);
      mbar_wait<32>(rd, i & 1, ws);
      tc_fence_after();
      if (elect_one()) {
        tc_mma_unit<kStepDesc>(d, a_tmem, desc, C::kIdesc, 0u);
        tc_commit(fr);
      }
      __syncwarp();
      mbar_wait<32>(rd + 8, i & 1, ws);
      tc_fence_after();
      if (elect_one()) {
        tc_mma_unit<kStepDesc>(d, a_tmem + 32, desc + (C::kActUnitBytes >> 4), C::kIdesc, 1u);
        tc_commit(act_done + 8 * r);
        tc_commit(fr + 8);
      }
      __syncwarp();
    }
  } else if (warp >= C::kTeamBase) {
    // ================================================================== teams: thread = weight column = TMEM lane
    const int team = (warp - C::kTeamBase) >> 2;
    const int quarter = warp & 3;
    const int c = quarter * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t a_tmem = lane_base + C::kTmemA + team * 64;
    const uint32_t d0 = lane_base + C::kTmemD + team * 2 * NT;
    const uint32_t rd = ready + 16 * team, fr = freed + 16 * team;
    const uint32_t lds_lo = c * 32 + 16 * ((c >> 2) & 1);          // words 0..3 of the column; words 4..7 at ^ 16
    const uint32_t lds_hi = lds_lo ^ 16;
    const int row0 = team * C::kOutRows;

    float acc[NT];
#pragma unroll
    for (int m = 0; m < NT; ++m) acc[m] = 0.f;

    int cur = s_first;                           // the strip whose slice `acc` belongs to
    // the slice of strip `cur` is complete in all teams: pool, then write it out, leave it as a partial or sum the strip
    auto finish = [&]() {
      const int s = cur;
      const bool is6 = s >= geo.strips4;
      const int strip = is6 ? s - geo.strips4 : s;
      const int b0 = s == s_first ? blk_first : 0;
      const int b1 = min(kb, B1 - s * kb);
      named_bar_sync(1, C::kTeamThreads);        // the sums of the slice before have been read
#pragma unroll
      for (int m = 0; m < NT; ++m) sts_f32(pool + ((team * NT + m) * kStripCols + c) * 4, acc[m]);
      if (C::kSumHelpers && b0 == 0 && b1 < kb) return;      // at the kernel's end, with the helpers
      named_bar_sync(1, C::kTeamThreads);
      if (team >= C::kOutTeams) return;
      constexpr int RR = C::kOutRows;
      float out[RR];
      pooled_sums<C>(pool, row0, c, out);
      uint32_t tag = 0;
      if (b0 > 0 || b1 < kb) {
        mbar_wait(epoch_bar, 0, ws);
        tag = misc[1] + 1;                           // launch epoch + 1
      }
      if (b0 > 0) {
        store_partial<RR>(p, cta, NT, row0, c, tag, out);
        return;
      }
      if (b1 < kb) add_partials<RR>(p, cta, (s + 1) * kb, NT, row0, c, tag, out, ws);
      finish_column_rows<RR>(p, row0, is6, strip, c, out);
    };
    auto add_sums = [&](uint32_t d, uint32_t scale_raw) {
      const float scale = __half2float(__ushort_as_half((unsigned short)scale_raw));
#pragma unroll
      for (int m0 = 0; m0 < NT; m0 += 16) {
        float v[16];
        tc_ld16(d + m0, v);
#pragma unroll
        for (int m = 0; m < 16; ++m) acc[m0 + m] = fmaf(scale, v[m], acc[m0 + m]);
      }
      tc_fence_before();
    };

    int s = s_first, stage = team;
    uint32_t i = 0, wphase = 0, scale_prev = 0;
    bool is6 = false, scaled = false;
    uint32_t unit_bytes = 0, two_off = 0;
    int n_end = 0;                               // first segment (of the CTA) beyond strip s; 0: strip s is not open
    --s;
#pragma unroll 1
    for (int n = team; n < nseg; n += T, ++i) {
      while (n >= n_end) {
        ++s;
        n_end = min(nseg, (s + 1) * kb - B0);
        is6 = s >= geo.strips4;
        const int nq = is6 ? strip_quads(geo.n6, s - geo.strips4) : strip_quads(geo.n4, s);
        unit_bytes = nq * (is6 ? kFp6UnitQuadBytes : kInt4UnitQuadBytes);
        two_off = nq * kInt4UnitQuadBytes + c * 16;
        scaled = !is6 && geo.groups > 1;
      }
      // Columns of padded quads read stale bytes of the stage and produce values nobody stores.
      const uint32_t st = w_base + stage * kStageW;
      mbar_wait(w_full + 8 * stage, wphase, ws);
      uint4 lo = lds128(st + lds_lo), hi = lds128(st + lds_hi), two = {};
      if (is6) two = lds128(st + two_off);
      mbar_wait(fr, (i & 1) ^ 1, ws);            // the MMAs of the team's segment before are done with this half of the slot
      tc_fence_after();
      if (is6) expand_words<true>(lo, hi, two, a_tmem);
      else expand_words<false>(lo, hi, two, a_tmem);
      lo = lds128(st + unit_bytes + lds_lo);
      hi = lds128(st + unit_bytes + lds_hi);
      if (is6) two = lds128(st + unit_bytes + two_off);
      const uint32_t scale_raw = scaled ? lds_u16(st + kStageScaleOff + 2 * c) : 0x3C00u;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(rd);
        mbar_arrive(w_empty + 8 * stage);
      }
      mbar_wait(fr + 8, (i & 1) ^ 1, ws);
      tc_fence_after();
      if (is6) expand_words<true>(lo, hi, two, a_tmem + 32);
      else expand_words<false>(lo, hi, two, a_tmem + 32);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(rd + 8);
      if constexpr (EARLY) grid_dependency_wait();       // before the first wait for an MMA, and before anything is written
      if (i > 0) add_sums(d0 + ((i - 1) & 1) * NT, scale_prev);
      while (cur < s) {
        finish();
#pragma unroll
        for (int m = 0; m < NT; ++m) acc[m] = 0.f;
        ++cur;
      }
      scale_prev = scale_raw;
      stage += T;
      if (stage >= S) { stage -= S; wphase ^= 1; }
    }
    if constexpr (EARLY) grid_dependency_wait();         // (a team without segments)
    if (i > 0) {
      mbar_wait(fr + 8, (i - 1) & 1, ws);
      tc_fence_after();
      add_sums(d0 + ((i - 1) & 1) * NT, scale_prev);
    }
    const int s_last = (B1 - 1) / kb;
    while (cur <= s_last) {
      finish();
#pragma unroll
      for (int m = 0; m < NT; ++m) acc[m] = 0.f;
      ++cur;
    }
  }
  if constexpr (C::kSumHelpers) {
    const int s = (B1 - 1) / kb;
    if (warp >= C::kTeamBase - 4 && (s > s_first || blk_first == 0) && B1 < (s + 1) * kb) {
      // the CTA's last strip starts here and goes on in the next CTA; the teams have left their sums of it in the pool
      named_bar_sync(2, C::kTeamThreads + 128);
      const int group = warp >= C::kTeamBase ? (warp - C::kTeamBase) >> 2 : T;
      constexpr int RR = C::kSumRows;
      const int row0 = group * RR, c = (warp & 3) * 32 + lane;
      const bool is6 = s >= geo.strips4;
      const int strip = is6 ? s - geo.strips4 : s;
      float out[RR];
      pooled_sums<C>(pool, row0, c, out);
      mbar_wait(epoch_bar, 0, ws);
      add_partials<RR>(p, cta, (s + 1) * kb, NT, row0, c, misc[1] + 1, out, ws);
      finish_column_rows<RR>(p, row0, is6, strip, c, out);
    }
  }
  report_waits(ws, p.status);
  // ---- all roles are done with tensor memory: give it back
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kTmemCols) : "memory");
  }
}

using Team16 = TeamCfg<16, 12, 3, 2>;
using Team16Cut = TeamCfg<16, 12, 3, 4>;
using Team32 = TeamCfg<32, 9, 3, 2>;
using Team32Cut = TeamCfg<32, 9, 3, 4>;

template <class C, bool EARLY>
cudaError_t launch_instance(const MulParams& p, cudaStream_t stream) {
  static std::atomic<bool> configured[64] = {};       // threads that find it false set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(w46_gemm_team_kernel<C, EARLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
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
  cfg.numAttrs = 1;
  alignas(64) CUtensorMap amap;
  cudaError_t me = (p.K & 63) == 0 ? encode_activation_segment_map(p.A, p.M, p.K, C::NT, &amap)
                                   : encode_activation_map(p.A, p.M, p.K, C::NT, &amap);
  if (me != cudaSuccess) return me;
  return cudaLaunchKernelEx(&cfg, w46_gemm_team_kernel<C, EARLY>, p, amap);
}

template <class C>
cudaError_t launch_team(const MulParams& p, cudaStream_t stream) {
  return p.expand_early ? launch_instance<C, true>(p, stream) : launch_instance<C, false>(p, stream);
}

}  // namespace

cudaError_t launch_gemm_team(const MulParams& p, cudaStream_t stream) {
  // Four groups pay where strips are cut over many CTAs.  Up to 16 rows that is at least four on average (us at 16 rows, two groups -> four:
  // sixteen CTAs per strip 16384 x 1024 12.2 -> 10.5, nine 11008 x 2048 10.1 -> 9.5, eight 8192 x 2048 9.2 -> 8.8, four 4096 x 1024 7.70 -> 7.65
  // and 4096 x 4096 equal, but 2.3 K = N = 8192 13.3 -> 13.6, 1.5 4096 x 12288 11.4 -> 11.9, one 1024 x 1024 6.4 -> 6.7); up to 32 rows more than
  // one (at 32 rows sixteen 18.3 -> 14.2, eight 12.7 -> 10.8, four 9.6 -> 9.0 and 9.9 -> 9.5, 2.3 15.2 -> 15.1, 1.5 13.0 -> 12.9, but one 7.39 -> 7.44
  // and 0.7 8192 x 28672 36.3 -> 36.5).
  const int ctas = p.sched.ctas, strips = p.geo.strips4 + p.geo.strips6;
  if (p.M > 16) return ctas > strips ? launch_team<Team32Cut>(p, stream) : launch_team<Team32>(p, stream);
  return ctas >= 4 * strips ? launch_team<Team16Cut>(p, stream) : launch_team<Team16>(p, stream);
}

}  // namespace fp6m
