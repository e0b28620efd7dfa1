// Tensor-core path: y^T[n, m] = W[n, :] . x[m, :] with the WEIGHT rows as the UMMA M dimension
// (128) and the activation batch as the UMMA N dimension (16..256), so that even a single
// activation row fills the 5th-generation tensor core.  No counterpart in the reference, whose
// kernels are CUDA-core GEMVs only (qfactory/include/gptq_gemv.h:14-154).
//
// Data flow of one CTA (one 128-row weight tile x one batch tile x one K split), in stages
// of 128 k:
//
//   TMA (2 threads)   packed weights (one contiguous bulk copy per stage) and the fp16
//                     activation tile (two 128-byte-swizzled tensor boxes) -> two independent
//                     shared-memory rings; the weight ring is released by the decode warps as
//                     soon as the codes are in registers, the activation ring by MMA completion
//   decode (8 or 16 warps)  packed codes -> exact (q - z) fp16 pairs in registers (LOP3 / PRMT magic
//                     numbers) -> tcgen05.st into TENSOR MEMORY as the A operand.  The fp16
//                     weights never touch shared memory, whose bandwidth could not carry the
//                     4x-expanded stream at HBM rate.  Thread (row, half) owns 64 codes of a stage.
//   MMA (1-2 threads) tcgen05.mma kind::f16, A from tensor memory, B (activations) from shared
//                     memory, fp32 accumulators in tensor memory.  ONE tcgen05.commit per stage
//                     feeds every consumer of "stage done".  With per-stage accumulators (POST)
//                     two threads issue alternate stages, since a skinny MMA costs more to issue
//                     than to execute.
//   scale (4 warps)   POST mode (small batches): one accumulator per quantisation group; the
//                     group's fp32 partial is read back with tcgen05.ld and folded into register
//                     accumulators with ONE fp32 FMA by the row's scale, so the decode needs a
//                     single fp16 instruction per code pair.  PRE mode (large batches): the
//                     decode multiplies by the scale and one accumulator spans all of K.
//
// Every mbarrier wait is bounded: on a time-out the CTA raises a flag, all roles drain, tensor
// memory is released and a status word is written for the host.
#include "qfb_common.cuh"
#include "qfb_kernels.h"
#include "qfb_ptx.cuh"
#include "qfb_tc_stage.cuh"

namespace qfb {

using namespace ptx;

// DG = decode groups: 1 -> 8 decode warps (512 threads, two CTAs per SM for the smallest batch
// tile), 2 -> two groups of 8 decode warps that take alternate stages (768 threads, one CTA per SM).
template <int BITS, int NB, bool POST, int DG>
struct TcCfg {
  static constexpr int kThreads = 128 + 256 * DG + 128;
  static constexpr int kScaleWarp0 = 4 + 8 * DG;
  static constexpr int kWBytes = 128 * kStageK * BITS / 8;
  static constexpr int kXBytes = NB * kStageK * 2;
  static constexpr int kZSlot = 256;   // effective zeros of a stage: 128 rows x up to 2 groups
  static constexpr int kSSlot = 512;   // fp16 scales of a stage (PRE mode only)
  static constexpr int kQBytes = kZSlot + (POST ? 0 : kSSlot);
  // two CTAs share an SM (98 KB of shared memory, 256 tensor-memory columns, 64 registers each):
  // the narrow per-stage-accumulator tiles, and with one decode group the scale-in-the-decode tiles
  // up to 128 columns (two independent pipelines hide each other's hand-off latencies)
  static constexpr bool kTwoPerSM = DG == 1 && (POST ? NB <= 32 : NB <= 128);
  static constexpr int kBudget = kTwoPerSM ? 98 * 1024 : 224 * 1024;
  static constexpr int kXStages = (kTwoPerSM && !POST) ? (NB <= 32 ? 6 : NB <= 64 ? 3 : 2)
                                  : NB <= 16 ? 6 : NB <= 32 ? (POST ? 4 : 8) : NB <= 64 ? 6 : NB <= 128 ? 4 : (BITS == 8 ? 2 : 3);
  static constexpr int kWStagesRaw = (kBudget - kXStages * kXBytes) / (kWBytes + kQBytes);
  // with two decode groups an even number of slots: a wait on the parity of a full barrier is only sound for a thread
  // that knows the phase before the awaited one to be complete, and with an odd number the previous stage in a slot
  // belongs to the other group, whose bulk copy may land later than the copies after it (the wait then fell through
  // and the group decoded a slot that was still being filled)
  static constexpr int kWStagesCap = kWStagesRaw > 16 ? 16 : kWStagesRaw;
  static constexpr int kWStages = DG == 2 ? kWStagesCap & ~1 : kWStagesCap;
  static constexpr int kTmemCols = kTwoPerSM ? 256 : 512;
  // ring of R slots in tensor memory: A operand (64 columns) + in POST mode one accumulator each
  static constexpr int kSlotCols = kAColsPerSlot + (POST ? NB : 0);
  // PRE mode with skinny MMAs (N <= 128) is issue-bound too: two issuers, one accumulator each
  static constexpr int kIssuers = POST ? 2 : ((NB <= 128 && !(kTwoPerSM && NB > 64)) ? 2 : 1);
  static constexpr int kRingRaw = (kTmemCols - (POST ? 0 : kIssuers * NB)) / kSlotCols;
  static constexpr int kRingCap = kXStages < 6 ? kXStages : 6;   // never deeper than the activation ring
  static constexpr int kRing = kRingRaw > kRingCap ? kRingCap : kRingRaw;
  static constexpr int kDBase = kRing * kAColsPerSlot;
  // What the CTA works on is not kept through the roles for the results, but worked out again: where two CTAs share an SM
  // the decode loop needs every one of the 64 registers.  (28672,8192): 3 bits at 64 rows 95.8 -> 88.4 us, 4 bits at 128 rows
  // 71.2 -> 69.4; not at 64 columns with the smaller decoders (4 bits at 64 rows 62.0 -> 66.4: the results' code spills)
  // nor with one CTA per SM (no difference, and 1 us more where K is split).
  static constexpr bool kRederive = kTwoPerSM && !POST && (NB > 64 || BITS == 3);
  static constexpr size_t kSmemBytes = 1024 + (size_t)kXStages * kXBytes + (size_t)kWStages * (kWBytes + kQBytes);
  static_assert(kWStages >= 2, "weight ring too shallow");
  static_assert(kRing >= 2, "need at least two tensor-memory slots");
  static_assert(kDBase + (POST ? kRing * NB : kIssuers * NB) <= kTmemCols, "tensor memory over-subscribed");
};

// Sum of the split-K partials of one warp's 32 rows over all S splits, in split order, rounded to fp16 into y, for the
// tiles with per-stage accumulators.  part -> partial of split 0, batch column 0, the warp's first row; `sstride` floats
// between splits, `cstride` between batch columns (both multiples of 128); y -> y[first batch row][the warp's first
// output feature], `ystride` halfs between batch rows; `cols` valid batch columns, `rows` valid rows.
// A lane sums four rows of every fourth column: 16 columns of two splits, eight 16-byte loads a lane, are in flight per
// round.  With a row per lane and 32 loads of 4 bytes in flight this build's 64 registers did not suffice: it spilled and
// waited in between.  Measured, that -> this, (4096,11008), 9 splits: 16 rows (tile layout) 30.0 -> 15.8 us, 32 rows 31.2 ->
// 20.9; 8-bit (8192,8192) at 24 rows 27.6 -> 23.9 (launches one after the other from a graph).
template <int NB>
__device__ __forceinline__ void splitk_reduce(const float* part, uint32_t sstride, uint32_t cstride, int S, int cols, int rows,
                                              __half* y, size_t ystride, int lane) {
  // (opaque: from strides it knows to be products of launch constants the compiler precomputes more addresses than the
  // build has registers for)
  asm("" : "+r"(sstride), "+r"(cstride));
  const int r = (lane & 7) * 4, cg = lane >> 3;
  const bool vec = rows >= r + 4 && ystride % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 7u) == 0;
#pragma unroll 1
  for (int c0 = cg; c0 - cg < NB && c0 - cg < cols; c0 += 16) {
    float4 sum[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* b = part + (size_t)(c0 * cstride + r);
#pragma unroll 1
    for (int sp = 0; sp < S; sp += 2, b += 2 * (size_t)sstride) {
      float4 t[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          t[u][j] = (sp + u < S && c0 + 4 * j < cols) ? __ldcg(reinterpret_cast<const float4*>(b + u * sstride + 4 * j * cstride))
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (sp + u < S) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            sum[j].x += t[u][j].x;
            sum[j].y += t[u][j].y;
            sum[j].z += t[u][j].z;
            sum[j].w += t[u][j].w;
          }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = c0 + 4 * j;
      if (c >= cols) continue;
      __half* dst = y + (size_t)c * ystride + r;
      const __half2 lo = __floats2half2_rn(sum[j].x, sum[j].y), hi = __floats2half2_rn(sum[j].z, sum[j].w);
      if (vec) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(as_u32(lo), as_u32(hi));
      } else {
        if (r < rows) dst[0] = __low2half(lo);
        if (r + 1 < rows) dst[1] = __high2half(lo);
        if (r + 2 < rows) dst[2] = __low2half(hi);
        if (r + 3 < rows) dst[3] = __high2half(hi);
      }
    }
  }
}

// What a CTA works on.  Two grid shapes.  Uniform: grid (row tiles, batch tiles, K splits).  Tail-split (p.tail_split > 0,
// one-dimensional grid): the first p.full_units CTAs own a whole (row tile, batch tile) unit each,
// the remaining units (the last, partly filled wave of a launch) are cut into p.tail_split K ranges
// of one CTA each, so that the tail costs a fraction of a wave.
struct TcUnit {
  int tile, mtile, split, S;   // K range `split` of the unit's S
  int ctr;                     // index of the unit's arrival counters
  int tail;                    // >= 0: this CTA writes compact partials of tail unit `tail`
  int kb0, nkb;                // the range's first stage and how many it has
};
__device__ __forceinline__ TcUnit tc_unit(const TcParams& p, int cx, int cy, int cz) {
  TcUnit u;
  u.tile = cx;
  u.mtile = cy;
  u.split = cz;
  u.S = gridDim.z;
  u.ctr = cy * gridDim.x + cx;
  u.tail = -1;
  if (p.tail_split > 0) {
    int unit = cx;
    u.split = 0;
    u.S = 1;
    if (cx >= p.full_units) {
      const int j = cx - p.full_units;
      u.tail = j / p.tail_split;
      unit = p.full_units + u.tail;
      u.split = j - u.tail * p.tail_split;
      u.S = p.tail_split;
      u.ctr = u.tail;
    }
    u.tile = unit / p.mtiles;
    u.mtile = unit - u.tile * p.mtiles;
  }
  u.kb0 = (int)(((long long)u.split * p.kblocks) / u.S);
  u.nkb = (int)(((long long)(u.split + 1) * p.kblocks) / u.S) - u.kb0;
  return u;
}

// FRAG = the layer is in the fragment layout (a build of its own: with both decoders behind a run-time branch in
// the decode loop the compiler allots registers for the larger of the two)
// ASYM = the layer has scales AND zero points (the common case; a build of its own for the same reason; used
// where the scale is applied in the decode)
template <int BITS, int NB, bool POST, int DG, bool FRAG, bool ASYM>
__global__ void __launch_bounds__(TcCfg<BITS, NB, POST, DG>::kThreads, (TcCfg<BITS, NB, POST, DG>::kTwoPerSM ? 2 : 1))
qgemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const TcParams p) {
  using Cfg = TcCfg<BITS, NB, POST, DG>;
  constexpr int NS = Cfg::kWStages;   // weight ring
  constexpr int NX = Cfg::kXStages;   // activation ring
  constexpr int R = Cfg::kRing;       // tensor-memory slot ring

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_wfull[NS], bar_wempty[NS], bar_xfull[NX], bar_xempty[NX];
  __shared__ uint64_t bar_afull[R], bar_done[R], bar_dempty[R], bar_final;
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  __shared__ unsigned tail_seen[4];   // per 32 rows: K ranges that have arrived / this one is the last

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TcUnit unit = tc_unit(p, blockIdx.x, blockIdx.y, blockIdx.z);
  const int tile = unit.tile, mtile = unit.mtile, split = unit.split, S = unit.S, kb0 = unit.kb0, nkb = unit.nkb;

  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
  constexpr uint32_t x_off = 0;
  constexpr uint32_t w_off = NX * Cfg::kXBytes;
  constexpr uint32_t z_off = w_off + NS * Cfg::kWBytes;
  constexpr uint32_t s_off = z_off + NS * Cfg::kZSlot;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(smem_u32(&bar_wfull[i]), 1);
      mbar_init(smem_u32(&bar_wempty[i]), kDecodeWarps);  // the eight warps of the group that decodes the stage
    }
    for (int i = 0; i < NX; ++i) {
      mbar_init(smem_u32(&bar_xfull[i]), 1);
      mbar_init(smem_u32(&bar_xempty[i]), 1);
    }
    for (int i = 0; i < R; ++i) {
      mbar_init(smem_u32(&bar_afull[i]), kDecodeWarps);
      mbar_init(smem_u32(&bar_done[i]), 1);
      mbar_init(smem_u32(&bar_dempty[i]), 4);
    }
    mbar_init(smem_u32(&bar_final), Cfg::kIssuers);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(&tmem_holder), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  volatile int* abortp = &abort_flag;
  const long long wait_limit = p.stall_test ? 200000LL : kWaitLimitCycles;
  // Builds with two CTAs per SM let the next kernel in only when their stages are done: its CTAs would fill the slots this
  // grid leaves free, two on some SMs beside others with none, and stay there.  Launches in a row, at once -> late:
  // (12288,4096) at 24 rows, 96 CTAs, 29.5 -> 24.5 us; (25600,8192) at 33 rows, 252 CTAs, 61.2 -> 47.8; (28672,8192) at 64, 224
  // CTAs, 63.2 -> 62.0; with all slots taken no difference.  (A layer that reads early gains more from being in early.)
  if (p.early || !Cfg::kTwoPerSM) grid_launch_dependents();
  if (!p.early) grid_dependency_wait();

  const bool has_z = ASYM || p.qz != nullptr;
  const bool has_s = ASYM || p.qs != nullptr;

  if (warp == 0) {
    // ------------------------------ weight producer ---------------------------
    // (depends on the preceding kernel only where TcParams::early is not set: the wait above)
    if (lane == 0) {
      if constexpr (kSwizzledStage<BITS, FRAG, POST>) prefetch_tensormap(&tmap_w);
      const uint8_t* wsrc = reinterpret_cast<const uint8_t*>(p.qw) + (size_t)tile * p.k * (16 * BITS) + (size_t)kb0 * Cfg::kWBytes;
      int s = 0;
      uint32_t ph = 1;  // first pass over the ring: parity 1 of a fresh barrier passes at once
      // group of the stage's first 64 k, tracked without divisions in the loop
      const int hpg = p.halfstages_per_group;
      int g0 = (kb0 * 2) / hpg, gpos = (kb0 * 2) % hpg;
      const uint32_t ng = hpg == 1 ? 2u : 1u;
      const uint32_t zb = has_z ? ng * 128u : 0u, sb = (!POST && has_s) ? ng * 256u : 0u;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(smem_u32(&bar_wempty[s]), ph, abortp, kSleepProducer, wait_limit)) break;
        const uint32_t bar = smem_u32(&bar_wfull[s]);
        // (K an odd multiple of 64: the last stage is half a stage of codes, and one group of 64)
        const bool half = !FRAG && p.half_tail && kb0 + i == p.kblocks - 1;
        const uint32_t wb = half ? Cfg::kWBytes / 2 : Cfg::kWBytes;
        const uint32_t zn = half && hpg == 1 ? zb / 2 : zb, sn = half && hpg == 1 ? sb / 2 : sb;
        // zeros / scales of the groups this stage touches: one group, or two when the group is 64
        mbar_arrive_expect_tx(bar, wb + zn + sn + ((p.stall_test && i == 0) ? 16u : 0u));
        if constexpr (kSwizzledStage<BITS, FRAG, POST>) {
          // the stage is two runs: 8 k-steps (2 * BITS rows of 64 bytes each) of the upper and of the lower 64 rows
          const int r0 = (tile * 2 * p.kblocks + kb0 + i) * (16 * BITS);
          tma_tensor_2d_g2s(sbase + w_off + s * Cfg::kWBytes, &tmap_w, 0, r0, bar);
          tma_tensor_2d_g2s(sbase + w_off + s * Cfg::kWBytes + Cfg::kWBytes / 2, &tmap_w, 0, r0 + p.kblocks * (16 * BITS), bar);
        } else if (FRAG) {
          // the stage is two runs: 8 k-steps (128 * BITS bytes each) of the upper and of the lower 64 rows
          const uint8_t* f0 = reinterpret_cast<const uint8_t*>(p.qw) +
                              (((size_t)tile * 2) * (size_t)(p.kblocks * 8) + (size_t)(kb0 + i) * 8) * (128 * BITS);
          tma_bulk_g2s(sbase + w_off + s * Cfg::kWBytes, f0, Cfg::kWBytes / 2, bar);
          tma_bulk_g2s(sbase + w_off + s * Cfg::kWBytes + Cfg::kWBytes / 2,
                       f0 + (size_t)p.kblocks * 8 * (128 * BITS), Cfg::kWBytes / 2, bar);
        } else {
          tma_bulk_g2s(sbase + w_off + s * Cfg::kWBytes, wsrc + (size_t)i * Cfg::kWBytes, wb, bar);
        }
        if (zn) tma_bulk_g2s(sbase + z_off + s * Cfg::kZSlot, p.qz + ((size_t)tile * p.groups + g0) * kTileRows, zn, bar);
        if (sn) tma_bulk_g2s(sbase + s_off + s * Cfg::kSSlot, p.qs + ((size_t)tile * p.groups + g0) * kTileRows, sn, bar);
        gpos += 2;
        if (hpg == 1) { g0 += 2; gpos = 0; } else if (gpos >= hpg) { gpos = 0; ++g0; }
        if (++s == NS) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------ activation producer -----------------------
    if (lane == 0) {
      prefetch_tensormap(&tmap_x);
      grid_dependency_wait();
      int s = 0;
      uint32_t ph = 1;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(smem_u32(&bar_xempty[s]), ph, abortp, kSleepProducer, wait_limit)) break;
        const uint32_t bar = smem_u32(&bar_xfull[s]);
        const uint32_t dst = sbase + x_off + s * Cfg::kXBytes;
        mbar_arrive_expect_tx(bar, Cfg::kXBytes);
        tma_tensor_2d_g2s(dst, &tmap_x, (kb0 + i) * kStageK, mtile * NB, bar);
        tma_tensor_2d_g2s(dst + NB * 128, &tmap_x, (kb0 + i) * kStageK + 64, mtile * NB, bar);
        if (++s == NX) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1 || (warp == 2 && Cfg::kIssuers == 2)) {
    // ------------------------------ MMA issuer(s) -----------------------------
    // Issuer e takes stages e, e + kIssuers, ...  POST: every stage has its own accumulator.
    // PRE: every issuer has its own accumulator over all its stages; the epilogue adds them.
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_f16_m128(NB);
      const int e = (warp == 1) ? 0 : 1;
      for (int i = e; i < nkb; i += Cfg::kIssuers) {
        const int xs = i % NX, r = i % R;
        const uint32_t phx = (uint32_t)(i / NX) & 1u, phr = (uint32_t)(i / R) & 1u;
        // (the operand in tensor memory first: its decode waited for the MMAs of stage i - R, so the previous stage in
        // the activation slot, which may be the other issuer's, has landed and the parity of xfull is unambiguous)
        if (!mbar_wait(smem_u32(&bar_afull[r]), phr, abortp, kSleepMma, wait_limit)) break;
        if (!mbar_wait(smem_u32(&bar_xfull[xs]), phx, abortp, kSleepMma, wait_limit)) break;
        if (POST) {
          if (!mbar_wait(smem_u32(&bar_dempty[r]), phr ^ 1u, abortp, kSleepMma, wait_limit)) break;
        }
        tc_fence_after();
        const uint32_t a_tmem = tmem_base + r * kAColsPerSlot;
        const uint32_t d_tmem = tmem_base + Cfg::kDBase + (POST ? r * NB : e * NB);
        const uint32_t xsm = sbase + x_off + xs * Cfg::kXBytes;
        const uint64_t bd0 = smem_desc_k_sw128(xsm), bd1 = smem_desc_k_sw128(xsm + NB * 128);
        mma_f16_ts_stage8(d_tmem, a_tmem, (uint32_t)bd0, (uint32_t)bd1, (uint32_t)(bd0 >> 32), idesc,
                          POST ? 0u : (i >= Cfg::kIssuers ? 1u : 0u));
        mma_commit(smem_u32(&bar_done[r]));
      }
      mma_commit(smem_u32(&bar_final));  // every MMA this thread issued is complete
    }
    __syncwarp();
  } else if (warp >= 4 && warp < Cfg::kScaleWarp0) {
    // ------------------------------ decode warps ------------------------------
    // group `grp` takes stages grp, grp + DG, ...; inside a group thread (row, h) owns 64 codes
    const int grp = (warp - 4) >> 3;
    const int q = warp & 3, h = ((warp - 4) >> 2) & 1;
    const int row = q * 32 + lane;
    // with groups of 64 the two halves of a stage belong to different groups: half h reads
    // the second record of the stage's zero / scale slot
    const int qsel = (p.halfstages_per_group == 1 && h == 1) ? kTileRows : 0;
    constexpr bool frag = FRAG;
    // position of the row's scale / zero inside the tile's 128 (fragment layers keep them in fragment order)
    const int qrow = qsel + (frag ? frag_pos_of_row(row) : row);
    for (int i = grp; i < nkb; i += DG) {
      // ring positions and phases of stage i (NS, R, NX are compile-time constants: multiply-shift, no division)
      const int s = i % NS, r = i % R;
      const uint32_t phs = (uint32_t)(i / NS) & 1u, phr = ((uint32_t)(i / R) & 1u) ^ 1u;
      if (!mbar_wait(smem_u32(&bar_wfull[s]), phs, abortp, kSleepDecode, wait_limit)) break;
      const uint32_t z = has_z ? (uint32_t)gbase[z_off + s * Cfg::kZSlot + qrow] : p.zconst;
      __half2 d[32];
      if constexpr (FRAG) StageDecodeFragment<BITS, kSwizzledStage<BITS, FRAG, POST>>::run(gbase + w_off + s * Cfg::kWBytes, row, h, z, d);
      else StageDecode<BITS>::run(gbase + w_off + s * Cfg::kWBytes, row, h, z, d);
      uint32_t rr[32];
      if (!POST && has_s) {
        const __half2 s2 = __half2half2(reinterpret_cast<const __half*>(gbase + s_off + s * Cfg::kSSlot)[qrow]);
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = as_u32(__hmul2(d[j], s2));
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = as_u32(d[j]);
      }
      // the upper half of a half-filled last stage: its activations are zero-filled, its slot holds older bytes
      if (!FRAG && p.half_tail && h == 1 && kb0 + i == p.kblocks - 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = 0u;
      }
      // the packed stage is in registers: hand the shared-memory slot back to the producer
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_wempty[s]));
      // slot r was last read by the MMAs of stage i - R
      if (!mbar_wait(smem_u32(&bar_done[r]), phr, abortp, kSleepDecode, wait_limit)) break;
      // ... and the activation tile of that stage is free as well: tell its producer.  The
      // decode warps cannot fall behind the commits (the MMAs need their stores), so this
      // relay never misses a phase; R <= NX makes it reach every tile that is still needed.
      if (i >= R && (warp & 7) == 4 && lane == 0) mbar_arrive(smem_u32(&bar_xempty[(i - R) % NX]));
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + r * kAColsPerSlot + h * 32;
      tmem_st_x16(taddr, reinterpret_cast<const uint32_t(&)[16]>(rr[0]));
      tmem_st_x16(taddr + 16, reinterpret_cast<const uint32_t(&)[16]>(rr[16]));
      // publish at once: the MMAs of this stage start a whole decode earlier than with a deferred
      // hand-off, which matters more than the store latency exposed here (measured)
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_afull[r]));
    }
  } else if (warp >= Cfg::kScaleWarp0) {
    // ------------------------------ scale / epilogue warps --------------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int n = tile * kTileRows + row;
    const int m0 = mtile * NB;
    if constexpr (POST) {
      bool ok = true;
      // one 16-column chunk of results: fp16 output, or fp32 split-K partial
      auto store_chunk = [&](int c, const float* v) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int m = m0 + c + j;
          if (m < p.m) {
            if (S == 1) {
              if (n < p.n) p.y[(size_t)m * p.n + n] = __float2half_rn(v[j]);
            } else {
              p.partial[((size_t)split * p.m + m) * p.npad + n] = v[j];
            }
          }
        }
      };
      // split-K: every epilogue warp publishes its 32 rows; per row quarter, the LAST warp to arrive
      // over all splits sums that quarter's partials in split order (splitk_reduce)
      auto finish_split = [&]() {
        if (S <= 1) return;
        __threadfence();
        __syncwarp();
        unsigned prev = 0;
        unsigned* ctr = p.counters + (unit.ctr * 4 + q);
        if (lane == 0) prev = atomicAdd(ctr, 1u);
        prev = __shfl_sync(0xffffffffu, prev, 0);
        if (prev != (unsigned)(S - 1)) return;
        __threadfence();
        const int n0 = n - lane;
        splitk_reduce<NB>(p.partial + (size_t)m0 * p.npad + n0, (uint32_t)p.m * p.npad, (uint32_t)p.npad, S, p.m - m0,
                          p.n - n0, p.y + (size_t)m0 * p.n + n0, (size_t)p.n, lane);
        if (lane == 0) *ctr = 0u;
      };
      float acc[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j) acc[j] = 0.f;
      const size_t sz_row = (size_t)tile * p.groups * kTileRows +
                            (FRAG ? frag_pos_of_row(row) : row);
      // (POST needs groups of whole stages, but for a group-less layer of K = 64: half a stage)
      const int stages_per_group = max(1, p.halfstages_per_group >> 1);
      int r = 0;
      uint32_t phr = 0;
      // scales are fetched two stages ahead of their use
      // group of stage kb0 + j, advanced without divisions: (gq, gr) = divmod(kb0 + j, stages_per_group)
      int gq = (kb0 + 2) / stages_per_group, gr = (kb0 + 2) % stages_per_group;
      auto scale_at = [&](int j, int grp) -> __half {
        return (has_s && j < nkb) ? p.qs[sz_row + (size_t)grp * kTileRows] : __ushort_as_half(0x3C00);
      };
      __half sc0 = scale_at(0, kb0 / stages_per_group), sc1 = scale_at(1, (kb0 + 1) / stages_per_group);
      for (int i = 0; i < nkb; ++i) {
        const float sval = __half2float(sc0);
        sc0 = sc1;
        sc1 = scale_at(i + 2, gq);
        if (++gr == stages_per_group) { gr = 0; ++gq; }
        if (!mbar_wait(smem_u32(&bar_done[r]), phr, abortp, kSleepScale, wait_limit)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + Cfg::kDBase + r * NB;
        constexpr int CH = NB < 32 ? NB : 32;  // columns read back per wait
#pragma unroll
        for (int c0 = 0; c0 < NB; c0 += CH) {
          uint32_t v[CH];
#pragma unroll
          for (int c = 0; c < CH; c += 16) tmem_ld_x16(taddr + c0 + c, reinterpret_cast<uint32_t(&)[16]>(v[c]));
          tmem_wait_ld();
          if (c0 + CH == NB) {  // the accumulator is free as soon as its last chunk is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_dempty[r]));
          }
#pragma unroll
          for (int j = 0; j < CH; ++j) acc[c0 + j] = fmaf(sval, __uint_as_float(v[j]), acc[c0 + j]);
        }
        if (++r == R) { r = 0; phr ^= 1; }
      }
      if (!p.early) grid_launch_dependents();
      if (ok) {
        grid_dependency_wait();  // y and the workspace may still be in use by the preceding kernel
#pragma unroll
        for (int c = 0; c < NB; c += 16) store_chunk(c, &acc[c]);
        finish_split();
      }
    } else {
      mbar_wait(smem_u32(&bar_final), 0, abortp, 500, wait_limit);   // (the results: all warps, below)
    }
  }

  if constexpr (!POST) {
    // ------------------------------ results, one accumulator over the K range: all warps ----
    // (with the four epilogue warps alone a split of (2048,2048) at 64 rows cost 6 us: chains of dependent loads)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (Cfg::kTwoPerSM && !p.early) grid_launch_dependents();
    if (!*abortp) {   // (an abandoned launch stores nothing)
      grid_dependency_wait();
      // (kRederive: worked out again from what the hardware knows)
      int cx = blockIdx.x, cy = blockIdx.y, cz = blockIdx.z, tid = threadIdx.x;
      if constexpr (Cfg::kRederive)
        asm volatile("mov.u32 %0, %%ctaid.x;\n\tmov.u32 %1, %%ctaid.y;\n\tmov.u32 %2, %%ctaid.z;\n\tmov.u32 %3, %%tid.x;"
                     : "=r"(cx), "=r"(cy), "=r"(cz), "=r"(tid));
      const TcUnit u = Cfg::kRederive ? tc_unit(p, cx, cy, cz) : unit;
      const int warp = tid >> 5, lane = tid & 31, split = u.split, S = u.S, tail_unit = u.tail;
      const int q = warp & 3, m0 = u.mtile * NB, n0 = u.tile * kTileRows + q * 32, n = n0 + lane;
      const int cols = min(NB, p.m - m0);
      const int c0 = (warp >> 2) * 16;
      constexpr int kStep = Cfg::kThreads / 128 * 16;
      const uint32_t acc = (Cfg::kRederive ? *static_cast<volatile uint32_t*>(&tmem_holder) : tmem_base) + ((uint32_t)(q * 32) << 16) + Cfg::kDBase;
      const bool two = Cfg::kIssuers == 2 && u.nkb >= 2;  // the second accumulator holds something
      const bool vec = n0 + 32 <= p.n && p.n % 8 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15u) == 0;
      __half* y = p.y + (size_t)m0 * p.n + n0;
      auto load16 = [&](int c, float (&f)[16]) {
        uint32_t v[16], v2[16];
        tmem_ld_x16(acc + c, v);
        if (two) tmem_ld_x16(acc + NB + c, v2);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; ++k) f[k] = two ? __uint_as_float(v[k]) + __uint_as_float(v2[k]) : __uint_as_float(v[k]);
      };
      // partial sums: [range][unit][column][128] of the units that are cut, or [range][batch row][row]
      const size_t sstride = tail_unit >= 0 ? (size_t)p.tail_units * NB * kTileRows : (size_t)p.m * p.npad;
      const size_t cstride = tail_unit >= 0 ? (size_t)kTileRows : (size_t)p.npad;
      float* part = tail_unit >= 0 ? p.partial + (size_t)tail_unit * NB * kTileRows + q * 32 + lane
                                   : p.partial + (size_t)m0 * p.npad + n;
      // the ranges in the order of K, the own one from tensor memory (the same bits) or, like the others, from memory
      auto sum = [&](int own) {
#pragma unroll 1
        for (int c = c0; c < cols; c += kStep) {
          float s[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) s[k] = 0.f;
#pragma unroll 1
          for (int sp = 0; sp < S; ++sp) {
            float f[16];
            if (sp == own) {
              load16(c, f);
            } else {
              const float* b = part + (size_t)sp * sstride + (size_t)c * cstride;
#pragma unroll
              for (int k = 0; k < 16; ++k) f[k] = c + k < cols ? __ldcg(b + (size_t)k * cstride) : 0.f;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) s[k] += f[k];
          }
          put_rows<16>(y, p.n, c, cols, n < p.n, vec, lane, s);
        }
      };
      if (S == 1) {
#pragma unroll 1
        for (int c = c0; c < cols; c += kStep) {
          float f[16];
          load16(c, f);
          put_rows<16>(y, p.n, c, cols, n < p.n, vec, lane, f);
        }
      } else {
        // the last range to arrive, per 32 rows, sums them all; one that finds the others there when it comes needs
        // no partial sums of its own in memory
        unsigned* ctr = p.counters + (u.ctr * 4 + q);
        if (warp < 4 && lane == 0) {
          unsigned seen;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(ctr) : "memory");
          tail_seen[q] = seen;
        }
        __syncthreads();
        const bool there = tail_seen[q] == (unsigned)(S - 1);
        if (there) {
          sum(split);
        } else {
#pragma unroll 1
          for (int c = c0; c < cols; c += kStep) {
            float f[16];
            load16(c, f);
            float* b = part + (size_t)split * sstride + (size_t)c * cstride;
#pragma unroll
            for (int k = 0; k < 16; ++k)
              if (c + k < cols) __stcg(b + (size_t)k * cstride, f[k]);
          }
          __threadfence();
        }
        __syncthreads();
        if (warp < 4 && lane == 0) {
          if (there) {
            *ctr = 0u;
            tail_seen[q] = 0u;
          } else {
            __threadfence();
            tail_seen[q] = atomicAdd(ctr, 1u) == (unsigned)(S - 1) ? 1u : 0u;
            __threadfence();
          }
        }
        __syncthreads();
        if (tail_seen[q]) {
          __threadfence();
          sum(-1);
          if (warp < 4 && lane == 0) *ctr = 0u;
        }
      }
      tc_fence_before();
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before();
  __syncthreads();   // every role has left its loop (a role that ran out of work early must not
                     // look at the abort flag before the others had the chance to raise it)
  if (*abortp) {
    // give bulk copies still in flight time to land before shared memory is released (bounded)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1u);
  }
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(Cfg::kRederive ? *static_cast<volatile uint32_t*>(&tmem_holder) : tmem_base, Cfg::kTmemCols);
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
template <int BITS, int NB, bool POST, int DG, bool FRAG>
static cudaError_t launch_cfg_layout(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, dim3 grid, cudaStream_t st);

template <int BITS, int NB, bool POST, int DG>
static cudaError_t launch_cfg(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, dim3 grid, cudaStream_t st) {
  if (p.layout == QFB_LAYOUT_FRAGMENT) return launch_cfg_layout<BITS, NB, POST, DG, true>(tm, tw, p, grid, st);
  return launch_cfg_layout<BITS, NB, POST, DG, false>(tm, tw, p, grid, st);
}

template <int BITS, int NB, bool POST, int DG, bool FRAG>
static cudaError_t launch_cfg_layout(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, dim3 grid, cudaStream_t st) {
  using Cfg = TcCfg<BITS, NB, POST, DG>;
  auto kern = qgemm_tc_kernel<BITS, NB, POST, DG, FRAG, false>;
  // scale-in-the-decode mode: the common case of scales and zero points present has a build of its own (measured:
  // 2-6 % faster from 64 rows up; with per-stage accumulators the same specialisation was 3 % slower, not used)
  if constexpr (!POST) {
    if (p.qz && p.qs) kern = qgemm_tc_kernel<BITS, NB, POST, DG, FRAG, true>;
  }
  // the attribute belongs to the (function, device) pair: set it on every launch, it is cheap
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(Cfg::kThreads);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, tm, tw, p);
}

template <int BITS, int DG>
static cudaError_t launch_nb(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, int nb, bool post, dim3 grid,
                             cudaStream_t st) {
  if (post) {
    if (DG != 1) return cudaErrorInvalidValue;  // (narrow batch tiles: one decode group only)
    switch (nb) {
      case 16: return launch_cfg<BITS, 16, true, 1>(tm, tw, p, grid, st);
      case 32: return launch_cfg<BITS, 32, true, 1>(tm, tw, p, grid, st);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (nb) {
    case 64: return launch_cfg<BITS, 64, false, DG>(tm, tw, p, grid, st);
    case 128: return launch_cfg<BITS, 128, false, DG>(tm, tw, p, grid, st);
    case 256: return launch_cfg<BITS, 256, false, DG>(tm, tw, p, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int DG>
static cudaError_t launch_bits(const CUtensorMap& tmap_x, const CUtensorMap& tmap_w, const TcParams& p, int bits, int nb, bool post, dim3 grid,
                               cudaStream_t st) {
  switch (bits) {
    case 2: return launch_nb<2, DG>(tmap_x, tmap_w, p, nb, post, grid, st);
    case 3: return launch_nb<3, DG>(tmap_x, tmap_w, p, nb, post, grid, st);
    case 4: return launch_nb<4, DG>(tmap_x, tmap_w, p, nb, post, grid, st);
    case 8: return launch_nb<8, DG>(tmap_x, tmap_w, p, nb, post, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_gemm_tc(const CUtensorMap& tmap_x, const CUtensorMap& tmap_w, const TcParams& p, int bits, int nb, bool post, int decode_groups,
                           dim3 grid, cudaStream_t st) {
  // two decode groups (768 threads, one CTA per SM) where the scale is applied in the decode:
  // measured +10-17 % from 33 rows up, bit-identical results; three groups (1024 threads, 64
  // registers) were 3-6 % slower than two, and the narrow per-stage-accumulator tiles gain nothing
  if (decode_groups == 2 && !post) return launch_bits<2>(tmap_x, tmap_w, p, bits, nb, post, grid, st);
  return launch_bits<1>(tmap_x, tmap_w, p, bits, nb, post, grid, st);
}

}  // namespace qfb
