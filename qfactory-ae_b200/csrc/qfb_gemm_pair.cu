// Tensor-core path for wide batches: y^T[n, m] = W[n, :] . x[m, :] on CTA pairs (tcgen05 cta_group::2).
// No counterpart in the reference, whose kernels are CUDA-core GEMVs only (qfactory/include/gptq_gemv.h:14-154).
//
// The roles and the data flow are those of qfb_gemm_tc.cu with the scale applied in the decode; what differs:
//
//   pair        two CTAs (two neighbouring 128-row weight tiles) run ONE 256-row MMA.  Each decodes its own weight
//               rows into its own tensor memory, loads HALF of the activation tile into its own shared memory, and
//               keeps the accumulators of its own rows.  A single CTA streams the whole tile (64 KB a stage of 128 k
//               at 256 columns) at 7-8 TB/s of L2 -> SM traffic, which paced the wide tiles; the pair halves that and
//               the shared-memory reads of the MMAs, and the ring gets twice as deep.
//   persistent  one pair per two SMs.  The 128-k stages of all (row tile pair, batch tile) units form one line that
//               is cut into equal runs, one per pair, so that no wave is partly filled; the producers and the decode
//               run ahead into the next unit while the accumulators of the last one are stored.  A unit cut by a run
//               boundary is summed from fp32 partials, in the order of K, by the last of its CTAs to arrive.
//   batch tile  a run-time multiple of 32 columns, so that a batch is cut into equal tiles and not into full ones and
//               a remainder.
//
// Barriers: the leader (rank 0) issues every MMA.  Its `xfull` counts the bytes of both CTAs' activation copies, its
// `afull` the decode warps of both, its `dfree` the epilogue warps of both; `done`, `xempty` and `dfull` are committed
// to both.  Every wait is bounded as in qfb_gemm_tc.cu; both CTAs pass one cluster barrier before either leaves, so
// nothing is signalled to or read from a CTA that has gone.
//
// Measured (us, single-CTA kernel -> this): (28672,8192) at 256 / 1024 rows 137 -> 104 and 486 -> 375 (the latter 1.28
// PFLOP/s and limited by power: 322 with the operands zeroed), (8192,8192) at 256 rows 64 -> 44, (12288,4096) at 1024
// rows 125 -> 88, 8-bit (8192,8192) at 512 rows 81 -> 58 (launches in a row, workspaces with room to cut units; without it
// every unit runs whole).  Up to 128 columns it is slower than the single-CTA kernel
// (64 / 128 rows 81 / 85 against 63 / 77): the chain of hand-offs of a stage, longer across two CTAs, bounds both there.
#include "qfb_common.cuh"
#include "qfb_kernels.h"
#include "qfb_ptx.cuh"
#include "qfb_tc_stage.cuh"

namespace qfb {

using namespace ptx;

constexpr int kPairCols = 256;   // accumulator columns: the widest batch tile

template <int BITS>
struct PairCfg {
  static constexpr int kGroups = 2;                       // decode groups of 8 warps, alternate stages
  static constexpr int kThreads = 128 + 256 * kGroups + 128;
  static constexpr int kEpilogueWarp0 = 4 + 8 * kGroups;
  static constexpr int kWBytes = 128 * kStageK * BITS / 8;
  static constexpr int kXBytes = kPairCols / 2 * kStageK * 2;   // this CTA's half of the activation tile
  static constexpr int kZSlot = 256, kSSlot = 512;
  static constexpr int kRing = 4;                         // operand slots in tensor memory beside the accumulators
  static constexpr int kXStages = 4;
  static constexpr int kWRaw = (224 * 1024 - kXStages * kXBytes) / (kWBytes + kZSlot + kSSlot);
  // even, like every ring here: a parity wait is only sound for a thread that knows the phase before the awaited one
  // to be complete, so a slot always belongs to the same decode group
  static constexpr int kWStages = (kWRaw > 12 ? 12 : kWRaw) & ~1;
  static constexpr int kDBase = kRing * kAColsPerSlot;
  static constexpr size_t kSmemBytes = 1024 + (size_t)kXStages * kXBytes + (size_t)kWStages * (kWBytes + kZSlot + kSSlot);
  static_assert(kWStages >= 2 && kRing % 2 == 0, "rings");
  static_assert(kDBase + kPairCols <= 512, "tensor memory over-subscribed");
};

// One contiguous piece of a unit's K range, run by one pair.
struct PairJob {
  int unit, kb0, nkb;
};
// Runs: pair p takes stages [start(p), start(p + 1)) of the line of units * kblocks stages.  A boundary closer than
// kSnap stages to a unit's end moves there: a piece that short costs more in partial sums than it balances.  (The host
// asks for runs of at least kblocks or 16 stages, so that no two boundaries inside a unit fall together.)
struct PairRuns {
  static constexpr int kSnap = 6;
  long long total;
  int kblocks, pairs, cut;   // cut = 0: whole units only
  __device__ __forceinline__ long long start(int p) const {
    if (p >= pairs) return total;
    const long long s = (long long)p * total / pairs;
    const int r = (int)(s % kblocks);
    if (!cut) return s - r;
    return r < kSnap ? s - r : kblocks - r < kSnap ? s + kblocks - r : s;
  }
  __device__ __forceinline__ int pair_of(long long s) const {
    int p = (int)(((s + 1) * pairs - 1) / total);
    while (p + 1 < pairs && start(p + 1) <= s) ++p;
    while (p > 0 && start(p) > s) --p;
    return p;
  }
  __device__ __forceinline__ PairJob job(long long s, long long end) const {
    PairJob j;
    j.unit = (int)(s / kblocks);
    j.kb0 = (int)(s - (long long)j.unit * kblocks);
    const long long left = end - s;
    j.nkb = (int)(left < kblocks - j.kb0 ? left : kblocks - j.kb0);
    return j;
  }
};

// The finished accumulators of one job, as seen by one warp: lane = weight row, 32 of the tile's 128 rows.
struct PairTile {
  static constexpr size_t kTileFloats = (size_t)kPairCols * kTileRows;
  int pieces, piece, cols, n_total;
  uint32_t acc;             // tensor-memory column 0 of the accumulators, the warp's 32 lanes
  bool row_ok, vec;
  __half* y;                // first batch column of the tile, first row of the warp
  const float* part;        // this lane's row in piece 0 of the pair that starts the unit
  unsigned* ctr;
  int lane;

  __device__ __forceinline__ PairTile(const TcParams& p, const PairRuns& runs, const PairJob& j, int pair, uint32_t rank,
                                      uint32_t tmem_acc, int q, int lane_) : lane(lane_) {
    int first_pair = pair;
    pieces = 1;
    piece = 0;
    if (j.nkb < p.kblocks) {
      first_pair = runs.pair_of((long long)j.unit * p.kblocks);
      pieces = runs.pair_of((long long)(j.unit + 1) * p.kblocks - 1) - first_pair + 1;
      piece = pair - first_pair;
    }
    const int n0 = (j.unit / p.mtiles * 2 + (int)rank) * kTileRows + q * 32, m0 = (j.unit % p.mtiles) * p.nb;
    cols = min(p.nb, p.m - m0);
    n_total = p.n;
    row_ok = n0 + lane < p.n;
    y = p.y + (size_t)m0 * p.n + n0;
    // 16-byte stores: whole rows of the warp inside the layer, every output row 16-byte aligned
    vec = n0 + 32 <= p.n && p.n % 8 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15u) == 0;
    acc = tmem_acc + ((uint32_t)(q * 32) << 16);
    // partial sums: [pair][piece that starts its unit / other][rank][column][128]; a pair has at most one of each
    part = p.partial + ((size_t)first_pair * 4 + rank) * kTileFloats + q * 32 + lane;
    ctr = p.counters + (first_pair * 2 + (int)rank) * 4 + q;   // (a pair starts at most one cut unit)
  }
  __device__ __forceinline__ float* piece_base(int sp) const {
    return const_cast<float*>(part) + (sp == 0 ? 0 : (size_t)(2 * sp + 1) * 2 * kTileFloats);
  }
  // 16 columns at c
  __device__ __forceinline__ void load16(int c, float* f) const {
    uint32_t v[16];
    tmem_ld_x16(acc + c, v);
    tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k] = __uint_as_float(v[k]);
  }
  __device__ __forceinline__ void put(int c, const float (&f)[32]) const {
    put_rows<32>(y, n_total, c, cols, row_ok, vec, lane, f);
  }
  __device__ __forceinline__ void store(int c0, int step) const {
#pragma unroll 1
    for (int c = c0; c < cols; c += step) {
      float f[32];
      load16(c, f);
      load16(c + 16, f + 16);
      put(c, f);
    }
  }
  __device__ __forceinline__ void publish(int c0, int step) const {
    float* mine = piece_base(piece);
#pragma unroll 1
    for (int c = c0; c < cols; c += step) {
      float f[32];
      load16(c, f);
      load16(c + 16, f + 16);
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (c + k < cols) __stcg(mine + (size_t)(c + k) * kTileRows, f[k]);
    }
  }
  // the pieces in the order of K, the own one from tensor memory (the same bits) or, like the others, from memory
  __device__ __forceinline__ void sum(int c0, int step, bool own_in_tmem) const {
#pragma unroll 1
    for (int c = c0; c < cols; c += step) {
      float s[32];
#pragma unroll
      for (int h = 0; h < 32; h += 16) {
#pragma unroll
        for (int k = 0; k < 16; ++k) s[h + k] = 0.f;
#pragma unroll 1
        for (int sp = 0; sp < pieces; ++sp) {
          float f[16];
          if (own_in_tmem && sp == piece) {
            load16(c + h, f);
          } else {
            const float* b = piece_base(sp);
#pragma unroll
            for (int k = 0; k < 16; ++k) f[k] = c + h + k < cols ? __ldcg(b + (size_t)(c + h + k) * kTileRows) : 0.f;
          }
#pragma unroll
          for (int k = 0; k < 16; ++k) s[h + k] += f[k];
        }
      }
      put(c, s);
    }
  }
  // How many pieces have arrived (their sums are visible to the warp); called by whole warps.  Lane 0 acquires; the
  // barrier hands what it has seen to the other lanes, which a shuffle alone would not.
  __device__ __forceinline__ unsigned arrived() const {
    unsigned v = 0;
    if (lane == 0) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
    __syncwarp();
    return __shfl_sync(0xffffffffu, v, 0);
  }
  __device__ __forceinline__ unsigned arrive_lane() const { return atomicAdd(ctr, 1u); }
  // the warp's sums are out (every lane's, by the barrier and lane 0's fence after it), and those of the pieces that
  // arrived before are visible to every lane
  __device__ __forceinline__ unsigned arrive() const {
    unsigned prev = 0;
    __syncwarp();
    if (lane == 0) {
      __threadfence();
      prev = arrive_lane();
      __threadfence();
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, prev, 0);
  }
  __device__ __forceinline__ void reset_lane() const { *ctr = 0u; }
  __device__ __forceinline__ void reset() const {
    __syncwarp();
    if (lane == 0) reset_lane();
  }
};

template <int BITS, bool FRAG, bool ASYM>
__global__ void __launch_bounds__(PairCfg<BITS>::kThreads, 1)
qgemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const TcParams p) {
  using Cfg = PairCfg<BITS>;
  constexpr int NS = Cfg::kWStages, NX = Cfg::kXStages, R = Cfg::kRing, DG = Cfg::kGroups;

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_wfull[NS], bar_wempty[NS], bar_xfull[NX], bar_xempty[NX];
  __shared__ uint64_t bar_afull[R], bar_done[R], bar_dfull, bar_dfree;
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  __shared__ unsigned tail_seen[4];   // per 32 rows, of the last job: pieces that have arrived / this one is the last

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  PairRuns runs;
  runs.total = (long long)p.units * p.kblocks;
  runs.kblocks = p.kblocks;
  runs.pairs = gridDim.x >> 1;
  runs.cut = p.partial != nullptr;
  const int pair = blockIdx.x >> 1;
  const long long s_begin = runs.start(pair), s_end = runs.start(pair + 1);
  const int nb = p.nb;

  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
  constexpr uint32_t x_off = 0;
  constexpr uint32_t w_off = NX * Cfg::kXBytes;
  constexpr uint32_t z_off = w_off + NS * Cfg::kWBytes;
  constexpr uint32_t s_off = z_off + NS * Cfg::kZSlot;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(smem_u32(&bar_wfull[i]), 1);
      mbar_init(smem_u32(&bar_wempty[i]), kDecodeWarps);
    }
    for (int i = 0; i < NX; ++i) {
      mbar_init(smem_u32(&bar_xfull[i]), 1);
      mbar_init(smem_u32(&bar_xempty[i]), 1);
    }
    for (int i = 0; i < R; ++i) {
      mbar_init(smem_u32(&bar_afull[i]), 2 * kDecodeWarps);
      mbar_init(smem_u32(&bar_done[i]), 1);
    }
    mbar_init(smem_u32(&bar_dfull), 1);
    mbar_init(smem_u32(&bar_dfree), 8);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 2) tmem_alloc_pair(smem_u32(&tmem_holder), 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the barriers of both CTAs are initialised
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  volatile int* abortp = &abort_flag;
  const long long wait_limit = p.stall_test ? 200000LL : kWaitLimitCycles;
  grid_launch_dependents();
  if (!p.early) grid_dependency_wait();

  const bool has_z = ASYM || p.qz != nullptr;
  const bool has_s = ASYM || p.qs != nullptr;

  if (warp == 0) {
    // ------------------------------ weight producer ---------------------------
    if (lane == 0) {
      if constexpr (kSwizzledStage<BITS, FRAG, false>) prefetch_tensormap(&tmap_w);
      const int hpg = p.halfstages_per_group;
      const uint32_t ng = hpg == 1 ? 2u : 1u;
      const uint32_t zb = has_z ? ng * 128u : 0u, sb = has_s ? ng * 256u : 0u;
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (long long at = s_begin; ok && at < s_end;) {
        const PairJob j = runs.job(at, s_end);
        at += j.nkb;
        // (an odd number of row tiles: the last pair's second CTA repeats the last tile and stores nothing)
        const int tile = min(j.unit / p.mtiles * 2 + (int)rank, p.tiles - 1);
        int g0 = (j.kb0 * 2) / hpg, gpos = (j.kb0 * 2) % hpg;
        for (int i = 0; i < j.nkb; ++i) {
          if (!mbar_wait(smem_u32(&bar_wempty[s]), ph, abortp, kSleepProducer, wait_limit)) { ok = false; break; }
          const uint32_t bar = smem_u32(&bar_wfull[s]);
          // (K an odd multiple of 64: the last stage is half a stage of codes, and one group of 64)
          const bool half = !FRAG && p.half_tail && j.kb0 + i == p.kblocks - 1;
          const uint32_t wb = half ? Cfg::kWBytes / 2 : Cfg::kWBytes;
          const uint32_t zn = half && hpg == 1 ? zb / 2 : zb, sn = half && hpg == 1 ? sb / 2 : sb;
          mbar_arrive_expect_tx(bar, wb + zn + sn + ((p.stall_test && at == s_begin + j.nkb && i == 0) ? 16u : 0u));
          const uint32_t dst = sbase + w_off + s * Cfg::kWBytes;
          if constexpr (kSwizzledStage<BITS, FRAG, false>) {
            const int r0 = (tile * 2 * p.kblocks + j.kb0 + i) * (16 * BITS);
            tma_tensor_2d_g2s(dst, &tmap_w, 0, r0, bar);
            tma_tensor_2d_g2s(dst + Cfg::kWBytes / 2, &tmap_w, 0, r0 + p.kblocks * (16 * BITS), bar);
          } else if (FRAG) {
            const uint8_t* f0 = reinterpret_cast<const uint8_t*>(p.qw) +
                                (((size_t)tile * 2) * (size_t)(p.kblocks * 8) + (size_t)(j.kb0 + i) * 8) * (128 * BITS);
            tma_bulk_g2s(dst, f0, Cfg::kWBytes / 2, bar);
            tma_bulk_g2s(dst + Cfg::kWBytes / 2, f0 + (size_t)p.kblocks * 8 * (128 * BITS), Cfg::kWBytes / 2, bar);
          } else {
            tma_bulk_g2s(dst, reinterpret_cast<const uint8_t*>(p.qw) + (size_t)tile * p.k * (16 * BITS) +
                                  (size_t)(j.kb0 + i) * Cfg::kWBytes, wb, bar);
          }
          if (zn) tma_bulk_g2s(sbase + z_off + s * Cfg::kZSlot, p.qz + ((size_t)tile * p.groups + g0) * kTileRows, zn, bar);
          if (sn) tma_bulk_g2s(sbase + s_off + s * Cfg::kSSlot, p.qs + ((size_t)tile * p.groups + g0) * kTileRows, sn, bar);
          gpos += 2;
          if (hpg == 1) { g0 += 2; gpos = 0; } else if (gpos >= hpg) { gpos = 0; ++g0; }
          if (++s == NS) { s = 0; ph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------ activation producer -----------------------
    // this CTA's half of the columns; the bytes of both halves are counted on the leader's barrier (a copy of the
    // peer cannot run ahead of the phase: its slot is released by MMAs that waited for the phase before)
    if (lane == 0) {
      prefetch_tensormap(&tmap_x);
      grid_dependency_wait();
      const int half = nb >> 1;
      const uint32_t atom = (uint32_t)half * 128u;
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (long long at = s_begin; ok && at < s_end;) {
        const PairJob j = runs.job(at, s_end);
        at += j.nkb;
        const int row0 = (j.unit % p.mtiles) * nb + (int)rank * half;
        for (int i = 0; i < j.nkb; ++i) {
          if (!mbar_wait(smem_u32(&bar_xempty[s]), ph, abortp, kSleepProducer, wait_limit)) { ok = false; break; }
          const uint32_t bar = mapa(smem_u32(&bar_xfull[s]), 0);
          const uint32_t dst = sbase + x_off + s * Cfg::kXBytes;
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&bar_xfull[s]), 4u * atom);
          tma_tensor_2d_g2s_pair(dst, &tmap_x, (j.kb0 + i) * kStageK, row0, bar);
          tma_tensor_2d_g2s_pair(dst + atom, &tmap_x, (j.kb0 + i) * kStageK + 64, row0, bar);
          if (++s == NX) { s = 0; ph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer, leader only -------------------
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = idesc_f16_m256(nb);
      const uint32_t d_tmem = tmem_base + Cfg::kDBase;
      bool ok = true;
      int it0 = 0, jn = 0;   // stages before this job, jobs done
      for (long long at = s_begin; ok && at < s_end; ++jn) {
        const PairJob j = runs.job(at, s_end);
        at += j.nkb;
        // the epilogue warps of both CTAs have read the accumulators of the job before
        if (jn > 0 && !mbar_wait_cluster(smem_u32(&bar_dfree), (uint32_t)(jn - 1) & 1u, abortp, kSleepMma, wait_limit)) break;
        uint32_t acc = 0;
        for (int i = 0; i < j.nkb; ++i) {
          const int it = it0 + i, xs = it % NX, r = it % R;
          if (!mbar_wait_cluster(smem_u32(&bar_afull[r]), (uint32_t)(it / R) & 1u, abortp, kSleepMma, wait_limit) ||
              !mbar_wait(smem_u32(&bar_xfull[xs]), (uint32_t)(it / NX) & 1u, abortp, kSleepMma, wait_limit)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t xsm = sbase + x_off + xs * Cfg::kXBytes;
          const uint64_t bd0 = smem_desc_k_sw128(xsm), bd1 = smem_desc_k_sw128(xsm + (uint32_t)(nb >> 1) * 128u);
          mma_f16_ts_stage8_pair(d_tmem, tmem_base + r * kAColsPerSlot, (uint32_t)bd0, (uint32_t)bd1, (uint32_t)(bd0 >> 32),
                                 idesc, acc);
          acc = 1;
          mma_commit_pair(smem_u32(&bar_done[r]));
          mma_commit_pair(smem_u32(&bar_xempty[xs]));
        }
        if (!ok) break;
        it0 += j.nkb;
        mma_commit_pair(smem_u32(&bar_dfull));   // every MMA of the job is complete
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < Cfg::kEpilogueWarp0) {
    // ------------------------------ decode warps ------------------------------
    const int grp = (warp - 4) >> 3;
    const int q = warp & 3, h = ((warp - 4) >> 2) & 1;
    const int row = q * 32 + lane;
    const int qsel = (p.halfstages_per_group == 1 && h == 1) ? kTileRows : 0;
    const int qrow = qsel + (FRAG ? frag_pos_of_row(row) : row);
    const uint32_t afull0 = mapa(smem_u32(&bar_afull[0]), 0);
    const int n_stages = (int)(s_end - s_begin), kb_first = (int)(s_begin % p.kblocks);
    for (int i = grp; i < n_stages; i += DG) {
      const int s = i % NS, r = i % R;
      if (!mbar_wait(smem_u32(&bar_wfull[s]), (uint32_t)(i / NS) & 1u, abortp, kSleepDecode, wait_limit)) break;
      const uint32_t z = has_z ? (uint32_t)gbase[z_off + s * Cfg::kZSlot + qrow] : p.zconst;
      __half2 d[32];
      if constexpr (FRAG) StageDecodeFragment<BITS, kSwizzledStage<BITS, FRAG, false>>::run(gbase + w_off + s * Cfg::kWBytes, row, h, z, d);
      else StageDecode<BITS>::run(gbase + w_off + s * Cfg::kWBytes, row, h, z, d);
      uint32_t rr[32];
      if (has_s) {
        const __half2 s2 = __half2half2(reinterpret_cast<const __half*>(gbase + s_off + s * Cfg::kSSlot)[qrow]);
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = as_u32(__hmul2(d[j], s2));
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = as_u32(d[j]);
      }
      // the upper half of a half-filled last stage: its activations are zero-filled, its slot holds older bytes
      if (!FRAG && p.half_tail && h == 1 && (kb_first + i) % p.kblocks == p.kblocks - 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j) rr[j] = 0u;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_wempty[s]));
      // the slot was last read by the MMAs of stage i - R
      if (!mbar_wait(smem_u32(&bar_done[r]), ((uint32_t)(i / R) & 1u) ^ 1u, abortp, kSleepDecode, wait_limit)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + r * kAColsPerSlot + h * 32;
      tmem_st_x16(taddr, reinterpret_cast<const uint32_t(&)[16]>(rr[0]));
      tmem_st_x16(taddr + 16, reinterpret_cast<const uint32_t(&)[16]>(rr[16]));
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(afull0 + r * 8);
    }
  } else if (warp >= Cfg::kEpilogueWarp0) {
    // ------------------------------ epilogue warps ----------------------------
    // every job but the last of the run, beside the next job's stages
    const uint32_t dfree = mapa(smem_u32(&bar_dfree), 0);
    int jn = 0;
    for (long long at = s_begin; at < s_end; ++jn) {
      const PairJob j = runs.job(at, s_end);
      at += j.nkb;
      // (an abandoned launch stores nothing)
      if (!mbar_wait(smem_u32(&bar_dfull), (uint32_t)jn & 1u, abortp, 200, wait_limit) || *abortp) break;
      tc_fence_after();
      if (jn == 0) grid_dependency_wait();  // y and the workspace may still be in use by the preceding kernel
      if (at == s_end) break;
      PairTile tl(p, runs, j, pair, rank, tmem_base + Cfg::kDBase, warp & 3, lane);
      if (tl.pieces == 1) {
        tl.store(0, 32);
      } else if (tl.arrived() == (unsigned)(tl.pieces - 1)) {
        tl.sum(0, 32, true);   // the others are there: this piece's sums need not pass through memory
        tl.reset();
      } else {
        tl.publish(0, 32);
        if (tl.arrive() == (unsigned)(tl.pieces - 1)) {
          tl.sum(0, 32, false);
          tl.reset();
        }
      }
      // the accumulators are free for the next job
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(dfree);
    }
  }

  // ------------------------------ the last job's results, by all warps --------
  // (the epilogue warps have waited for its MMAs; with those four warps alone the SM would sit behind their loads and
  // stores for many stages' time: (8192,8192) at 256 rows 64 us instead of 44)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (s_begin < s_end && !*abortp) {
    grid_dependency_wait();
    long long at = s_begin;
    PairJob j = runs.job(at, s_end);
    while (at + j.nkb < s_end) {
      at += j.nkb;
      j = runs.job(at, s_end);
    }
    constexpr int kStep = Cfg::kThreads / 128 * 32;
    const int c0 = (warp >> 2) * 32;
    PairTile tl(p, runs, j, pair, rank, tmem_base + Cfg::kDBase, warp & 3, lane);
    if (tl.pieces == 1) {
      tl.store(c0, kStep);
    } else {
      if (warp < 4) {
        const unsigned seen = tl.arrived();
        if (lane == 0) tail_seen[warp] = seen;
      }
      __syncthreads();
      if (tail_seen[warp & 3] == (unsigned)(tl.pieces - 1)) {
        tl.sum(c0, kStep, true);
      } else {
        tl.publish(c0, kStep);
        __threadfence();
      }
      __syncthreads();
      if (warp < 4 && lane == 0) {
        if (tail_seen[warp] == (unsigned)(tl.pieces - 1)) {
          tl.reset_lane();
          tail_seen[warp] = 0u;
        } else {
          __threadfence();
          tail_seen[warp] = tl.arrive_lane() == (unsigned)(tl.pieces - 1) ? 1u : 0u;
          __threadfence();
        }
      }
      __syncthreads();
      if (tail_seen[warp & 3]) {
        __threadfence();
        tl.sum(c0, kStep, false);
        if (warp < 4 && lane == 0) tl.reset_lane();
      }
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abortp) {
    // give bulk copies still in flight time to land before shared memory is released (bounded)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1u);
  }
  cluster_sync_all();   // the other CTA signals and reads nothing here any more
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
template <int BITS, bool FRAG>
static cudaError_t launch_pair_cfg(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, int pairs, cudaStream_t st) {
  using Cfg = PairCfg<BITS>;
  auto kern = p.qz && p.qs ? qgemm_pair_kernel<BITS, FRAG, true> : qgemm_pair_kernel<BITS, FRAG, false>;
  // the attribute belongs to the (function, device) pair: set it on every launch, it is cheap
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(Cfg::kThreads);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, tm, tw, p);
}

template <int BITS>
static cudaError_t launch_pair_bits(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, int pairs, cudaStream_t st) {
  return p.layout == QFB_LAYOUT_FRAGMENT ? launch_pair_cfg<BITS, true>(tm, tw, p, pairs, st)
                                         : launch_pair_cfg<BITS, false>(tm, tw, p, pairs, st);
}

cudaError_t launch_gemm_pair(const CUtensorMap& tm, const CUtensorMap& tw, const TcParams& p, int bits, int pairs,
                             cudaStream_t st) {
  switch (bits) {
    case 2: return launch_pair_bits<2>(tm, tw, p, pairs, st);
    case 3: return launch_pair_bits<3>(tm, tw, p, pairs, st);
    case 4: return launch_pair_bits<4>(tm, tw, p, pairs, st);
    case 8: return launch_pair_bits<8>(tm, tw, p, pairs, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qfb
