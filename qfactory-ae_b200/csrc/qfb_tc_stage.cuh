// What the tcgen05 kernels share: the decode of a 128-k weight stage into fp16 pairs and the sum of split-K partials.
#pragma once

#include "qfb_common.cuh"
#include "qfb_ptx.cuh"

namespace qfb {

using namespace ptx;

constexpr int kStageK = 128;              // k per pipeline stage
constexpr int kStepsPerStage = kStageK / 16;
constexpr int kAColsPerSlot = kStageK / 2;  // one 32-bit column holds two fp16 k
constexpr int kDecodeWarps = 8;
// sleep between polls of a barrier that is not ready yet, per role (ns)
constexpr unsigned kSleepScale = 100, kSleepProducer = 100, kSleepMma = 20, kSleepDecode = 20;

// Weight stages of 4- and 8-bit fragment layers arrive through a tensor map of 64-byte rows with the 64-byte swizzle.
// As plain bytes the 32 lanes of a decode warp read words 64 bytes apart: 4-way bank conflicts on each of the 16
// reads, 512 shared-memory cycles a stage beside the MMAs' and the copies' own (launches in a row, (28672,8192) at 64 /
// 1024 rows on one CTA 67.5 -> 62 and 580 -> 491 us, (8192,28672) at 128 rows 85 -> 75 us).  Not for 2 bits, whose words are 32 bytes apart
// (2-way, and 32-byte rows would double the copy's requests), nor for 3, whose planes are read without conflicts
// inside a row block; nor with per-stage accumulators (up to 32 rows), where it changes nothing ((8192,8192)
// 8-bit at 24 rows 27.7 us with it, 27.6 without).
template <int BITS, bool FRAG, bool POST> constexpr bool kSwizzledStage = FRAG && !POST && (BITS == 4 || BITS == 8);

// ---- decode of the 64 codes thread (row, h) owns in a 128-k stage -> 32 fp16 pairs ------
template <int BITS> struct StageDecode;
template <> struct StageDecode<4> {
  // stage = [4 units][128 rows][16 B]; thread owns units 2h, 2h+1
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const Codec<4>::ZM zm = Codec<4>::zmagic(z);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint4 v = *reinterpret_cast<const uint4*>(w + (((2 * h + u) * kTileRows + row) << 4));
      const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __half2 t[4];
        Codec<4>::word(ww[j], zm, t);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[16 * u + 4 * j + i] = t[i];
      }
    }
  }
};
// Fragment layouts: stage = [2 halves of 64 rows][8 k-steps of 128 * BITS bytes] (qfb_common.cuh).
// Row wt*64 + rb*16 + hh*8 + g owns, in the word frag_word_of(rb, hh) of lane g*4+t, the codes of
// k 4t..4t+3 of a step: two exact fp16 pairs in k order per word.
// SWZ (kSwizzledStage): the 64 bytes of a g (the words of t 0..3, 16 bytes each) arrived 64-byte-swizzled: the chunk
// of t sits at t ^ (g >> 1).
template <int BITS, bool SWZ> struct StageDecodeFragment;
template <bool SWZ> struct StageDecodeFragment<4, SWZ> {
  // nibbles 0,4,2,6 (hh = 0) or 1,5,3,7 (hh = 1): two LOP3 with the row's mask / magic
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const Codec<4>::ZM zm = Codec<4>::zmagic(z);
    const int wt = row >> 6, rb = (row >> 4) & 3, hh = (row >> 3) & 1, g = row & 7;
    const uint32_t mask = hh ? 0x00f000f0u : 0x000f000fu, magic = hh ? 0x54005400u : 0x64006400u;
    const __half2 zs = as_h2(hh ? zm.hi : zm.lo);
    const uint8_t* base = w + wt * 4096 + (4 * h) * 512 + g * 64 + rb * 4;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t word = *reinterpret_cast<const uint32_t*>(base + ks * 512 + ((SWZ ? t ^ (g >> 1) : t) << 4));
        d[ks * 8 + t * 2] = __hsub2(as_h2(lop3_and_or(word, mask, magic)), zs);
        d[ks * 8 + t * 2 + 1] = __hsub2(as_h2(lop3_and_or(word >> 8, mask, magic)), zs);
      }
  }
};
template <bool SWZ> struct StageDecodeFragment<8, SWZ> {
  // one word = the row's four bytes of k 4t..4t+3
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const Codec<8>::ZM zm = Codec<8>::zmagic(z);
    const int wt = row >> 6, rb = (row >> 4) & 3, hh = (row >> 3) & 1, g = row & 7;
    const uint8_t* base = w + wt * 8192 + (4 * h) * 1024 + frag_word_offset(8, g * 4, rb * 2 + hh);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t word = *reinterpret_cast<const uint32_t*>(base + ks * 1024 + ((SWZ ? t ^ (g >> 1) : t) << 4));
        d[ks * 8 + t * 2] = __hsub2(as_h2(prmt(word, 0x64646464u, 0x4140u)), as_h2(zm.m));
        d[ks * 8 + t * 2 + 1] = __hsub2(as_h2(prmt(word, 0x64646464u, 0x4342u)), as_h2(zm.m));
      }
  }
};
template <bool SWZ> struct StageDecodeFragment<2, SWZ> {
  // one word = two row blocks; the row's fields sit at bit o = 4 (rb & 1) + 2 hh of each byte pair
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const Codec<2>::ZM zm = Codec<2>::zmagic(z);
    const int wt = row >> 6, rb = (row >> 4) & 3, hh = (row >> 3) & 1, g = row & 7;
    const int oi = (rb & 1) * 2 + hh;  // bit offset / 2
    const uint32_t mask = 0x00030003u << (2 * oi);
    const uint32_t magic = oi == 0 ? 0x64006400u : oi == 1 ? 0x5C005C00u : oi == 2 ? 0x54005400u : 0x4C004C00u;
    const __half2 zs = as_h2(oi == 0 ? zm.m[0] : oi == 1 ? zm.m[1] : oi == 2 ? zm.m[2] : zm.m[3]);
    const uint8_t* base = w + wt * 2048 + (4 * h) * 256 + g * 32 + (rb >> 1) * 4;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t word = *reinterpret_cast<const uint32_t*>(base + ks * 256 + t * 8);
        d[ks * 8 + t * 2] = __hsub2(as_h2(lop3_and_or(word, mask, magic)), zs);
        d[ks * 8 + t * 2 + 1] = __hsub2(as_h2(lop3_and_or(word >> 8, mask, magic)), zs);
      }
  }
};
template <bool SWZ> struct StageDecodeFragment<3, SWZ> {
  // word j of lane g*4+t sits in plane j (128 bytes) of the k-step (384 bytes).  Row blocks 0..2: word rb, the
  // row's fields at bit offset 0 (rows g) or 3 (rows g + 8) for k 4t, 4t+1 and 9 bits higher for k 4t+2, 4t+3.
  // Row block 3: offset 6 of words 0 / 1 (rows g) and of word 2 (rows g + 8, k 4t, 4t+1); rows g + 8,
  // k 4t+2, 4t+3 are collected from the spare bits 15 / 31 of the three words.
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const int wt = row >> 6, rb = (row >> 4) & 3, hh = (row >> 3) & 1, g = row & 7;
    const uint8_t* base = w + wt * 3072 + (4 * h) * 384 + g * 16;
    if (rb < 3) {
      // the field as the low mantissa bits of 2^(10 - offset): exact q + 2^(10 - offset), minus the same with z
      const uint32_t mask = hh ? 0x00380038u : 0x00070007u, magic = hh ? 0x58005800u : 0x64006400u;
      const __half2 zs = as_h2(magic | ((z << (hh ? 3 : 0)) * 0x00010001u));
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t word = *reinterpret_cast<const uint32_t*>(base + ks * 384 + rb * 128 + t * 4);
          d[ks * 8 + t * 2] = __hsub2(as_h2(lop3_and_or(word, mask, magic)), zs);
          d[ks * 8 + t * 2 + 1] = __hsub2(as_h2(lop3_and_or(word >> 9, mask, magic)), zs);
        }
    } else {
      const uint32_t mask = 0x01C001C0u, magic = 0x4C004C00u;
      const __half2 zs = as_h2(magic | ((z << 6) * 0x00010001u));
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint8_t* p = base + ks * 384 + t * 4;
          const uint32_t w0 = *reinterpret_cast<const uint32_t*>(p), w1 = *reinterpret_cast<const uint32_t*>(p + 128),
                         w2 = *reinterpret_cast<const uint32_t*>(p + 256);
          const uint32_t spare = ((w0 >> 9) & 0x00400040u) | ((w1 >> 8) & 0x00800080u) | ((w2 >> 7) & 0x01000100u);
          const uint32_t lo = hh ? (w2 & mask) : (w0 & mask), hi = hh ? spare : (w1 & mask);
          d[ks * 8 + t * 2] = __hsub2(as_h2(lo | magic), zs);
          d[ks * 8 + t * 2 + 1] = __hsub2(as_h2(hi | magic), zs);
        }
    }
  }
};
template <> struct StageDecode<8> {
  // stage = [8 units][128 rows][16 B]; thread owns units 4h .. 4h+3
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const Codec<8>::ZM zm = Codec<8>::zmagic(z);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint4 v = *reinterpret_cast<const uint4*>(w + (((4 * h + u) * kTileRows + row) << 4));
      const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        d[8 * u + 2 * j] = __hsub2(as_h2(prmt(ww[j], 0x64646464u, 0x4140u)), as_h2(zm.m));
        d[8 * u + 2 * j + 1] = __hsub2(as_h2(prmt(ww[j], 0x64646464u, 0x4342u)), as_h2(zm.m));
      }
    }
  }
};
template <> struct StageDecode<2> {
  // stage = [2 units][128 rows][16 B]; thread owns unit h
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const uint4 v = *reinterpret_cast<const uint4*>(w + ((h * kTileRows + row) << 4));
    const Codec<2>::ZM zm = Codec<2>::zmagic(z);
    const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      __half2 t[4];
      Codec<2>::half_word(ww[j], zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[8 * j + i] = t[i];
      Codec<2>::half_word(ww[j] >> 8, zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[8 * j + 4 + i] = t[i];
    }
  }
};
template <> struct StageDecode<3> {
  // stage = one 3-bit unit = [3 vectors][128 rows][16 B]: two 2-bit-plane vectors and the
  // 1-bit-plane vector; thread owns 2-bit vector h and words 2h, 2h+1 of the plane vector
  __device__ static __forceinline__ void run(const uint8_t* w, int row, int h, uint32_t z, __half2 (&d)[32]) {
    const uint4 a = *reinterpret_cast<const uint4*>(w + ((h * kTileRows + row) << 4));
    const uint2 b = *reinterpret_cast<const uint2*>(w + ((2 * kTileRows + row) << 4) + (h << 3));
    const Codec<3>::ZM zm = Codec<3>::zmagic(z);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
    const uint32_t bw[2] = {b.x, b.y};
#pragma unroll
    for (int j = 0; j < 2; ++j) {  // 32 codes: 2-bit words aw[2j], aw[2j+1] with plane word bw[j]
      __half2 t[4];
      Codec<3>::half_word(aw[2 * j], bw[j] << 2, zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[16 * j + i] = t[i];
      Codec<3>::half_word(aw[2 * j] >> 8, bw[j] << 1, zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[16 * j + 4 + i] = t[i];
      Codec<3>::half_word(aw[2 * j + 1], bw[j] >> 6, zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[16 * j + 8 + i] = t[i];
      Codec<3>::half_word(aw[2 * j + 1] >> 8, bw[j] >> 7, zm, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[16 * j + 12 + i] = t[i];
    }
  }
};

// 32 rows (lane = row) x W columns of a warp, rounded to fp16 into y[column][row] (y: column 0, first row of the warp).
// With `vec` (whole 8-row runs inside the layer, every y row 16-byte aligned) three exchanges between lanes turn a row
// per lane into eight rows of W / 8 columns per lane: W / 8 stores of 16 bytes instead of W of 2.
template <int W>
__device__ __forceinline__ void put_rows(__half* y, int n_total, int c, int cols, bool row_ok, bool vec, int lane,
                                         const float (&f)[W]) {
  if (!vec) {
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (c + k < cols && row_ok) y[(size_t)(c + k) * n_total + lane] = __float2half_rn(f[k]);
    return;
  }
  uint32_t a[W / 2], b[W / 2];
  const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;
#pragma unroll
  for (int k = 0; k < W / 2; ++k) {   // a[k]: column 2 k + bit 0 of the lane, rows (lane & ~1) ..+1
    const uint32_t own = as_u32(__floats2half2_rn(f[2 * k], f[2 * k + 1]));
    a[k] = prmt(own, __shfl_xor_sync(0xffffffffu, own, 1), sel);
  }
  const bool h2 = lane & 2, h4 = lane & 4;
#pragma unroll
  for (int k = 0; k < W / 4; ++k) {    // b[2 k ..]: column 4 k + bits 0, 1, rows (lane & ~3) ..+3
    const uint32_t r = __shfl_xor_sync(0xffffffffu, h2 ? a[2 * k] : a[2 * k + 1], 2);
    b[2 * k] = h2 ? r : a[2 * k];
    b[2 * k + 1] = h2 ? a[2 * k + 1] : r;
  }
#pragma unroll
  for (int k = 0; k < W / 8; ++k) {    // column 8 k + bits 0, 1, 2, rows (lane & ~7) ..+7
    const uint32_t r0 = __shfl_xor_sync(0xffffffffu, h4 ? b[4 * k] : b[4 * k + 2], 4);
    const uint32_t r1 = __shfl_xor_sync(0xffffffffu, h4 ? b[4 * k + 1] : b[4 * k + 3], 4);
    const uint4 v = h4 ? make_uint4(r0, r1, b[4 * k + 2], b[4 * k + 3]) : make_uint4(b[4 * k], b[4 * k + 1], r0, r1);
    const int col = c + 8 * k + (lane & 7);
    if (col < cols) *reinterpret_cast<uint4*>(y + (size_t)col * n_total + (lane & ~7)) = v;
  }
}

}  // namespace qfb
