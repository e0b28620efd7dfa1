// Offline packer (replaces qfactory/convert.py:55-81 of the reference) and its inverse.
//
// The packer turns GPTQ-style tensors -- int32 codes [K,N], fp16 scales [K/GS,N], int32
// zeros [K/GS,N] -- into the tile-128 interleaved layout described in qfactory_b200.h.
// The inverse kernels run the SAME Codec<> bit extraction the compute kernels use, so a
// pack -> unpack round trip proves the in-kernel decode bit-exact.
#include "qfb_common.cuh"
#include "qfb_kernels.h"

namespace qfb {

// element held by field f of a 2/4/8-bit word (pair interleave: even elements low half)
__device__ __forceinline__ int field_element(int bits, int f) {
  if (bits == 8) return f;
  const int half_fields = 16 / bits;
  return f < half_fields ? 2 * f : 2 * (f - half_fields) + 1;
}

// bit position of element e (0..31) inside a word of the 3-bit format's 1-bit plane
__device__ __forceinline__ int plane1_bit(int e) {
  const int h = e >> 4, el = e & 15, f = el >> 1, parity = el & 1;
  const int variant = 2 * h + (f >> 2);
  const int base = (variant == 0) ? 0 : (variant == 1) ? 1 : (variant == 2) ? 8 : 9;
  return base + 2 * (f & 3) + 16 * parity;
}

// ---- packing --------------------------------------------------------------------------------------------------
// One CTA packs a block of 128 rows (output features) x 128 k: the codes are brought into shared memory as bytes
// [row][k], four consecutive k to a word, whatever the source holds, and the packed words of either layout are put
// together from there and leave in runs of 512 bytes.  HBM bound: the source is read once, coalesced along the
// rows, and the packed bytes are written once.  Measured, (8192,28672) 4-bit from a checkpoint's words to the packed
// layer: 58 us (4.2 TB/s of the 244 MB in and out); unpacking to int32, the range check and one thread per packed word
// took 1790.
// Row stride 36 words: a multiple of 4, so that sixteen codes are one 16-byte store, and 4 (mod 32), so that the
// fragment order's reads (8 rows x 4 words) and those stores meet no bank twice.
constexpr int kPackRow = 36;
constexpr int kPackK = 128;
constexpr int kPackThreads = 256;

// the codes of rows n0.. and k k0 .. k0 + klen of the CTA's block, four k per 32-bit word, rows past n zero
template <int BITS, int SRC>
__device__ __forceinline__ unsigned stage_codes(const PackParams& p, uint32_t* s, int n0, int k0, int klen) {
  const int row = threadIdx.x & 127, n = n0 + row;
  constexpr uint32_t kMask = (1u << BITS) - 1u;
  unsigned bad = 0;
  constexpr int kChunks = kPackK / 16 / (kPackThreads / 128);   // runs of 16 k of one row per thread
  constexpr int NWORD = SRC == kPackCodes ? 1 : BITS / 2;        // (int32 codes: a run at a time, 16 loads in flight)
  // checkpoint words (32 / BITS consecutive k of one row each): all of the thread's loads are in flight together
  uint32_t w[kChunks][NWORD];
  if (SRC == kPackGptq) {
#pragma unroll
    for (int u = 0; u < kChunks; ++u) {
      const int c = (threadIdx.x >> 7) + u * (kPackThreads / 128);
      const uint32_t* src = p.gptq_codes + (size_t)((k0 + c * 16) / (32 / BITS)) * p.n + n;
#pragma unroll
      for (int i = 0; i < NWORD; ++i) w[u][i] = (n < p.n && c * 16 < klen) ? __ldcs(src + (size_t)i * p.n) : 0u;
    }
  }
#pragma unroll
  for (int u = 0; u < kChunks; ++u) {
    const int c = (threadIdx.x >> 7) + u * (kPackThreads / 128);
    if (c * 16 >= klen) break;
    uint32_t o[4] = {0u, 0u, 0u, 0u};
    if (SRC == kPackCodes) {
      if (n < p.n) {
        const int32_t* src = p.codes + (size_t)(k0 + c * 16) * p.n + n;
        uint32_t q[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) q[i] = (uint32_t)__ldcs(src + (size_t)i * p.n);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          bad |= q[i] & ~kMask;
          o[i >> 2] |= (q[i] & kMask) << (8 * (i & 3));
        }
      }
    } else if constexpr (BITS == 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = w[u][i < NWORD ? i : 0];
    } else if constexpr (BITS == 4) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // even and odd nibbles as bytes, then interleaved
        const uint32_t x = w[u][i < NWORD ? i : 0], lo = x & 0x0f0f0f0fu, hi = (x >> 4) & 0x0f0f0f0fu;
        o[2 * i] = prmt(lo, hi, 0x5140u);
        o[2 * i + 1] = prmt(lo, hi, 0x7362u);
      }
    } else {
      // fields 4i .. 4i + 3 are those of byte i of the word
      const uint32_t x = w[u][0], f0 = x & 0x03030303u, f1 = (x >> 2) & 0x03030303u, f2 = (x >> 4) & 0x03030303u,
                     f3 = (x >> 6) & 0x03030303u;
      const uint32_t a = prmt(f0, f1, 0x5140u), b = prmt(f2, f3, 0x5140u), e = prmt(f0, f1, 0x7362u), d = prmt(f2, f3, 0x7362u);
      o[0] = prmt(a, b, 0x5410u);
      o[1] = prmt(a, b, 0x7632u);
      o[2] = prmt(e, d, 0x5410u);
      o[3] = prmt(e, d, 0x7632u);
    }
    *reinterpret_cast<uint4*>(s + row * kPackRow + c * 4) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  return bad ? kRangeCodes : 0u;
}

// the packed words of the staged block
template <int BITS, bool FRAG>
__device__ __forceinline__ void write_block(const PackParams& p, const uint32_t* s, int tile, int k0, int klen) {
  if (FRAG) {
    const int ksteps = p.k / 16, nks = klen >> 4;
    for (int i = threadIdx.x; i < 2 * nks * 32; i += kPackThreads) {
      const int lane = i & 31, wt = (i >> 5) >= nks ? 1 : 0, ks = (i >> 5) - wt * nks;
      const int g = lane >> 2, t = lane & 3;
      uint32_t word[BITS];
#pragma unroll
      for (int j = 0; j < BITS; ++j) word[j] = 0;
#pragma unroll
      for (int rb = 0; rb < 4; ++rb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t q4 = s[(wt * 64 + rb * 16 + h * 8 + g) * kPackRow + ks * 4 + t];
          if (BITS != 3) {  // frag_bit_of: the four k are bytes in order (8 bits) or in the order 0, 2, 1, 3
            word[frag_word_of(BITS, rb, h)] |= (BITS == 8 ? q4 : prmt(q4, 0u, 0x3120u)) << frag_bit_of(BITS, rb, h, 0);
          } else {
            // bit by bit: one of a lane's sixteen field pairs is spread over the spare bits of its three words
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint32_t q = (q4 >> (8 * kk)) & ((1u << BITS) - 1u);
#pragma unroll
              for (int b = 0; b < 3; ++b) {
                int wj = 0, bit = 0;
                frag_code_bit(3, rb, h, kk, b, &wj, &bit);
#pragma unroll
                for (int j = 0; j < BITS; ++j)
                  if (wj == j) word[j] |= ((q >> b) & 1u) << bit;
              }
            }
          }
        }
      char* base = reinterpret_cast<char*>(p.qw) + ((size_t)(tile * 2 + wt) * ksteps + (k0 >> 4) + ks) * frag_step_bytes(BITS);
      if constexpr (BITS == 4 || BITS == 8) {
#pragma unroll
        for (int j = 0; j < BITS; j += 4)
          *reinterpret_cast<uint4*>(base + frag_word_offset(BITS, lane, j)) = make_uint4(word[j], word[j + 1], word[j + 2], word[j + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < BITS; ++j) *reinterpret_cast<uint32_t*>(base + frag_word_offset(BITS, lane, j)) = word[j];
      }
    }
  } else {
    const int nv = unit_vecs(BITS), uk = unit_k(BITS);
    for (int i = threadIdx.x; i < (klen / uk) * nv * kTileRows; i += kPackThreads) {
      const int row = i & 127, v = (i >> 7) % nv, u = (i >> 7) / nv;
      const uint32_t* src = s + row * kPackRow + u * (uk / 4);
      uint32_t word[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (BITS != 3) {
          constexpr int PF = 32 / BITS;
#pragma unroll
          for (int f = 0; f < PF; ++f) {
            const int e = j * PF + field_element(BITS, f);
            word[j] |= ((src[e >> 2] >> (8 * (e & 3))) & 0xffu) << (f * BITS);
          }
        } else if (v < 2) {  // 2-bit plane: low two bits of 16 codes
#pragma unroll
          for (int f = 0; f < 16; ++f) {
            const int e = v * 64 + j * 16 + field_element(2, f);
            word[j] |= ((src[e >> 2] >> (8 * (e & 3))) & 3u) << (f * 2);
          }
        } else {  // 1-bit plane: bit 2 of 32 codes
#pragma unroll
          for (int e = 0; e < 32; ++e)
            word[j] |= ((src[(j * 32 + e) >> 2] >> (8 * (e & 3) + 2)) & 1u) << plane1_bit(e);
        }
      }
      *reinterpret_cast<uint4*>(p.qw + ((((size_t)tile * p.units + k0 / uk + u) * nv + v) * kTileRows + row) * 4) =
          make_uint4(word[0], word[1], word[2], word[3]);
    }
  }
}

// GPTQ "zero - 1" convention, clamped like the reference packer
__device__ __forceinline__ uint8_t effective_zero(int z, int bits) { return (uint8_t)min(z + 1, (1 << bits) - 1); }

template <int BITS, int SRC, bool FRAG>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(const PackParams p) {
  __shared__ __align__(16) uint32_t s[kTileRows * kPackRow];
  // (row tiles fastest: concurrent CTAs read whole rows of the source; one grid dimension, which has room for any K)
  const int tile = blockIdx.x % p.tiles, n0 = tile * kTileRows;
  const int k0 = (int)(blockIdx.x / p.tiles) * kPackK, klen = min(kPackK, p.k - k0);
  unsigned bad = stage_codes<BITS, SRC>(p, s, n0, k0, klen);
  // scales and zeros of the groups that begin in this block (at most two)
  if (p.qs) {
    const int g0 = (k0 + p.group_size - 1) / p.group_size, g1 = (k0 + klen + p.group_size - 1) / p.group_size;
    for (int i = threadIdx.x; i < (g1 - g0) * kTileRows; i += kPackThreads) {
      const int g = g0 + (i >> 7), pos = i & 127, n = n0 + (FRAG ? frag_row_of_pos(pos) : pos);
      const size_t o = ((size_t)tile * p.groups + g) * kTileRows + pos;
      p.qs[o] = n < p.n ? p.scales[(size_t)g * p.n + n] : __ushort_as_half(0);
      if (p.qz) {
        uint8_t ze = 0;
        if (n < p.n) {
          int z;
          if (SRC == kPackCodes) {
            z = p.zeros[(size_t)g * p.n + n];
            if (z < 0 || z >= (1 << BITS)) bad |= kRangeZeros;
          } else {
            constexpr int PF = 32 / BITS;
            z = (int)((p.gptq_zeros[(size_t)g * p.zero_words + n / PF] >> (n % PF * BITS)) & ((1u << BITS) - 1u));
          }
          ze = effective_zero(z, BITS);
        }
        p.qz[o] = ze;
      }
    }
  }
  if (SRC == kPackCodes && p.range_flags && bad) atomicOr(p.range_flags, bad);
  __syncthreads();
  write_block<BITS, FRAG>(p, s, tile, k0, klen);
}

template <int BITS>
static cudaError_t launch_pack_bits(const PackParams& p, cudaStream_t st) {
  const unsigned grid = (unsigned)p.tiles * ((p.k + kPackK - 1) / kPackK);
  const bool frag = p.layout == QFB_LAYOUT_FRAGMENT;
  if (p.gptq_codes) {
    if constexpr (BITS != 3) {
      if (frag) pack_kernel<BITS, kPackGptq, true><<<grid, kPackThreads, 0, st>>>(p);
      else pack_kernel<BITS, kPackGptq, false><<<grid, kPackThreads, 0, st>>>(p);
    } else {
      return cudaErrorInvalidValue;
    }
  } else {
    if (frag) pack_kernel<BITS, kPackCodes, true><<<grid, kPackThreads, 0, st>>>(p);
    else pack_kernel<BITS, kPackCodes, false><<<grid, kPackThreads, 0, st>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_pack(const PackParams& p, cudaStream_t st) {
  switch (p.bits) {
    case 2: return launch_pack_bits<2>(p, st);
    case 3: return launch_pack_bits<3>(p, st);
    case 4: return launch_pack_bits<4>(p, st);
    case 8: return launch_pack_bits<8>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

// inverse through FragCodec<BITS>::decode, the extraction the mma kernel itself runs: one thread
// per (lane, k-step, half tile)
template <int BITS>
__global__ void unpack_frag_kernel(const UnpackParams p) {
  using FC = FragCodec<BITS>;
  const int ksteps = p.k / 16;
  const long long total = (long long)p.tiles * 2 * ksteps * 32;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int lane = (int)(idx & 31);
  long long t = idx >> 5;
  const int ks = (int)(t % ksteps); t /= ksteps;
  const int wt = (int)(t & 1);
  const int tile = (int)(t >> 1);
  const int g = lane >> 2;
  const int k0 = ks * 16 + 4 * (lane & 3);
  const char* base = reinterpret_cast<const char*>(p.qw) + ((size_t)(tile * 2 + wt) * ksteps + ks) * frag_step_bytes(BITS);
  uint32_t v[BITS];
#pragma unroll
  for (int j = 0; j < BITS; ++j) v[j] = *reinterpret_cast<const uint32_t*>(base + frag_word_offset(BITS, lane, j));
  const int grp = k0 / (p.k / p.groups);
#pragma unroll
  for (int rb = 0; rb < 4; ++rb) {
    uint32_t a[4];
    FC::decode(v, rb, a);
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // h = 0: row g (registers a[0], a[2]); h = 1: row g + 8 (a[1], a[3])
      const int n = tile * kTileRows + wt * 64 + rb * 16 + h * 8 + g;
      if (n >= p.n) continue;
      const int sh = h ? FC::shift_hi(rb) : FC::shift_lo(rb);
      const uint32_t lo = a[h] >> sh, hi = a[2 + h] >> sh, m = (1u << BITS) - 1u;
      const int q[4] = {(int)(lo & m), (int)((lo >> 16) & m), (int)(hi & m), (int)((hi >> 16) & m)};
      const size_t sz = ((size_t)tile * p.groups + grp) * kTileRows + wt * 64 + g * 8 + rb * 2 + h;
      const __half sc = p.qs ? p.qs[sz] : __ushort_as_half(0x3C00);
      const int z = p.qz ? (int)p.qz[sz] : (int)p.zconst;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p.codes_out) p.codes_out[(size_t)(k0 + i) * p.n + n] = q[i];
        if (p.w_out) p.w_out[(size_t)(k0 + i) * p.n + n] = __hmul(__int2half_rn(q[i] - z), sc);
      }
    }
  }
}

template <int BITS>
__global__ void unpack_kernel(const UnpackParams p) {
  using G = Geo<BITS>;
  using C = Codec<BITS>;
  const long long total = (long long)p.tiles * p.units * kTileRows;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int r = (int)(idx % kTileRows);
  const int unit = (int)((idx / kTileRows) % p.units);
  const int tile = (int)(idx / ((long long)kTileRows * p.units));
  const int n = tile * kTileRows + r;
  if (n >= p.n) return;
  uint4 v[G::kUnitVecs];
#pragma unroll
  for (int i = 0; i < G::kUnitVecs; ++i)
    v[i] = ldg_stream_v4(p.qw + (((size_t)tile * p.units + unit) * G::kUnitVecs + i) * kTileRows + r);
  const int k0 = unit * G::kUnitK;
  if (p.codes_out) {
    const typename C::ZM zm = C::zmagic(0);
    C::unit(v, zm, [&](int j8, __half2(&d)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(d[i]);
        p.codes_out[(size_t)(k0 + j8 * 8 + 2 * i) * p.n + n] = (int32_t)f.x;
        p.codes_out[(size_t)(k0 + j8 * 8 + 2 * i + 1) * p.n + n] = (int32_t)f.y;
      }
    });
  }
  if (p.w_out) {
    const int g = unit / p.units_per_group;
    const size_t sz = ((size_t)tile * p.groups + g) * kTileRows + r;
    const __half2 s2 = __half2half2(p.qs ? p.qs[sz] : __ushort_as_half(0x3C00));
    const typename C::ZM zm = C::zmagic(p.qz ? (uint32_t)p.qz[sz] : p.zconst);
    C::unit(v, zm, [&](int j8, __half2(&d)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 w = __hmul2(d[i], s2);
        p.w_out[(size_t)(k0 + j8 * 8 + 2 * i) * p.n + n] = __low2half(w);
        p.w_out[(size_t)(k0 + j8 * 8 + 2 * i + 1) * p.n + n] = __high2half(w);
      }
    });
  }
}

// fp16 weight [K, N] -> group-wise asymmetric codes, scales and GPTQ-convention zeros, the front end
// of "construct a layer from an fp16 weight" (reference: tests/acc_gptq.py:10-29).  One thread per
// (group, column); every operation is rounded to fp16 exactly where the reference's fp16 tensor
// expression rounds (each division and product computed in fp32 and rounded once), so the result
// equals the framework expression bit for bit.
__device__ __forceinline__ __half h_div(__half a, __half b) { return __float2half_rn(__half2float(a) / __half2float(b)); }
__device__ __forceinline__ __half h_mul(__half a, float b) { return __float2half_rn(__half2float(a) * b); }

__global__ void quantize_kernel(const __half* __restrict__ w, int k, int n, int group_size, int levels,
                                int32_t* __restrict__ codes, __half* __restrict__ scales, int32_t* __restrict__ zeros) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int groups = k / group_size;
  if (idx >= (long long)groups * n) return;
  const int col = (int)(idx % n), g = (int)(idx / n);
  const __half* src = w + (size_t)g * group_size * n + col;
  __half wmax = src[0], wmin = src[0];
  for (int i = 1; i < group_size; ++i) {
    const __half v = src[(size_t)i * n];
    wmax = __hmax(wmax, v);
    wmin = __hmin(wmin, v);
  }
  const __half span = __hsub_rn(wmax, wmin);
  scales[idx] = __float2half_rn(__half2float(span) / (float)levels);
  // zero = trunc(max(-min / span * levels - 1, 0))
  const __half zf = __hsub_rn(h_mul(h_div(__hneg(wmin), span), (float)levels), __float2half_rn(1.f));
  zeros[idx] = (int32_t)__half2float(__hmax(zf, __float2half_rn(0.f)));
  for (int i = 0; i < group_size; ++i) {
    const __half q = h_mul(h_div(__hsub_rn(src[(size_t)i * n], wmin), span), (float)levels);
    codes[(size_t)(g * group_size + i) * n + col] = (int32_t)__half2float(q);
  }
}

cudaError_t launch_quantize(const __half* w, int k, int n, int bits, int group_size, int32_t* codes, __half* scales,
                            int32_t* zeros, cudaStream_t st) {
  const long long total = (long long)(k / group_size) * n;
  quantize_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(w, k, n, group_size, (1 << bits) - 1, codes, scales,
                                                                    zeros);
  return cudaGetLastError();
}

// The same quantisation straight into the packed layout: neither the int32 codes (four bytes each) nor the int32 zeros
// ever reach memory.  One CTA owns the 128 rows of a tile and one run of k: a whole group, or two groups of 64.  Thread
// (pair of rows c, quarter h) holds 32 k of its two rows of a 128-k block in registers, so a group of at most 128 is
// read once; a longer one is read a second time (from L2) after its extremes are known.
// (w - min) / span is computed as (w - min) * (1 / span), both operations rounded to fp32, then rounded to fp16.  Where
// the quotient is a normal fp16 value that equals the division's result: with a = w - min and b = span in fp16 (11-bit
// significands) the product is within 2^-23 (1 + 2^-25) of a / b, relative, while a / b stays more than that away from
// every midpoint m of two neighbouring normal values (12 bits): it is never equal to one, since m * b has at least 12
// bits, and |a - m b| is at least one unit against m b < 2^23 units.  A quotient below 2^-14 can come out one subnormal
// step off (its midpoints have fewer bits); times at most 255 levels it is less than one either way, so that the code
// is 0 and the zero point, which is that less one, is 0.
// Instruction bound at about twice the memory time: (8192,28672) 4-bit, groups of 128, 182 us for 592 MB in and out.
template <int BITS, bool FRAG>
__global__ void __launch_bounds__(kPackThreads, 4) quantize_pack_kernel(const PackParams p, int run) {
  __shared__ __align__(16) uint32_t s[kTileRows * kPackRow];
  __shared__ __half2 ext[2][4][64];   // largest and smallest value per quarter and pair of rows
  const int tile = blockIdx.x % p.tiles, n0 = tile * kTileRows;
  const int kbeg = (int)(blockIdx.x / p.tiles) * run, kend = min(kbeg + run, p.k);
  const int c = threadIdx.x & 63, h = threadIdx.x >> 6, n = n0 + 2 * c;
  // both rows exist and every row of the source is aligned to pairs (the source itself may begin at any fp16 value)
  const bool pair = n + 1 < p.n && (p.n & 1) == 0 && (reinterpret_cast<uintptr_t>(p.weight) & 3u) == 0;
  constexpr int kLevels = (1 << BITS) - 1;
  const int gs = p.group_size;
  unsigned bad = 0;
  auto fetch = [&](int k0, int klen, __half2 (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      v[i] = __half2half2(__ushort_as_half(0));
      if (h * 32 + i < klen) {
        const __half* src = p.weight + (size_t)(k0 + h * 32 + i) * p.n + n;
        if (pair) v[i] = *reinterpret_cast<const __half2*>(src);
        else if (n < p.n) v[i] = __halves2half2(src[0], n + 1 < p.n ? src[1] : src[0]);
      }
    }
  };
  __half2 v[32];
  __half2 vmax = __half2half2(__ushort_as_half(0x7E00)), vmin = vmax;   // NaN, which max and min ignore
  for (int k0 = kbeg; k0 < kend; k0 += kPackK) {
    const int klen = min(kPackK, kend - k0);
    fetch(k0, klen, v);
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (h * 32 + i < klen) {
        vmax = __hmax2(vmax, v[i]);
        vmin = __hmin2(vmin, v[i]);
      }
  }
  ext[0][h][c] = vmax;
  ext[1][h][c] = vmin;
  __syncthreads();
  // this thread's group: all four quarters, or the two quarters of its 64-k half
  const int q0 = gs == 64 ? (h & 2) : 0, q1 = gs == 64 ? q0 + 2 : 4;
  vmax = ext[0][q0][c];
  vmin = ext[1][q0][c];
  for (int q = q0 + 1; q < q1; ++q) {
    vmax = __hmax2(vmax, ext[0][q][c]);
    vmin = __hmin2(vmin, ext[1][q][c]);
  }
  const __half2 span = __halves2half2(__hsub_rn(__low2half(vmax), __low2half(vmin)), __hsub_rn(__high2half(vmax), __high2half(vmin)));
  const float2 fspan = __half22float2(span);
  const float inv[2] = {1.f / fspan.x, 1.f / fspan.y};
  auto ratio = [&](__half2 a) {
    const float2 f = __half22float2(a);
    return __floats2half2_rn(__fmul_rn(f.x, inv[0]), __fmul_rn(f.y, inv[1]));
  };
  const __half2 levels2 = __float2half2_rn((float)kLevels);   // (an fp16 value times it is exact in fp32: one rounding either way)
  // the group's scale and zero: written by the first quarter of the group (both rows)
  const int grp = (kbeg + (gs == 64 ? (h >> 1) * 64 : 0)) / gs;
  if (h == q0 && (gs != 64 || kbeg + (h >> 1) * 64 < kend)) {
    // zero = trunc(max(-min / span * levels - 1, 0))
    const __half2 zf = __hsub2_rn(__hmul2_rn(ratio(__hneg2(vmin)), levels2), __float2half2_rn(1.f));
    const __half2 zh = __hmax2(zf, __float2half2_rn(0.f));
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = 2 * c + e;
      const size_t o = ((size_t)tile * p.groups + grp) * kTileRows + (FRAG ? frag_pos_of_row(row) : row);
      const bool valid = n + e < p.n;
      const int z = (int32_t)(e ? __high2float(zh) : __low2float(zh));
      if (valid && (z < 0 || z > kLevels)) bad |= kRangeZeros;
      p.qs[o] = valid ? __float2half_rn((e ? fspan.y : fspan.x) / (float)kLevels) : __ushort_as_half(0);
      p.qz[o] = valid ? effective_zero(z, BITS) : (uint8_t)0;
    }
  }
  for (int k0 = kbeg; k0 < kend; k0 += kPackK) {
    const int klen = min(kPackK, kend - k0);
    if (run > kPackK) fetch(k0, klen, v);   // (one block: still in registers)
    // code = trunc((w - min) / span * levels), never out of range: w - min <= span in fp16 too, and a NaN (0 / 0, an
    // infinity) becomes 0 as in a float-to-integer conversion.  The integer part is read from the low bits of a sum
    // with 2^23 rounded towards zero: a conversion instruction per code runs at an eighth of the rate.
#pragma unroll
    for (int i0 = 0; i0 < 32; i0 += 16) {
      if (h * 32 + i0 < klen) {
        uint32_t o[2][4];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          uint32_t q[2][4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __half2 r = ratio(__hsub2_rn(v[i0 + i + j], vmin));
            const float2 f = __half22float2(__hmax2(__hmul2_rn(r, levels2), __float2half2_rn(0.f)));
            q[0][j] = __float_as_uint(__fadd_rz(f.x, 8388608.f));
            q[1][j] = __float_as_uint(__fadd_rz(f.y, 8388608.f));
          }
#pragma unroll
          for (int e = 0; e < 2; ++e)
            o[e][i >> 2] = n + e < p.n ? prmt(prmt(q[e][0], q[e][1], 0x0040u), prmt(q[e][2], q[e][3], 0x0040u), 0x5410u) : 0u;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<uint4*>(s + (2 * c + e) * kPackRow + h * 8 + i0 / 4) = make_uint4(o[e][0], o[e][1], o[e][2], o[e][3]);
      }
    }
    __syncthreads();
    write_block<BITS, FRAG>(p, s, tile, k0, klen);
    __syncthreads();
  }
  if (bad) atomicOr(p.range_flags, bad);
}

template <int BITS>
static cudaError_t launch_quantize_pack_bits(const PackParams& p, cudaStream_t st) {
  const int run = p.group_size == 64 ? 128 : p.group_size;
  const unsigned grid = (unsigned)p.tiles * ((p.k + run - 1) / run);
  if (p.layout == QFB_LAYOUT_FRAGMENT) quantize_pack_kernel<BITS, true><<<grid, kPackThreads, 0, st>>>(p, run);
  else quantize_pack_kernel<BITS, false><<<grid, kPackThreads, 0, st>>>(p, run);
  return cudaGetLastError();
}

cudaError_t launch_quantize_pack(const PackParams& p, cudaStream_t st) {
  switch (p.bits) {
    case 2: return launch_quantize_pack_bits<2>(p, st);
    case 3: return launch_quantize_pack_bits<3>(p, st);
    case 4: return launch_quantize_pack_bits<4>(p, st);
    case 8: return launch_quantize_pack_bits<8>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_unpack(const UnpackParams& p, cudaStream_t st) {
  if (p.layout == QFB_LAYOUT_FRAGMENT) {
    const int block = 256;
    const long long tf = (long long)p.tiles * 2 * (p.k / 16) * 32;
    const unsigned gridf = (unsigned)((tf + block - 1) / block);
    if (p.bits == 4) unpack_frag_kernel<4><<<gridf, block, 0, st>>>(p);
    else if (p.bits == 8) unpack_frag_kernel<8><<<gridf, block, 0, st>>>(p);
    else if (p.bits == 2) unpack_frag_kernel<2><<<gridf, block, 0, st>>>(p);
    else if (p.bits == 3) unpack_frag_kernel<3><<<gridf, block, 0, st>>>(p);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
  }
  const long long total = (long long)p.tiles * p.units * kTileRows;
  const int block = 128;
  const unsigned grid = (unsigned)((total + block - 1) / block);
  switch (p.bits) {
    case 2: unpack_kernel<2><<<grid, block, 0, st>>>(p); break;
    case 3: unpack_kernel<3><<<grid, block, 0, st>>>(p); break;
    case 4: unpack_kernel<4><<<grid, block, 0, st>>>(p); break;
    case 8: unpack_kernel<8><<<grid, block, 0, st>>>(p); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace qfb
