// gf2cuda DVB-T2 outer BCH code (sm_100a): batch encoder and decoder.
//
// The reference's binary BCH outer code of DVB-T2 (crates/gf2-coding/src/bch):
//   parameters DvbBchParams::for_code          bch/dvb_t2/params.rs:56-85
//   generator g = g_1 ... g_t                  bch/dvb_t2/generators.rs:14-62
//   BchEncoder::encode: [message | parity], bit i at polynomial degree n-1-i,
//     parity = x^r m(x) mod g(x)               bch/core.rs:421-480
//   BchDecoder::decode: syndromes S_j = r(alpha^j), j = 1..2t; all zero ->
//     the received message; else Berlekamp-Massey, Chien search over
//     alpha^-i, flip bit n-1-i for every root i, first k bits
//                                            bch/core.rs:562-818
// alpha = x in GF(2^m) modulo the DVB-T2 primitive polynomial.
//
// GPU layout: one warp per frame.
//  * Odd syndromes S_j, j = 2s+1 < 2t (shared by encoder and decoder):
//    S_j = alpha^(j(n-1)) sum_i b_i beta^i, beta = alpha^-j.  Lane l takes the
//    64-bit words w = l + 32u (coalesced) and runs Horner over u from the top,
//    acc <- acc * beta^2048 + q_w, where q_w = sum over the word's 8 bytes of a
//    per-(byte position, value) table entry that packs four syndromes in 8
//    bytes; the multiply by the constant beta^2048 is two byte lookups.  The
//    lane's sum is scaled by alpha^(j(n-1-64l)) and XOR-reduced over the warp.
//    All tables live in shared memory.  Even syndromes are squares:
//    S_(2^a o) = S_o^(2^a) for a binary received word.
//  * Encoder: the odd syndromes of [message | 0] fix the parity, because the
//    map from the r parity bits to the r = t m odd-syndrome bits is invertible
//    (g is the product of the minimal polynomials of alpha^j, j odd < 2t).
//    parity = A s with A the inverse of that GF(2) matrix (host-built); it
//    equals x^r m(x) mod g, the unique systematic parity.
//  * Decoder, kernel 1: syndromes, the message copy, and the reference's
//    Berlekamp-Massey step for step with lane i holding coefficient i of the
//    locator and of the correction polynomial (the discrepancy is a warp XOR
//    reduction).  It stores the locator as logarithms per frame.
//  * Decoder, kernel 2 (Chien search): the antilog table of the field in
//    shared memory, stored with an offset so that the exponents are reduced
//    mod N once per 8 position steps and the steps in between are constant
//    load offsets; lane l evaluates positions i = l + 32s with the terms'
//    exponents in registers (locator degrees 3..12 unrolled); a root i flips
//    bit n-1-i when it lies in the message.  Bound by the table loads (one per
//    term and position, shared memory 91 % busy), so a root found is divided
//    out of the locator (the rest of the scan has a term less) and a locator of
//    degree 2 or 1 is solved in closed form; both give the same root set as the
//    full search.  Kernel 1 files each frame under its locator
//    degree; kernel 2 takes the frames degree by degree, highest first.
#include <algorithm>
#include <cstring>
#include <memory>
#include <utility>
#include <vector>

#include "bits.cuh"
#include "internal.h"

namespace gf2c {

static constexpr int kBchWarps = 8;          // warps per CTA in the syndrome kernels
static constexpr int kChienThreads = 1024;   // Chien kernel CTA size
static constexpr int kChienFastMax = 12;     // locator degrees with an unrolled evaluator
static constexpr int kChienSeg = 8;          // positions steps between exponent reductions
static constexpr int kChienUnroll = 2;      // position steps unrolled
static constexpr int kChienOff = 32 * kChienFastMax * kChienSeg;  // antilog table offset
static constexpr uint16_t kLogZero = 0xFFFF; // stored log of a zero coefficient

// ETSI EN 302 755 generator factors g_1..g_12 (exponent lists of binary
// polynomials; standard data).
constexpr int kShortGen[12][12] = {
    {0, 1, 3, 5, 14, -1},          {0, 6, 8, 11, 14, -1},         {0, 1, 2, 6, 9, 10, 14, -1},
    {0, 4, 7, 8, 10, 12, 14, -1},  {0, 2, 4, 6, 8, 9, 11, 13, 14, -1}, {0, 3, 7, 8, 9, 13, 14, -1},
    {0, 2, 5, 6, 7, 10, 11, 13, 14, -1}, {0, 5, 8, 9, 10, 11, 14, -1}, {0, 1, 2, 3, 9, 10, 14, -1},
    {0, 3, 6, 9, 11, 12, 14, -1},  {0, 4, 11, 12, 14, -1},        {0, 1, 2, 3, 5, 6, 7, 8, 10, 13, 14, -1}};
constexpr int kNormalGen[12][14] = {
    {0, 2, 3, 5, 16, -1},
    {0, 1, 4, 5, 6, 8, 16, -1},
    {0, 2, 3, 4, 5, 7, 8, 9, 10, 11, 16, -1},
    {0, 2, 4, 6, 9, 11, 12, 14, 16, -1},
    {0, 1, 2, 3, 5, 8, 9, 10, 11, 12, 16, -1},
    {0, 2, 4, 5, 7, 8, 9, 10, 12, 13, 14, 15, 16, -1},
    {0, 2, 5, 6, 8, 9, 10, 11, 13, 15, 16, -1},
    {0, 1, 2, 5, 6, 8, 9, 12, 13, 14, 16, -1},
    {0, 5, 7, 9, 10, 11, 16, -1},
    {0, 1, 2, 5, 7, 8, 10, 12, 13, 14, 16, -1},
    {0, 2, 3, 5, 9, 11, 12, 13, 16, -1},
    {0, 1, 5, 6, 7, 9, 11, 12, 16, -1}};

__host__ __device__ constexpr uint32_t factor_mask(const int* exponents) {
  uint32_t m = 0;
  for (int i = 0; exponents[i] >= 0; i++) m |= 1u << exponents[i];
  return m;
}

struct BchDev {
  int n, k, t, r, m, N, words_n, words_k, rw;  // rw = 32-bit words of the parity
  const uint16_t* exp;   // [2N]
  const uint16_t* log;   // [N + 1]
  const uint16_t* half;  // [N + 1]: half[c] = a root of z^2 + z = c, 0 where there is none (or c = 0)
  const uint2* quad;     // [3][8][256]: 4 odd syndromes per entry, byte position p
  const uint16_t* mul;   // [t][512]: (v * gamma_s), (v << 8) * gamma_s
  const uint32_t* lf;    // [t][32]: exponent of alpha^(j(n-1-64 lane)) mod N
  const uint32_t* acol;  // [r][rw]: parity pattern of syndrome bit b
  const uint16_t* lane_mul;  // [t][512]: product with alpha^-j in the basis of powers of alpha^(32 j)
  const uint16_t* lane_out;  // [t][512]: field element of a vector in that basis, times alpha^(j(n-1-32(steps-1)))
};

// shared-memory image of the syndrome tables
struct SynTab {
  const uint2* quad;
  const uint16_t* mul;
  const uint32_t* lf;
};

__device__ __forceinline__ uint32_t gf_mul(const BchDev& B, uint32_t a, uint32_t b) {
  if (!a || !b) return 0;
  return __ldg(&B.exp[__ldg(&B.log[a]) + __ldg(&B.log[b])]);
}

__device__ __forceinline__ uint32_t warp_xor(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v ^= __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Stage the syndrome tables into shared memory; returns the end of the area.
template <int T>
__device__ __forceinline__ SynTab load_syn_tables(const BchDev& B, unsigned char* smem) {
  uint2* q = (uint2*)smem;
  uint16_t* mu = (uint16_t*)(q + 3 * 8 * 256);
  uint32_t* lf = (uint32_t*)(mu + T * 512);
  for (int i = threadIdx.x; i < 3 * 8 * 256; i += blockDim.x) q[i] = B.quad[i];
  for (int i = threadIdx.x; i < T * 512; i += blockDim.x) mu[i] = B.mul[i];
  for (int i = threadIdx.x; i < T * 32; i += blockDim.x) lf[i] = B.lf[i];
  return SynTab{q, mu, lf};
}

template <int T>
__host__ __device__ constexpr size_t syn_smem_bytes() {
  return (size_t)3 * 8 * 256 * 8 + (size_t)T * 512 * 2 + (size_t)T * 32 * 4;
}

// Odd syndromes S_(2s+1), s < T, of the first `nbits` bits of the packed frame
// `c` (the remaining codeword bits zero); every lane returns all T values.
// Words below `copy_words` are also written to `copy` (the last one masked to
// `copy_bits`).
template <int T>
__device__ __forceinline__ void odd_syndromes(const BchDev& B, const SynTab& S, const uint64_t* __restrict__ c,
                                              int nbits, uint64_t* __restrict__ copy, int copy_bits, int lane,
                                              uint32_t so[T]) {
  const int nwords = (nbits + 63) >> 6;
  const int cwords = (copy_bits + 63) >> 6;
  uint32_t acc[T];
#pragma unroll
  for (int s = 0; s < T; s++) acc[s] = 0;
  const int U = (nwords + 31) >> 5;
  for (int u = U - 1; u >= 0; u--) {
    const int w = lane + 32 * u;
    uint64_t word = 0;
    if (w < nwords) {
      word = __ldg(&c[w]);
      if (copy && w < cwords) copy[w] = (w == cwords - 1 && (copy_bits & 63)) ? word & ((1ull << (copy_bits & 63)) - 1ull) : word;
      if (w == nwords - 1 && (nbits & 63)) word &= (1ull << (nbits & 63)) - 1ull;
    }
#pragma unroll
    for (int s = 0; s < T; s++) {
      const uint32_t a = acc[s];
      acc[s] = (uint32_t)S.mul[s * 512 + (a & 0xffu)] ^ (uint32_t)S.mul[s * 512 + 256 + (a >> 8)];
    }
    if (word) {
      const uint32_t lo = (uint32_t)word, hi = (uint32_t)(word >> 32);
#pragma unroll
      for (int q = 0; q < (T + 3) / 4; q++) {
        uint32_t x0 = 0, x1 = 0;
#pragma unroll
        for (int p = 0; p < 8; p++) {
          const uint32_t v = ((p < 4 ? lo : hi) >> (8 * (p & 3))) & 0xffu;
          const uint2 e = S.quad[(q * 8 + p) * 256 + v];
          x0 ^= e.x;
          x1 ^= e.y;
        }
        if (4 * q + 0 < T) acc[4 * q + 0] ^= x0 & 0xffffu;
        if (4 * q + 1 < T) acc[4 * q + 1] ^= x0 >> 16;
        if (4 * q + 2 < T) acc[4 * q + 2] ^= x1 & 0xffffu;
        if (4 * q + 3 < T) acc[4 * q + 3] ^= x1 >> 16;
      }
    }
  }
  // scale by alpha^(j(n-1-64 lane)), then reduce two syndromes per shuffle
#pragma unroll
  for (int s = 0; s < T; s++)
    acc[s] = acc[s] ? __ldg(&B.exp[__ldg(&B.log[acc[s]]) + S.lf[s * 32 + lane]]) : 0u;
#pragma unroll
  for (int s = 0; s < T; s += 2) {
    uint32_t v = acc[s] | (s + 1 < T ? acc[s + 1] << 16 : 0u);
    v = warp_xor(v);
    so[s] = v & 0xffffu;
    if (s + 1 < T) so[s + 1] = v >> 16;
  }
}

template <int T>
__global__ void __launch_bounds__(kBchWarps * 32) bch_encode_kernel(const BchDev B, const uint64_t* __restrict__ msg,
                                                                    long long frames, uint64_t* __restrict__ cw) {
  extern __shared__ __align__(16) unsigned char smem[];
  const SynTab S = load_syn_tables<T>(B, smem);
  uint32_t* par_s = (uint32_t*)(smem + syn_smem_bytes<T>());  // [warps][8]
  uint16_t* syn_s = (uint16_t*)(par_s + kBchWarps * 8);         // [warps][16]
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t* par = par_s + wib * 8;
  uint16_t* sy = syn_s + wib * 16;
  const long long warps = (long long)gridDim.x * kBchWarps;
  for (long long f = (long long)blockIdx.x * kBchWarps + wib; f < frames; f += warps) {
    const uint64_t* m = msg + f * B.words_k;
    uint64_t* c = cw + f * B.words_n;
    uint32_t so[T];
    odd_syndromes<T>(B, S, m, B.k, c, B.k, lane, so);
#pragma unroll
    for (int s = 0; s < T; s++)
      if (lane == s) sy[s] = (uint16_t)so[s];
    __syncwarp();
    // parity = A s: lane takes syndrome bits b = lane + 32 z
    uint32_t p[6] = {0, 0, 0, 0, 0, 0};
    for (int b = lane; b < B.r; b += 32) {
      if ((sy[b / B.m] >> (b % B.m)) & 1u) {
        const uint32_t* col = B.acol + (size_t)b * B.rw;
#pragma unroll
        for (int q = 0; q < 6; q++)
          if (q < B.rw) p[q] ^= __ldg(&col[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 6; q++) p[q] = warp_xor(p[q]);
    uint32_t mine = 0;
#pragma unroll
    for (int q = 0; q < 6; q++)
      if (lane == q) mine = p[q];
    if (lane < 8) par[lane] = mine;
    __syncwarp();
    // codeword words from bit k on: parity bit q sits at codeword bit k + q
    for (int w = (B.k >> 6) + lane; w < B.words_n; w += 32) {
      const int o = 64 * w - B.k;  // parity bit at the word's bit 0 (negative in the message's tail word)
      uint64_t word;
      if (o >= 0) {
        const int q0 = o >> 5, sh = o & 31;
        const uint64_t lo = ((uint64_t)par[q0 + 1] << 32) | par[q0];
        const uint64_t hi = q0 + 2 < 8 ? par[q0 + 2] : 0u;
        word = sh ? (lo >> sh) | (hi << (64 - sh)) : lo;
      } else {
        const uint64_t low = ((uint64_t)par[1] << 32) | par[0];
        word = (m[w] & ((1ull << (B.k & 63)) - 1ull)) | (low << (-o));
      }
      if (w == B.words_n - 1 && (B.n & 63)) word &= (1ull << (B.n & 63)) - 1ull;
      c[w] = word;
    }
    __syncwarp();
  }
}

// Berlekamp-Massey of frame f from its odd syndromes (sS[2 s] = S_(2s+1), any =
// their OR): even syndromes, locator logarithms, degree, Chien work list.
template <int T>
__device__ __forceinline__ void bch_locator(const BchDev& B, uint16_t* sS, uint32_t any, long long f, long long frames,
                                            int lane, int32_t* __restrict__ nflips, uint16_t* __restrict__ synd_out,
                                            uint16_t* __restrict__ loc, int32_t* __restrict__ degs,
                                            uint32_t* __restrict__ bcnt, int32_t* __restrict__ blist) {
  // even syndromes: S_(2^a o) = S_o^(2^a)
  uint32_t ev = 0;
  const int j = lane + 1;
  const bool even = lane < 2 * T && !(j & 1);
  if (even) {
    const int a = __ffs(j) - 1;
    const uint32_t so_ = sS[(j >> a) - 1];
    ev = so_ ? __ldg(&B.exp[((uint32_t)__ldg(&B.log[so_]) << a) % (uint32_t)B.N]) : 0u;
  }
  __syncwarp();
  if (even) sS[lane] = (uint16_t)ev;
  __syncwarp();
  if (synd_out && lane < 2 * T) synd_out[f * 2 * T + lane] = sS[lane];
  if (!any) {
    if (lane == 0) {
      degs[f] = 0;
      if (nflips) nflips[f] = 0;
    }
    __syncwarp();
    return;
  }
  // Berlekamp-Massey: lane i holds lambda_i and b_i
  uint32_t lam = lane == 0, bb = lane == 0;
  int l = 0, mm = 1;
  for (int nn = 0; nn < 2 * T; nn++) {
    uint32_t prod = 0;
    if (lane == 0) prod = sS[nn];
    else if (lane <= l && lane <= nn) prod = gf_mul(B, lam, sS[nn - lane]);
    const uint32_t delta = warp_xor(prod);
    if (delta == 0) {
      mm += 1;
      continue;
    }
    const uint32_t tl = lam;
    const uint32_t bsh = __shfl_up_sync(0xffffffffu, bb, mm);
    if (lane >= mm) lam ^= gf_mul(B, delta, bsh);
    if (2 * l <= nn) {
      l = nn + 1 - l;
      const uint32_t di = __ldg(&B.exp[(B.N - __ldg(&B.log[delta])) % B.N]);
      bb = gf_mul(B, tl, di);
      mm = 1;
    } else {
      mm += 1;
    }
  }
  const int deg = 31 - __clz(__ballot_sync(0xffffffffu, lam != 0));
  const bool zero_coef = __any_sync(0xffffffffu, lane >= 1 && lane <= deg && lam == 0);
  loc[f * 32 + lane] = lam ? __ldg(&B.log[lam]) : kLogZero;
  if (lane == 0) {
    degs[f] = deg;
    if (deg == 0) {
      if (nflips) nflips[f] = 0;
    } else {  // Chien work list of the frame's bucket: its degree, or 0 for the generic evaluator
      const int bk = (deg <= kChienFastMax && !zero_coef) ? deg : 0;
      const uint32_t pos = atomicAdd(&bcnt[bk], 1u);
      blist[(size_t)bk * frames + pos] = (int32_t)f;
    }
  }
}

// Kernel 1 of the decoder for small batches: syndromes, message copy, Berlekamp-Massey.
template <int T>
__global__ void __launch_bounds__(kBchWarps * 32) bch_syndrome_bm_kernel(
    const BchDev B, const uint64_t* __restrict__ cw, long long frames, uint64_t* __restrict__ msg,
    int32_t* __restrict__ nflips, uint16_t* __restrict__ synd_out, uint16_t* __restrict__ loc,
    int32_t* __restrict__ degs, uint32_t* __restrict__ bcnt, int32_t* __restrict__ blist) {
  extern __shared__ __align__(16) unsigned char smem[];
  const SynTab S = load_syn_tables<T>(B, smem);
  uint16_t* syn_s = (uint16_t*)(smem + syn_smem_bytes<T>());  // [warps][32]
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint16_t* sS = syn_s + wib * 32;
  const long long warps = (long long)gridDim.x * kBchWarps;
  for (long long f = (long long)blockIdx.x * kBchWarps + wib; f < frames; f += warps) {
    uint32_t so[T];
    odd_syndromes<T>(B, S, cw + f * B.words_n, B.n, msg + f * B.words_k, B.k, lane, so);
    uint32_t any = 0;
#pragma unroll
    for (int s = 0; s < T; s++) {
      any |= so[s];
      if (lane == s) sS[2 * s] = (uint16_t)so[s];
    }
    __syncwarp();
    bch_locator<T>(B, sS, any, f, frames, lane, nflips, synd_out, loc, degs, bcnt, blist);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Syndromes of large batches, bit-sliced over 32 frames.  A 32 x 32 bit transpose
// turns word w of 32 frames into lane c holding bit 32 w + c of the frames.  For
// lane c, sum_w b_(32w+c) eta^(steps-1-w) with eta = alpha^(32 j) is Horner's rule
// in eta, and eta, a conjugate of alpha^j, has the same minimal polynomial: so
// the state is a shift register modulo the generator factor g_j, one word (32
// frames) per bit, advanced eight steps at a time (the eight bits shifted out
// are fed back by their powers' remainders: XORs of two of 2 x 16 combinations).
// A CTA takes 32 frames; its four warps load the rows coalesced, copy the
// message, share the transposed words through shared memory and take a quarter
// of the factors each.  At the end the states are transposed back and lane f
// combines the 32 states of frame f by Horner's rule in alpha^-j.  The odd
// syndromes go to the locator rows, where bch_locator_kernel takes them.
//
// Bound by issue and the planes' shared-memory loads (16384 normal 3/5 frames:
// issue slots 49 % busy at 12 warps per SM, short scoreboard 1.5 stalls per
// issue); the table kernel above is bound by its shared-memory lookups (L1 94 %).
// 65536 normal 3/5 frames, syndromes and Berlekamp-Massey: 1.23 -> 0.50 + 0.145 ms.
// One kernel with Berlekamp-Massey at the end was slower than the table kernel:
// few warps per SM run it for eight frames one after another (short 3/5, 65536
// frames, whole decode: 1.60 ms against 1.23, this one 0.95).
// ---------------------------------------------------------------------------
static constexpr int kSliceThreads = 128;

// x^e modulo the polynomial `poly` of degree M.
__host__ __device__ constexpr uint32_t x_power(uint32_t poly, int M, int e) {
  uint32_t v = 1;
  for (int i = 0; i < e; i++) {
    v <<= 1;
    if (v >> M & 1u) v ^= poly;
  }
  return v;
}
// Which of the eight bits shifted out feed bit i: bit k for x^(M + k).
__host__ __device__ constexpr uint32_t feed_mask(uint32_t poly, int M, int i) {
  uint32_t m = 0;
  for (int k = 0; k < 8; k++) m |= (x_power(poly, M, M + k) >> i & 1u) << k;
  return m;
}

template <int M, uint32_t POLY>
struct SlicedLfsr {
  uint32_t s[16];
  template <int I>
  static __device__ __forceinline__ uint32_t fed(const uint32_t (&lo)[16], const uint32_t (&hi)[16]) {
    constexpr uint32_t m = feed_mask(POLY, M, I);
    return lo[m & 15u] ^ hi[m >> 4];
  }
  template <int... I>
  __device__ __forceinline__ void advance(const uint32_t (&b)[8], std::integer_sequence<int, I...>) {
    uint32_t lo[16], hi[16];
    lo[0] = hi[0] = 0u;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int c = 0; c < 1 << k; c++) {
        lo[(1 << k) + c] = lo[c] ^ s[M - 8 + k];
        hi[(1 << k) + c] = hi[c] ^ s[M - 4 + k];
      }
    const uint32_t n[] = {((I >= 8 ? s[I >= 8 ? I - 8 : 0] : b[I < 8 ? 7 - I : 0]) ^ fed<I>(lo, hi))...};
#pragma unroll
    for (int i = 0; i < M; i++) s[i] = n[i];
  }
  __device__ __forceinline__ void step8(const uint32_t (&b)[8]) { advance(b, std::make_integer_sequence<int, M>{}); }
};

// The factors FIRST .. FIRST + COUNT - 1 of one warp.
template <int M, int FIRST, int COUNT>
struct SlicedGroup {
  static constexpr uint32_t poly(int i) { return factor_mask(M == 16 ? kNormalGen[FIRST + i] : kShortGen[FIRST + i]); }
  SlicedLfsr<M, poly(0)> a;
  SlicedLfsr<M, poly(COUNT > 1 ? 1 : 0)> b;
  SlicedLfsr<M, poly(COUNT > 2 ? 2 : 0)> c;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 16; i++) a.s[i] = b.s[i] = c.s[i] = 0u;
  }
  __device__ __forceinline__ void step8(const uint32_t (&w)[8]) {
    a.step8(w);
    if (COUNT > 1) b.step8(w);
    if (COUNT > 2) c.step8(w);
  }
};

// Row pitch (16-bit states) of one (factor, frame): odd in 32-bit words.
static constexpr int kStatePitch = 34;

// One step of the 16 x 16 bit transpose of both halves of s (a template, so that
// every index is known and s stays in registers).
template <int J, uint32_t MASK>
__device__ __forceinline__ void transpose_step(uint32_t (&s)[16]) {
#pragma unroll
  for (int k = 0; k < 16; k++)
    if (!(k & J)) {
      const uint32_t t = ((s[k] >> J) ^ s[k + J < 16 ? k + J : 0]) & MASK;
      s[k + J < 16 ? k + J : 0] ^= t;
      s[k] ^= t << J;
    }
}

// State words (bit planes over frames) -> states[(factor * 32 + frame) * pitch + lane].
__device__ __forceinline__ void store_states(uint32_t (&s)[16], uint16_t* states, int factor, int lane) {
  transpose_step<8, 0x00ff00ffu>(s);
  transpose_step<4, 0x0f0f0f0fu>(s);
  transpose_step<2, 0x33333333u>(s);
  transpose_step<1, 0x55555555u>(s);
  uint16_t* p = states + (size_t)factor * 32 * kStatePitch + lane;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    p[k * kStatePitch] = (uint16_t)s[k];
    p[(16 + k) * kStatePitch] = (uint16_t)(s[k] >> 16);
  }
}

// Shared memory: one block of rows, its transposed words, states, lane products.
static constexpr int kTilePitch = 33;
template <int T>
__host__ __device__ constexpr size_t slice_smem_bytes() {
  return (size_t)T * 1024 + 32 * 32 * 4 + 32 * kTilePitch * 4 + (size_t)T * 32 * kStatePitch * 2;
}
__host__ __device__ inline int slice_steps(int n) { return ((n + 31) / 32 + 31) / 32 * 32; }

// Low bits of 32-bit word w that a row of `bits` bits holds.
__device__ __forceinline__ uint32_t word_mask(int bits, int w) {
  const int left = bits - 32 * w;
  return left >= 32 ? ~0u : left > 0 ? (1u << left) - 1u : 0u;
}

// Barrier of a sliced CTA's warps.  They meet from different instances of
// sliced_pass, where __syncthreads() may not stand: it asks every thread of the
// CTA to reach the same barrier of the source.  A PTX barrier counts the threads
// that arrive at its number, wherever they arrive from.
__device__ __forceinline__ void slice_sync() {
  asm volatile("barrier.cta.sync.aligned 1, %0;" ::"n"(kSliceThreads) : "memory");
}

// One warp's factors over the whole frames; every warp of the CTA takes the same
// number of barriers.
template <int M, int FIRST, int COUNT>
__device__ __forceinline__ void sliced_pass(const BchDev& B, const uint64_t* __restrict__ cw,
                                            uint64_t* __restrict__ msg, long long f0, int nf, uint32_t* planes,
                                            uint32_t* tile, uint16_t* states, int warp, int lane) {
  SlicedGroup<M, FIRST, COUNT> g;
  g.clear();
  const Transpose32 tr(lane);
  const int blocks = slice_steps(B.n) >> 5, win = 2 * B.words_n, wout = 2 * B.words_k;
  const uint32_t* in = (const uint32_t*)(cw + (f0 + 8 * warp) * B.words_n) + lane;
  uint32_t* out = (uint32_t*)(msg + (f0 + 8 * warp) * B.words_k) + lane;
  const int rows = nf - 8 * warp;  // rows of this warp that exist: i < rows
  uint32_t x[8];
  auto fetch = [&](int blk) {
#pragma unroll
    for (int i = 0; i < 8; i++)
      x[i] = i < rows && 32 * blk + lane < win ? __ldg(in + (long long)i * win + 32 * blk) : 0u;
  };
  fetch(0);
  for (int blk = 0; blk < blocks; blk++) {
    const int w = 32 * blk + lane;
    const uint32_t mn = word_mask(B.n, w), mk = word_mask(B.k, w);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      tile[(8 * warp + i) * kTilePitch + lane] = x[i] & mn;
      if (i < rows && w < wout) out[(long long)i * wout + 32 * blk] = x[i] & mk;
    }
    if (blk + 1 < blocks) fetch(blk + 1);
    slice_sync();  // tile written; the last block's planes read
#pragma unroll
    for (int i = 0; i < 8; i++) planes[(8 * warp + i) * 32 + lane] = tr(tile[lane * kTilePitch + 8 * warp + i]);
    slice_sync();  // planes written, tile read
#pragma unroll 1
    for (int w0 = 0; w0 < 32; w0 += 8) {
      uint32_t b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) b[i] = planes[(w0 + i) * 32 + lane];
      g.step8(b);
    }
  }
  store_states(g.a.s, states, FIRST, lane);
  if (COUNT > 1) store_states(g.b.s, states, FIRST + 1, lane);
  if (COUNT > 2) store_states(g.c.s, states, FIRST + 2, lane);
}

template <int T, int M>
__global__ void __launch_bounds__(kSliceThreads, 4) bch_sliced_kernel(
    const BchDev B, const uint64_t* __restrict__ cw, long long frames, uint64_t* __restrict__ msg,
    uint16_t* __restrict__ loc) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* mul = (uint16_t*)smem;
  uint32_t* planes = (uint32_t*)(smem + T * 1024);
  uint32_t* tile = planes + 32 * 32;
  uint16_t* states = (uint16_t*)(tile + 32 * kTilePitch);
  for (int i = threadIdx.x; i < T * 64; i += kSliceThreads) ((uint4*)mul)[i] = __ldg((const uint4*)B.lane_mul + i);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long f0 = (long long)blockIdx.x * 32; f0 < frames; f0 += (long long)gridDim.x * 32) {
    const int nf = (int)min(32ll, frames - f0);
    switch (warp) {  // 12 factors: 3 per warp; 10: 3, 3, 2, 2
      case 0: sliced_pass<M, 0, 3>(B, cw, msg, f0, nf, planes, tile, states, warp, lane); break;
      case 1: sliced_pass<M, 3, 3>(B, cw, msg, f0, nf, planes, tile, states, warp, lane); break;
      case 2: sliced_pass<M, 6, T == 12 ? 3 : 2>(B, cw, msg, f0, nf, planes, tile, states, warp, lane); break;
      default: sliced_pass<M, T == 12 ? 9 : 8, T == 12 ? 3 : 2>(B, cw, msg, f0, nf, planes, tile, states, warp, lane);
    }
    __syncthreads();
    for (int s = warp; s < T; s += kSliceThreads / 32) {  // lane = frame
      const uint16_t* st = states + (s * 32 + lane) * kStatePitch;
      const uint16_t* mu = mul + s * 512;
      uint32_t acc = 0;
#pragma unroll 4
      for (int c = 31; c >= 0; c--) acc = (uint32_t)mu[acc & 0xffu] ^ (uint32_t)mu[256 + (acc >> 8)] ^ (uint32_t)st[c];
      const uint16_t* ou = B.lane_out + s * 512;
      if (lane < nf) loc[(f0 + lane) * 32 + s] = (uint16_t)(__ldg(&ou[acc & 0xffu]) ^ __ldg(&ou[256 + (acc >> 8)]));
    }
    __syncthreads();
  }
}

// Berlekamp-Massey behind bch_sliced_kernel: a warp per frame, at full occupancy
// (bound by the latency of the logarithm lookups).
template <int T>
__global__ void __launch_bounds__(kBchWarps * 32) bch_locator_kernel(
    const BchDev B, long long frames, int32_t* __restrict__ nflips, uint16_t* __restrict__ synd_out, uint16_t* loc,
    int32_t* __restrict__ degs, uint32_t* __restrict__ bcnt, int32_t* __restrict__ blist) {
  __shared__ uint16_t syn[kBchWarps][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  for (long long f = (long long)blockIdx.x * kBchWarps + wib; f < frames; f += (long long)gridDim.x * kBchWarps) {
    const uint32_t v = lane < T ? loc[f * 32 + lane] : 0u;
    if (lane < T) syn[wib][2 * lane] = (uint16_t)v;
    __syncwarp();
    bch_locator<T>(B, syn[wib], __any_sync(0xffffffffu, v != 0), f, frames, lane, nflips, synd_out, loc, degs, bcnt,
                   blist);
    __syncwarp();
  }
}

__device__ __forceinline__ void flip_root(const BchDev& B, int i, uint64_t* mo) {
  if (i >= B.r) {
    const int bit = B.n - 1 - i;
    atomicXor((unsigned long long*)&mo[bit >> 6], 1ull << (bit & 63));
  }
}

// x mod N for N = 2^m - 1 and x < 2^(2m).
__device__ __forceinline__ uint32_t mod_n(const BchDev& B, uint32_t x) {
  const uint32_t N = (uint32_t)B.N;
  x = (x & N) + (x >> B.m);
  x = (x & N) + (x >> B.m);
  return x >= N ? x - N : x;
}

// Scans position steps from s on for roots of a locator of degree D (logarithms
// of its coefficients, lane j holds coefficient j; with ZEROS some may be zero),
// up to the first segment of kChienSeg steps that holds one or the end.  Returns
// this lane's root steps in that segment (s then is the step behind it).  sexp[x] =
// alpha^(x - kChienOff); term j keeps Ep = (its exponent mod N) + kChienOff,
// which stays in [0, N + kChienOff) over a segment of steps of -32 j each, so
// the steps inside a segment are constant offsets of the load and the
// reduction mod N happens once per segment.
template <int D, bool ZEROS>
__device__ __forceinline__ uint32_t chien_scan(const BchDev& B, const uint16_t* __restrict__ sexp, uint32_t myL,
                                               int lane, int& s) {
  const uint32_t N = (uint32_t)B.N;
  const int steps = (B.n + 31) >> 5;
  uint32_t Ep[D], keep[ZEROS ? D : 1];  // keep: which terms are there
#pragma unroll
  for (int j = 1; j <= D; j++) {
    uint32_t Lj = __shfl_sync(0xffffffffu, myL, j);
    if (ZEROS) {
      keep[ZEROS ? j - 1 : 0] = Lj == kLogZero ? 0u : 0xffffu;
      Lj = Lj == kLogZero ? 0u : Lj;
    }
    const uint32_t back = mod_n(B, (uint32_t)j * (uint32_t)(32 * s + lane));
    Ep[j - 1] = (Lj >= back ? Lj - back : Lj + N - back) + kChienOff;
  }
  while (s < steps) {
    uint32_t hit = 0;
#pragma unroll 1
    for (int g0 = 0; g0 < kChienSeg; g0 += kChienUnroll) {
#pragma unroll
      for (int g = 0; g < kChienUnroll; g++) {
        uint32_t acc = 0;
#pragma unroll
        for (int j = 1; j <= D; j++) {
          const uint32_t v = sexp[Ep[j - 1] - 32u * j * g];
          acc ^= ZEROS ? v & keep[ZEROS ? j - 1 : 0] : v;
        }
        const int i = 32 * (s + g0 + g) + lane;
        hit |= (uint32_t)(acc == 1u && i < B.n) << (g0 + g);
      }
#pragma unroll
      for (int j = 1; j <= D; j++) Ep[j - 1] -= 32u * j * kChienUnroll;
    }
    s += kChienSeg;
    if (__any_sync(0xffffffffu, hit)) return hit;
#pragma unroll
    for (int j = 1; j <= D; j++) Ep[j - 1] = Ep[j - 1] < (uint32_t)kChienOff ? Ep[j - 1] + N : Ep[j - 1];
  }
  return 0;
}

// Coefficients (logarithms) of the locator divided by 1 - X x, X = alpha^i, i a
// root position: q_j = sum_(m <= j) lambda_m X^(j - m), a prefix XOR over the
// lanes of lambda_m X^-m.
__device__ __forceinline__ uint32_t chien_deflate(const BchDev& B, const uint16_t* __restrict__ sexp, uint32_t myL,
                                                  int lane, int i) {
  const uint32_t N = (uint32_t)B.N, ji = mod_n(B, (uint32_t)lane * (uint32_t)i);
  uint32_t v = myL == kLogZero ? 0u : sexp[(myL >= ji ? myL - ji : myL + N - ji) + kChienOff];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v ^= y;
  }
  if (!v) return kLogZero;
  const uint32_t e = __ldg(&B.log[v]) + ji;
  return e >= N ? e - N : e;
}

// The roots of a locator of degree 1 or 2 (logarithms L1, L2 of its
// coefficients) at positions from `from` on; flips them and returns their number.
// X^2 + q1 X + q2 = 0 with X = q1 z is z^2 + z = q2 / q1^2, solved by a table.
__device__ __forceinline__ int chien_close(const BchDev& B, const uint16_t* __restrict__ sexp, int deg, uint32_t L1,
                                           uint32_t L2, int from, int lane, uint64_t* mo) {
  const uint32_t N = (uint32_t)B.N;
  uint32_t at[2] = {N, N};
  if (deg == 1) {
    at[0] = L1;
  } else if (L1 == kLogZero) {  // X^2 = q2: one (double) root
    at[0] = (L2 & 1u ? L2 + N : L2) >> 1;
  } else {
    const uint32_t two = mod_n(B, 2u * L1);
    const uint32_t z = __ldg(&B.half[sexp[(L2 >= two ? L2 - two : L2 + N - two) + kChienOff]]);
    if (z) {
      at[0] = mod_n(B, L1 + __ldg(&B.log[z]));
      at[1] = mod_n(B, L1 + __ldg(&B.log[z ^ 1u]));
    }
  }
  int roots = 0;
#pragma unroll
  for (int r = 0; r < 2; r++)
    if (at[r] < N && (int)at[r] >= from && (int)at[r] < B.n) {
      roots++;
      if (lane == 0) flip_root(B, (int)at[r], mo);
    }
  return roots;
}

// Any degree (up to 31) and zero coefficients, positions from step s0 on.
__device__ __forceinline__ int chien_generic(const BchDev& B, const uint16_t* __restrict__ sexp, uint32_t myL, int deg,
                                          int s0, int lane, uint64_t* mo) {
  const uint32_t N = (uint32_t)B.N;
  uint32_t E[31], M[31];
  for (int j = 1; j <= deg; j++) {
    const uint32_t Lj = __shfl_sync(0xffffffffu, myL, j);
    M[j - 1] = Lj == kLogZero ? 0u : 0xffffu;
    E[j - 1] = Lj == kLogZero ? 0u : (Lj + N - (uint32_t)(j * (32 * s0 + lane)) % N) % N;
  }
  int roots = 0;
  const int steps = (B.n + 31) >> 5;
  for (int s = s0; s < steps; s++) {
    uint32_t acc = 0;
    for (int j = 1; j <= deg; j++) {
      acc ^= sexp[E[j - 1] + kChienOff] & M[j - 1];
      const uint32_t e = E[j - 1] - 32u * j;
      E[j - 1] = min(e, e + N);
    }
    const int i = 32 * s + lane;
    if (acc == 1u && i < B.n) {
      roots++;
      flip_root(B, i, mo);
    }
    if ((s & 7) == 7 && (int)__reduce_add_sync(0xffffffffu, (unsigned)roots) == deg) break;
  }
  return (int)__reduce_add_sync(0xffffffffu, (unsigned)roots);
}

// Kernel 2 of the decoder: Chien search of the frames with a nonzero locator.
// Each root divided out and degrees 1 and 2 in closed form: 65536 normal 3/5
// frames with 0..12 errors 2.6 -> 1.3 ms.  Two steps unrolled: the warps of an
// SM are at different degrees, and with all eight (and a flip in each) the
// kernel waited for instructions (14 stalls per issue, 2.1 ms).
// Work is taken from the per-degree lists in the order generic, 12, 11, ..., 1,
// so the warps of an SM mostly run the same unrolled evaluator (one
// instruction stream) and the longest frames start first.
__global__ void __launch_bounds__(kChienThreads, 1) bch_chien_kernel(const BchDev B, long long frames,
                                                                     const uint16_t* __restrict__ loc,
                                                                     const int32_t* __restrict__ degs,
                                                                     const uint32_t* __restrict__ bcnt,
                                                                     const int32_t* __restrict__ blist,
                                                                     uint64_t* __restrict__ msg,
                                                                     int32_t* __restrict__ nflips,
                                                                     unsigned long long* __restrict__ next) {
  extern __shared__ __align__(16) uint16_t sexp[];  // [N + kChienOff]: alpha^(x - kChienOff)
  __shared__ long long s_pre[kChienFastMax + 2];     // work offsets of the buckets in fetch order
  for (int i = threadIdx.x; i < B.N + kChienOff; i += blockDim.x) sexp[i] = B.exp[i + B.N - kChienOff];
  if (threadIdx.x == 0) {
    s_pre[0] = 0;
    for (int k = 0; k <= kChienFastMax; k++) s_pre[k + 1] = s_pre[k] + bcnt[k == 0 ? 0 : kChienFastMax + 1 - k];
  }
  __syncthreads();
  const long long total = s_pre[kChienFastMax + 1];
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(next, 1ull);
    w = __shfl_sync(0xffffffffu, w, 0);
    if ((long long)w >= total) break;
    int k = 0;
    while ((long long)w >= s_pre[k + 1]) k++;
    const int bk = k == 0 ? 0 : kChienFastMax + 1 - k;
    const long long f = blist[(size_t)bk * frames + (size_t)((long long)w - s_pre[k])];
    const uint32_t myL = loc[f * 32 + lane];
    uint64_t* mo = msg + f * B.words_k;
    int roots = 0, st = 0, deg = bk == 0 ? degs[f] : bk;
    uint32_t L = lane <= deg ? myL : (uint32_t)kLogZero;
    const int steps = (B.n + 31) >> 5;
    while (bk != 0 && deg > 2 && st < steps) {
      // A locator whose root is divided out may get a zero coefficient (about one
      // frame in 1000).  It is scanned with its terms masked; the general evaluator
      // takes several times as long, and a batch of one wave waits for such a frame
      // (4700 normal 1/2 frames of 15 errors: 688 us with it, 537 us).
      const bool zeros = __any_sync(0xffffffffu, lane >= 1 && lane <= deg && L == kLogZero);
      uint32_t hit = 0;
      switch (deg + (zeros ? 16 : 0)) {
#define GF2C_SCAN(D)                                                    \
  case D: hit = chien_scan<D, false>(B, sexp, L, lane, st); break;      \
  case D + 16: hit = chien_scan<D, true>(B, sexp, L, lane, st); break
        GF2C_SCAN(3);
        GF2C_SCAN(4);
        GF2C_SCAN(5);
        GF2C_SCAN(6);
        GF2C_SCAN(7);
        GF2C_SCAN(8);
        GF2C_SCAN(9);
        GF2C_SCAN(10);
        GF2C_SCAN(11);
#undef GF2C_SCAN
        case 12: hit = chien_scan<12, false>(B, sexp, L, lane, st); break;
      }
      // divide the roots of this segment out
      for (uint32_t who = __ballot_sync(0xffffffffu, hit != 0u); who; who &= who - 1) {
        const int l = __ffs(who) - 1;
        for (uint32_t h = __shfl_sync(0xffffffffu, hit, l); h; h &= h - 1) {
          const int i = 32 * (st - kChienSeg + __ffs(h) - 1) + l;
          if (lane == 0) flip_root(B, i, mo);
          L = chien_deflate(B, sexp, L, lane, i);
          roots++;
          deg--;
        }
      }
    }
    if (deg >= 1 && st < steps) {
      if (bk != 0)
        roots += chien_close(B, sexp, deg, __shfl_sync(0xffffffffu, L, 1), __shfl_sync(0xffffffffu, L, 2), 32 * st, lane,
                             mo);
      else
        roots += chien_generic(B, sexp, L, deg, st, lane, mo);
    }
    if (lane == 0 && nflips) nflips[f] = roots;
  }
}

}  // namespace gf2c

using namespace gf2c;

struct gf2c_bch {
  int frame = 0, rate = 0, dev = -1, sms = 148;
  int occ_syn = 1, occ_enc = 1, occ_chien = 1;
  BchDev d{};
  std::vector<uint16_t> h_exp, h_log, h_mul, h_half, h_lane_mul, h_lane_out;
  bool sliced = false;  // the bit-sliced tables fit the generator factors
  int occ_slice = 0, occ_loc = 1;
  std::vector<uint64_t> h_quad;
  std::vector<uint32_t> h_lf, h_acol;
  std::vector<uint8_t> g;
  std::vector<void*> allocs;
  static constexpr int kStages = 8;
  void* stage[kStages] = {};
  size_t stage_bytes[kStages] = {};
  ~gf2c_bch() {
    for (void* p : allocs) cudaFree(p);
    for (void* p : stage)
      if (p) cudaFree(p);
  }
  int ensure_stage(int i, size_t bytes) {
    if (bytes <= stage_bytes[i]) return GF2C_OK;
    if (stage[i]) cudaFree(stage[i]);
    stage[i] = nullptr;
    stage_bytes[i] = 0;
    GF2C_CUDA(cudaMalloc(&stage[i], std::max(bytes, (size_t)256)));
    stage_bytes[i] = std::max(bytes, (size_t)256);
    return GF2C_OK;
  }
};

namespace {

// The code's tables in one device allocation, 256-byte aligned parts.
struct BchUpload {
  struct Part {
    const void* src;
    size_t bytes;
    const void** out;
  };
  std::vector<Part> parts;
  template <class T, class U>
  void add(const std::vector<T>& v, const U** out) {
    parts.push_back(Part{v.data(), sizeof(T) * v.size(), (const void**)out});
  }
  int run(gf2c_bch* b) {
    auto padded = [](size_t x) { return (x + 255) / 256 * 256; };
    size_t total = 256;
    for (const Part& p : parts) total += padded(p.bytes);
    char* base = nullptr;
    GF2C_CUDA(cudaMalloc((void**)&base, total));
    b->allocs.push_back(base);
    for (const Part& p : parts) {
      GF2C_CUDA(cudaMemcpy(base, p.src, p.bytes, cudaMemcpyHostToDevice));
      *p.out = base;
      base += padded(p.bytes);
    }
    return GF2C_OK;
  }
};

template <int T>
size_t enc_smem() { return syn_smem_bytes<T>() + kBchWarps * 8 * 4 + kBchWarps * 16 * 2; }
template <int T>
size_t syn_smem() { return syn_smem_bytes<T>() + kBchWarps * 32 * 2; }

template <int T>
int set_kernel_attrs(gf2c_bch* b) {
  GF2C_CUDA(allow_smem((const void*)bch_encode_kernel<T>, enc_smem<T>()));
  GF2C_CUDA(allow_smem((const void*)bch_syndrome_bm_kernel<T>, syn_smem<T>()));
  GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->occ_enc, bch_encode_kernel<T>, kBchWarps * 32,
                                                          enc_smem<T>()));
  GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->occ_syn, bch_syndrome_bm_kernel<T>, kBchWarps * 32,
                                                          syn_smem<T>()));
  return GF2C_OK;
}

// Short codes have t = 12; normal ones 12 or 10.
const void* slice_kernel(int t, int m) {
  if (m == 14) return t == 12 ? (const void*)bch_sliced_kernel<12, 14> : nullptr;
  return t == 12 ? (const void*)bch_sliced_kernel<12, 16> : (const void*)bch_sliced_kernel<10, 16>;
}

int bch_upload(gf2c_bch* b) {
  int dev = 0;
  GF2C_CUDA(cudaGetDevice(&dev));
  if (b->dev == dev) return GF2C_OK;
  if (b->dev >= 0) return set_error(GF2C_ERR_UNSUPPORTED, "BCH code already bound to another device");
  BchUpload up;
  up.add(b->h_exp, &b->d.exp);
  up.add(b->h_log, &b->d.log);
  up.add(b->h_half, &b->d.half);
  up.add(b->h_lane_mul, &b->d.lane_mul);
  up.add(b->h_lane_out, &b->d.lane_out);
  up.add(b->h_quad, &b->d.quad);
  up.add(b->h_mul, &b->d.mul);
  up.add(b->h_lf, &b->d.lf);
  up.add(b->h_acol, &b->d.acol);
  int rc = up.run(b);
  if (rc) return rc;
  GF2C_CUDA(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev));
  if ((rc = b->d.t == 12 ? set_kernel_attrs<12>(b) : set_kernel_attrs<10>(b))) return rc;
  if (b->sliced) {
    const void* k = slice_kernel(b->d.t, b->d.m);
    const int sm = (int)(b->d.t == 12 ? slice_smem_bytes<12>() : slice_smem_bytes<10>());
    if (k) {
      GF2C_CUDA(allow_smem(k, sm));
      GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->occ_slice, k, kSliceThreads, sm));
      GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &b->occ_loc, b->d.t == 12 ? (const void*)bch_locator_kernel<12> : (const void*)bch_locator_kernel<10>,
          kBchWarps * 32, 0));
      b->occ_loc = std::max(b->occ_loc, 1);
    }
  }
  const int chien_smem = (b->d.N + kChienOff) * 2;
  GF2C_CUDA(allow_smem((const void*)bch_chien_kernel, chien_smem));
  GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b->occ_chien, bch_chien_kernel, kChienThreads, chien_smem));
  b->occ_enc = std::max(b->occ_enc, 1);
  b->occ_syn = std::max(b->occ_syn, 1);
  b->occ_chien = std::max(b->occ_chien, 1);
  b->dev = dev;
  return GF2C_OK;
}

int warp_grid(long long frames, int sms, int occ) {
  const long long want = (frames + kBchWarps - 1) / kBchWarps;
  return (int)std::max<long long>(1, std::min<long long>(want, (long long)sms * occ));
}

// Inverse over GF(2) of the r x r matrix given as rows of bits; false if singular.
bool gf2_invert(int r, std::vector<std::vector<uint64_t>>& rows, std::vector<std::vector<uint64_t>>& inv) {
  const int W = (r + 63) / 64;
  inv.assign(r, std::vector<uint64_t>(W, 0));
  for (int i = 0; i < r; i++) inv[i][i >> 6] |= 1ull << (i & 63);
  for (int c = 0; c < r; c++) {
    int piv = -1;
    for (int i = c; i < r; i++)
      if ((rows[i][c >> 6] >> (c & 63)) & 1) {
        piv = i;
        break;
      }
    if (piv < 0) return false;
    std::swap(rows[c], rows[piv]);
    std::swap(inv[c], inv[piv]);
    for (int i = 0; i < r; i++)
      if (i != c && ((rows[i][c >> 6] >> (c & 63)) & 1))
        for (int w = 0; w < W; w++) {
          rows[i][w] ^= rows[c][w];
          inv[i][w] ^= inv[c][w];
        }
  }
  return true;
}

}  // namespace

extern "C" {

int gf2c_bch_create_dvbt2(int32_t frame_size, int32_t rate, gf2c_bch** out) {
  if (!out) return set_error(GF2C_ERR_INVALID_ARG, "out is NULL");
  *out = nullptr;
  if (frame_size < 0 || frame_size > 1 || rate < 0 || rate > 5)
    return set_error(GF2C_ERR_INVALID_ARG, "DVB-T2 frame size must be 0/1 and rate 0..5");
  static const int kShortN[6] = {7200, 9720, 10800, 11880, 12600, 13320};
  static const int kShortK[6] = {7032, 9552, 10632, 11712, 12432, 13152};
  static const int kNormalN[6] = {32400, 38880, 43200, 48600, 51840, 54000};
  static const int kNormalK[6] = {32208, 38688, 43040, 48408, 51648, 53840};
  static const int kNormalT[6] = {12, 12, 10, 12, 12, 10};
  std::unique_ptr<gf2c_bch> b(new (std::nothrow) gf2c_bch());
  if (!b) return set_error(GF2C_ERR_NOMEM, "out of host memory");
  const bool shortf = frame_size == 1;
  BchDev& d = b->d;
  b->frame = frame_size;
  b->rate = rate;
  d.n = shortf ? kShortN[rate] : kNormalN[rate];
  d.k = shortf ? kShortK[rate] : kNormalK[rate];
  d.t = shortf ? 12 : kNormalT[rate];
  d.r = d.n - d.k;
  d.m = shortf ? 14 : 16;
  const uint32_t prim = shortf ? 0b100000000101011u : 0b10000000000101101u;
  const int q = 1 << d.m;
  d.N = q - 1;
  d.words_n = (d.n + 63) / 64;
  d.words_k = (d.k + 63) / 64;
  d.rw = (d.r + 31) / 32;
  // antilog / log tables of GF(2^m), alpha = x
  b->h_exp.assign(2 * d.N, 0);
  b->h_log.assign(q, 0);
  uint32_t x = 1;
  for (int e = 0; e < d.N; e++) {
    b->h_exp[e] = (uint16_t)x;
    b->h_log[x] = (uint16_t)e;
    x <<= 1;
    if (x & (uint32_t)q) x ^= prim;
  }
  for (int e = d.N; e < 2 * d.N; e++) b->h_exp[e] = b->h_exp[e - d.N];
  auto apow = [&](long long e) -> uint32_t { return b->h_exp[((e % d.N) + d.N) % d.N]; };
  auto mul = [&](uint32_t a, uint32_t c) -> uint32_t {
    return (a && c) ? b->h_exp[b->h_log[a] + b->h_log[c]] : 0u;
  };
  // z^2 + z is linear over GF(2): one bit of z at a time (Gray code)
  b->h_half.assign(q, 0);
  uint16_t image[16];
  for (int e = 0; e < d.m; e++) image[e] = (uint16_t)(mul(1u << e, 1u << e) ^ (1u << e));
  for (uint32_t i = 1, z = 0, c = 0; i < (uint32_t)q; i++) {
    const int e = __builtin_ctz(i);
    z ^= 1u << e;
    c ^= image[e];
    b->h_half[c] = (uint16_t)(z | 1u);
  }
  b->h_half[0] = 0;  // z = 0 and 1
  // generator g = g_1 ... g_t (binary)
  std::vector<uint8_t> g{1};
  for (int i = 0; i < d.t; i++) {
    std::vector<uint8_t> fct(d.m + 1, 0);
    for (int j = 0;; j++) {
      const int e = shortf ? kShortGen[i][j] : kNormalGen[i][j];
      if (e < 0) break;
      fct[e] = 1;
    }
    std::vector<uint8_t> p(g.size() + fct.size() - 1, 0);
    for (size_t a = 0; a < g.size(); a++)
      if (g[a])
        for (size_t c = 0; c < fct.size(); c++) p[a + c] ^= fct[c];
    g = p;
  }
  if ((int)g.size() - 1 != d.r || d.r != d.t * d.m)
    return set_error(GF2C_ERR_KERNEL, "internal: BCH generator degree mismatch");
  b->g = g;
  // syndrome tables, odd j = 2s+1, beta = alpha^-j
  b->h_quad.assign((size_t)3 * 8 * 256, 0);
  b->h_mul.assign((size_t)d.t * 512, 0);
  b->h_lf.assign((size_t)d.t * 32, 0);
  for (int s = 0; s < d.t; s++) {
    const long long j = 2 * s + 1;
    for (int p = 0; p < 8; p++) {
      uint32_t unit[8];
      for (int e = 0; e < 8; e++) unit[e] = apow(-j * (8 * p + e));
      uint64_t sum[256] = {0};  // each from the one without its lowest bit
      for (int v = 1; v < 256; v++) {
        sum[v] = sum[v & (v - 1)] ^ unit[__builtin_ctz(v)];
        b->h_quad[((size_t)(s / 4) * 8 + p) * 256 + v] |= sum[v] << (16 * (s % 4));
      }
    }
    const uint32_t gamma = apow(-j * 2048);
    for (int v = 0; v < 256; v++) {
      b->h_mul[(size_t)s * 512 + v] = (uint16_t)mul((uint32_t)v, gamma);
      const uint32_t hv = (uint32_t)v << 8;
      b->h_mul[(size_t)s * 512 + 256 + v] = hv < (uint32_t)q ? (uint16_t)mul(hv, gamma) : 0;
    }
    for (int lane = 0; lane < 32; lane++)
      b->h_lf[(size_t)s * 32 + lane] = (uint32_t)((j * (d.n - 1 - 64 * lane)) % d.N);
  }
  // bit-sliced syndromes: states are vectors in the basis 1, eta, .., eta^(m-1),
  // eta = alpha^(32 j); the generator factors must vanish at alpha^j
  b->sliced = true;
  b->h_lane_mul.assign((size_t)d.t * 512, 0);
  b->h_lane_out.assign((size_t)d.t * 512, 0);
  for (int s = 0; s < d.t; s++) {
    const long long j = 2 * s + 1;
    uint32_t at = 0;
    for (int i = 0; (shortf ? kShortGen[s][i] : kNormalGen[s][i]) >= 0; i++)
      at ^= apow(j * (shortf ? kShortGen[s][i] : kNormalGen[s][i]));
    // rows: field element of each basis vector; inverse by elimination
    uint32_t basis[16], inv[16];
    for (int i = 0; i < d.m; i++) {
      basis[i] = apow(32 * j * i);
      inv[i] = 1u << i;
    }
    bool ok = at == 0;
    for (int c = 0; c < d.m && ok; c++) {
      int piv = -1;
      for (int i = c; i < d.m && piv < 0; i++)
        if (basis[i] >> c & 1u) piv = i;
      if (piv < 0) {
        ok = false;
        break;
      }
      std::swap(basis[c], basis[piv]);
      std::swap(inv[c], inv[piv]);
      for (int i = 0; i < d.m; i++)
        if (i != c && (basis[i] >> c & 1u)) {
          basis[i] ^= basis[c];
          inv[i] ^= inv[c];
        }
    }
    b->sliced = b->sliced && ok;
    if (!ok) continue;
    auto vec_of = [&](uint32_t x) {  // field element -> vector
      uint32_t v = 0;
      for (int c = 0; c < d.m; c++)
        if (x >> c & 1u) v ^= inv[c];
      return v;
    };
    const uint32_t back = apow(-j), fin = apow(j * (d.n - 1 - 32ll * (slice_steps(d.n) - 1)));
    for (int half = 0; half < 2; half++)
      for (int e = 0; e < 8 && 8 * half + e < d.m; e++) {  // linear: powers of two, then sums
        const uint32_t x = apow(32 * j * (8 * half + e));
        uint16_t* lm = &b->h_lane_mul[(size_t)s * 512 + 256 * half];
        uint16_t* lo = &b->h_lane_out[(size_t)s * 512 + 256 * half];
        const uint16_t xm = (uint16_t)vec_of(mul(x, back)), xo = (uint16_t)mul(x, fin);
        for (int v = 0; v < 1 << e; v++) {
          lm[(1 << e) + v] = lm[v] ^ xm;
          lo[(1 << e) + v] = lo[v] ^ xo;
        }
      }
  }
  // parity from odd syndromes: P[b][q] = bit (b % m) of S_(2(b/m)+1) of parity bit q
  // (codeword bit k+q, degree r-1-q); A = P^-1, stored by column b
  {
    const int W = (d.r + 63) / 64;
    std::vector<std::vector<uint64_t>> P(d.r, std::vector<uint64_t>(W, 0)), A;
    for (int qb = 0; qb < d.r; qb++)
      for (int s = 0; s < d.t; s++) {
        const uint32_t v = apow((long long)(2 * s + 1) * (d.r - 1 - qb));
        for (int bp = 0; bp < d.m; bp++)
          if ((v >> bp) & 1) P[s * d.m + bp][qb >> 6] |= 1ull << (qb & 63);
      }
    if (!gf2_invert(d.r, P, A)) return set_error(GF2C_ERR_KERNEL, "internal: BCH parity map is singular");
    b->h_acol.assign((size_t)d.r * d.rw, 0);
    for (int qb = 0; qb < d.r; qb++)
      for (int bb = 0; bb < d.r; bb++)
        if ((A[qb][bb >> 6] >> (bb & 63)) & 1) b->h_acol[(size_t)bb * d.rw + (qb >> 5)] |= 1u << (qb & 31);
  }
  *out = b.release();
  return GF2C_OK;
}

int gf2c_bch_destroy(gf2c_bch* bch) {
  delete bch;
  return GF2C_OK;
}

int gf2c_bch_dims(const gf2c_bch* bch, int64_t* n, int64_t* k, int32_t* t, int32_t* field_m) {
  if (!bch) return set_error(GF2C_ERR_INVALID_ARG, "bch is NULL");
  if (n) *n = bch->d.n;
  if (k) *k = bch->d.k;
  if (t) *t = bch->d.t;
  if (field_m) *field_m = bch->d.m;
  return GF2C_OK;
}

int gf2c_bch_generator(const gf2c_bch* bch, uint8_t* coeffs) {
  if (!bch || !coeffs) return set_error(GF2C_ERR_INVALID_ARG, "NULL argument");
  std::memcpy(coeffs, bch->g.data(), bch->g.size());
  return GF2C_OK;
}

int gf2c_bch_encode_batch(gf2c_bch* bch, const uint64_t* msg_bits, int64_t frames, uint64_t* cw_bits,
                          int32_t mem, void* stream) {
  if (!bch || frames < 0 || (frames > 0 && (!msg_bits || !cw_bits)) || (mem != GF2C_MEM_HOST && mem != GF2C_MEM_DEVICE))
    return set_error(GF2C_ERR_INVALID_ARG, "bad arguments");
  if (frames == 0) return GF2C_OK;
  int rc = bch_upload(bch);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const BchDev& d = bch->d;
  const size_t bin = (size_t)frames * d.words_k * 8, bout = (size_t)frames * d.words_n * 8;
  const uint64_t* in = msg_bits;
  uint64_t* out = cw_bits;
  if (mem == GF2C_MEM_HOST) {
    if ((rc = bch->ensure_stage(0, bin)) || (rc = bch->ensure_stage(1, bout))) return rc;
    GF2C_CUDA(cudaMemcpyAsync(bch->stage[0], msg_bits, bin, cudaMemcpyHostToDevice, st));
    in = (const uint64_t*)bch->stage[0];
    out = (uint64_t*)bch->stage[1];
  }
  const int grid = warp_grid(frames, bch->sms, bch->occ_enc);
  if (d.t == 12) bch_encode_kernel<12><<<grid, kBchWarps * 32, enc_smem<12>(), st>>>(d, in, frames, out);
  else bch_encode_kernel<10><<<grid, kBchWarps * 32, enc_smem<10>(), st>>>(d, in, frames, out);
  GF2C_CUDA(cudaGetLastError());
  if (mem == GF2C_MEM_HOST) {
    GF2C_CUDA(cudaMemcpyAsync(cw_bits, out, bout, cudaMemcpyDeviceToHost, st));
    GF2C_CUDA(cudaStreamSynchronize(st));
  }
  return GF2C_OK;
}

int gf2c_bch_decode_batch(gf2c_bch* bch, const uint64_t* cw_bits, int64_t frames, uint64_t* msg_bits,
                          int32_t* corrected, uint16_t* syndromes, int32_t mem, void* stream) {
  if (!bch || frames < 0 || (frames > 0 && (!cw_bits || !msg_bits)) || (mem != GF2C_MEM_HOST && mem != GF2C_MEM_DEVICE))
    return set_error(GF2C_ERR_INVALID_ARG, "bad arguments");
  if (frames == 0) return GF2C_OK;
  int rc = bch_upload(bch);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const BchDev& d = bch->d;
  const size_t bin = (size_t)frames * d.words_n * 8, bout = (size_t)frames * d.words_k * 8;
  const size_t bc = (size_t)frames * 4, bs = (size_t)frames * 2 * d.t * 2;
  if ((rc = bch->ensure_stage(4, (size_t)frames * 32 * 2)) || (rc = bch->ensure_stage(5, (size_t)frames * 4)) ||
      (rc = bch->ensure_stage(6, 128)) || (rc = bch->ensure_stage(7, (size_t)(kChienFastMax + 1) * frames * 4)))
    return rc;
  const uint64_t* in = cw_bits;
  uint64_t* out = msg_bits;
  int32_t* cor = corrected;
  uint16_t* syn = syndromes;
  if (mem == GF2C_MEM_HOST) {
    if ((rc = bch->ensure_stage(0, bin)) || (rc = bch->ensure_stage(1, bout)) ||
        (corrected && (rc = bch->ensure_stage(2, bc))) || (syndromes && (rc = bch->ensure_stage(3, bs))))
      return rc;
    GF2C_CUDA(cudaMemcpyAsync(bch->stage[0], cw_bits, bin, cudaMemcpyHostToDevice, st));
    in = (const uint64_t*)bch->stage[0];
    out = (uint64_t*)bch->stage[1];
    cor = corrected ? (int32_t*)bch->stage[2] : nullptr;
    syn = syndromes ? (uint16_t*)bch->stage[3] : nullptr;
  }
  uint16_t* loc = (uint16_t*)bch->stage[4];
  int32_t* degs = (int32_t*)bch->stage[5];
  unsigned long long* next = (unsigned long long*)bch->stage[6];  // work counter, then bucket sizes
  uint32_t* bcnt = (uint32_t*)((char*)bch->stage[6] + 64);
  int32_t* blist = (int32_t*)bch->stage[7];
  GF2C_CUDA(cudaMemsetAsync(bch->stage[6], 0, 128, st));
  const int grid = warp_grid(frames, bch->sms, bch->occ_syn);
  // The bit-sliced kernel from 32 frames (one CTA) per SM on: below that SMs stay
  // idle and a CTA's own time shows (normal 3/5, 2368 frames: 481 us the whole
  // decode against 450 with the table kernel; 4736 frames: 494 against 520).
  if (bch->occ_slice > 0 && frames >= 32ll * bch->sms) {
    const size_t sm = d.t == 12 ? slice_smem_bytes<12>() : slice_smem_bytes<10>();
    const int sg = (int)std::min<long long>((frames + 31) / 32, (long long)bch->sms * bch->occ_slice);
    void* args[] = {(void*)&d, &in, &frames, &out, &loc};
    GF2C_CUDA(cudaLaunchKernel(slice_kernel(d.t, d.m), dim3(sg), dim3(kSliceThreads), args, sm, st));
    const int lg = warp_grid(frames, bch->sms, bch->occ_loc);
    if (d.t == 12)
      bch_locator_kernel<12><<<lg, kBchWarps * 32, 0, st>>>(d, frames, cor, syn, loc, degs, bcnt, blist);
    else
      bch_locator_kernel<10><<<lg, kBchWarps * 32, 0, st>>>(d, frames, cor, syn, loc, degs, bcnt, blist);
  } else if (d.t == 12)
    bch_syndrome_bm_kernel<12><<<grid, kBchWarps * 32, syn_smem<12>(), st>>>(d, in, frames, out, cor, syn, loc, degs, bcnt, blist);
  else
    bch_syndrome_bm_kernel<10><<<grid, kBchWarps * 32, syn_smem<10>(), st>>>(d, in, frames, out, cor, syn, loc, degs, bcnt, blist);
  GF2C_CUDA(cudaGetLastError());
  bch_chien_kernel<<<bch->sms * bch->occ_chien, kChienThreads, (size_t)(d.N + kChienOff) * 2, st>>>(
      d, frames, loc, degs, bcnt, blist, out, cor, next);
  GF2C_CUDA(cudaGetLastError());
  if (mem == GF2C_MEM_HOST) {
    GF2C_CUDA(cudaMemcpyAsync(msg_bits, out, bout, cudaMemcpyDeviceToHost, st));
    if (corrected) GF2C_CUDA(cudaMemcpyAsync(corrected, cor, bc, cudaMemcpyDeviceToHost, st));
    if (syndromes) GF2C_CUDA(cudaMemcpyAsync(syndromes, syn, bs, cudaMemcpyDeviceToHost, st));
    GF2C_CUDA(cudaStreamSynchronize(st));
  }
  return GF2C_OK;
}

}  // extern "C"
