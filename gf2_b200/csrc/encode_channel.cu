// gf2cuda encoder, syndrome and AWGN channel kernels (sm_100a).
//
// Encoder: the reference encodes with a dense k x m generator block
// (RuEncodingMatrices::encode, crates/gf2-coding/src/ldpc/encoding/richardson_urbanke.rs:263-289,
// 97.5% of its encode time in BitMatrix::matvec_transpose).  For DVB-T2 codes the
// parity part of H is the staircase, so the same unique codeword is
//   s = H_info u,  p[i] = s[0] ^ ... ^ s[i].
// With the checks of row group a = p mod q at positions t = p div q, s of a
// row group is a XOR of the 360-bit info blocks rotated by their addresses
// (32-bit windows), and p is a prefix over row groups plus a prefix along t;
// a warp-shuffle bit transpose puts the parity into natural order.  Other codes use the dense generator
// block of the right-to-left pivot search (the reference's columns).
//
// Syndrome: LdpcCode::syndrome (crates/gf2-coding/src/ldpc/core.rs:129-133).
// Channel: BpskModulator / AwgnChannel (crates/gf2-coding/src/channel.rs:51-218) with
// Philox4x32-10 and Box-Muller in place of rand_distr::Normal.
#include "bits.cuh"
#include "internal.h"
#include "numeric.cuh"

namespace gf2c {

static constexpr int kEncThreads = 1024;     // channel kernel (Philox + LLRs for one frame)
static constexpr int kEncodeThreads = 384;   // encode kernel (several frames per SM): a warp per 32 positions t

// Bit i of a u32-word bit array.
__device__ __forceinline__ uint32_t getbit(const uint32_t* w, int i) { return (w[i >> 5] >> (i & 31)) & 1u; }

// DVB-T2 structure (row group a holds the checks p = a + q t, t < 360): the
// info syndrome of row group a is
//   S_a[t] = XOR over its addresses x = a + q tau (info block b) of u[360 b + (t - tau) mod 360],
// a XOR of the info blocks rotated by tau.  A cyclic copy of each block makes a
// rotation a run of words at one shift, so a task takes several consecutive
// words of one row group: per address one table entry, then a load, a funnel
// shift and a XOR per word.
constexpr int kRowWords = 13;  // words per row group
constexpr int kBlkWords = 25;  // words per cyclic copy (24 used; odd, so that blocks start in different banks)

// One word of G frames side by side: G frames share a task's table entries and
// addresses, and their words come in one vector load.
template <int G>
struct alignas(4 * G) Words {
  uint32_t v[G];
};

// Shared-memory tables of a code, made once per CTA: entry e of enc_rg_ent as
// (first word of the rotated run in the block copies) | shift << 24.
__device__ __forceinline__ void dvbt2_build_entries(const DevCode& C, uint32_t* ent) {
  const int total = __ldg(&C.enc_rg_ptr[C.enc_q]);
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int x = __ldg(&C.enc_rg_ent[e]), tau = x & 0xffff, b = x >> 16;
    const int s = tau == 0 ? 0 : 360 - tau;
    ent[e] = (uint32_t)(kBlkWords * b + (s >> 5)) | (uint32_t)(s & 31) << 24;
  }
}

// Cyclic copies of the info blocks: bit j of a copy = block bit j mod 360, j < 743.
// u: G messages, `pitch` words apart.
template <int G>
__device__ __forceinline__ void dvbt2_build_blocks(const uint32_t* u, int pitch, int wk, int nblk, Words<G>* U2) {
  for (int idx = threadIdx.x; idx < nblk * G; idx += blockDim.x) {
    const int b = idx / G, f = idx % G;
    const int base = (360 * b) >> 5, sh = (360 * b) & 31;
    const uint32_t* uf = u + f * pitch;
    uint32_t x[12];
#pragma unroll
    for (int i = 0; i < 12; i++) {
      const uint32_t lo = uf[base + i], hi = base + i + 1 < wk ? uf[base + i + 1] : 0u;
      x[i] = __funnelshift_r(lo, hi, sh);
    }
    x[11] = (x[11] & 0xffu) | (x[0] << 8);  // block bits 352..359, then 0..23
    Words<G>* d = U2 + kBlkWords * b;
#pragma unroll
    for (int i = 0; i < 12; i++) d[i].v[f] = x[i];
#pragma unroll
    for (int i = 12; i < 23; i++) d[i].v[f] = __funnelshift_r(x[i - 12], x[i - 11], 24);
    d[23].v[f] = x[11] >> 24;
  }
}

// S[13 a + w] = word w (t = 32 w + bit) of the info syndrome of row group a,
// W words per task (13: a warp reads one word of 32 row groups).  With one or two
// words per task the tasks of a row group are neighbours, so that a warp reads few
// table entries and runs of words (the encoder in the channel kernel, 3000 normal
// 3/5 frames: 86 us, 99 us with a warp across 32 row groups).
template <int W, int G>
__device__ __forceinline__ void dvbt2_row_syndromes(const int* __restrict__ rg_ptr, const uint32_t* ent,
                                                    const Words<G>* U2, int q, Words<G>* S) {
  for (int idx = threadIdx.x; idx < (12 / W) * q; idx += blockDim.x) {
    constexpr int parts = 12 / W;
    const int a = W <= 2 ? idx / parts : idx % q, part = W <= 2 ? idx - a * parts : idx / q;
    Words<G> acc[W];
#pragma unroll
    for (int i = 0; i < W; i++)
#pragma unroll
      for (int f = 0; f < G; f++) acc[i].v[f] = 0u;
    const int e1 = __ldg(&rg_ptr[a + 1]);
    for (int e = __ldg(&rg_ptr[a]); e < e1; e++) {
      const uint32_t x = ent[e];
      const Words<G>* d = U2 + (x & 0xffffffu) + W * part;
      const int sh = (int)(x >> 24);
      Words<G> lo = d[0];
#pragma unroll
      for (int i = 0; i < W; i++) {
        const Words<G> hi = d[i + 1];
#pragma unroll
        for (int f = 0; f < G; f++) acc[i].v[f] ^= __funnelshift_r(lo.v[f], hi.v[f], sh);
        lo = hi;
      }
    }
    if (W * part + W == 12)
#pragma unroll
      for (int f = 0; f < G; f++) acc[W - 1].v[f] &= 0xffu;
#pragma unroll
    for (int i = 0; i < W; i++) S[kRowWords * a + W * part + i] = acc[i];
  }
}
// Words per task: as many tasks as fill the CTA in one round, the rest of a
// task's cost being its table entries (3 W + 4 instructions per address).
template <int G>
__device__ __forceinline__ void dvbt2_syndromes(const DevCode& C, const uint32_t* ent, const Words<G>* U2, Words<G>* S) {
  const int q = C.enc_q, T = blockDim.x;
  if (12 * q <= T) dvbt2_row_syndromes<1, G>(C.enc_rg_ptr, ent, U2, q, S);
  else if (6 * q <= T) dvbt2_row_syndromes<2, G>(C.enc_rg_ptr, ent, U2, q, S);
  else if (4 * q <= T) dvbt2_row_syndromes<3, G>(C.enc_rg_ptr, ent, U2, q, S);
  else if (3 * q <= T) dvbt2_row_syndromes<4, G>(C.enc_rg_ptr, ent, U2, q, S);
  else dvbt2_row_syndromes<6, G>(C.enc_rg_ptr, ent, U2, q, S);
}

// The row-group words of 32 positions t (lane's t = 32 T + lane) as bits over
// row groups: bit r of x[f][A] = check a + q t of frame f, a = 32 A + r (zero for
// a >= q).
template <int G>
__device__ __forceinline__ void dvbt2_columns(const Transpose32& tr, const Words<G>* S, int q, int T,
                                              uint32_t (&x)[G][3]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int A = 0; A < 3; A++) {
    Words<G> w;
#pragma unroll
    for (int f = 0; f < G; f++) w.v[f] = 0u;
    const int a = 32 * A + lane;
    if (a < q) w = S[kRowWords * a + T];
#pragma unroll
    for (int f = 0; f < G; f++) x[f][A] = 32 * A < q ? tr(w.v[f]) : 0u;
  }
}
// OR the q bits x of position t into dst at bit t q (natural check order).
__device__ __forceinline__ void dvbt2_or_bits(const uint32_t (&x)[3], int q, int t, uint32_t* dst) {
  const int p0 = t * q, w0 = p0 >> 5, sh = p0 & 31;
  uint32_t lo = 0;  // what spills over from the word before
#pragma unroll
  for (int A = 0; A < 3; A++) {
    if (32 * A >= q) break;
    const uint32_t v = (x[A] << sh) | lo;
    if (v) atomicOr(&dst[w0 + A], v);
    lo = sh ? x[A] >> (32 - sh) : 0u;
  }
  if (lo) atomicOr(&dst[w0 + (q + 31) / 32], lo);
}

// Info syndromes of the message bits u by row group (scratch: block copies).
template <int G>
__device__ __forceinline__ void dvbt2_row_groups(const DevCode& C, const uint32_t* u, int pitch, const uint32_t* ent,
                                                 Words<G>* U2, Words<G>* S) {
  dvbt2_build_blocks<G>(u, pitch, (C.k + 31) >> 5, C.k / 360, U2);
  __syncthreads();
  dvbt2_syndromes<G>(C, ent, U2, S);
  __syncthreads();
}

// Word w (32 bits) of the codeword [message u | parity P]; P has a zero word
// behind it and zero bits beyond m.
__device__ __forceinline__ uint32_t dvbt2_code_word(const uint32_t* u, const uint32_t* P, int k, int n, int w) {
  const int lo = 32 * w, off = lo - k;
  if (lo >= n) return 0u;
  if (off >= 0) return __funnelshift_r(P[off >> 5], P[(off >> 5) + 1], off & 31);
  if (off <= -32) return u[w];
  return (u[w] & ((1u << (k & 31)) - 1u)) | (P[0] << (k & 31));
}

// Parity of the message bits u (zero bits beyond k) of G frames: P = wm + 1
// words per frame.  Bit p is the XOR of the info syndromes of the checks up to
// p: a prefix over the q row groups of position t in a lane's registers, and
// over t by ballots (12 warps take 32 positions each; tot: 12 words per frame).
template <int G>
__device__ __forceinline__ void dvbt2_parity(const DevCode& C, const uint32_t* u, int pitch, const uint32_t* ent,
                                             Words<G>* U2, Words<G>* S, uint32_t* P, uint32_t* tot) {
  const int q = C.enc_q, wp = ((C.m + 31) >> 5) + 1;
  const int lane = threadIdx.x & 31, T = threadIdx.x >> 5;
  for (int w = threadIdx.x; w < G * wp; w += blockDim.x) P[w] = 0u;
  dvbt2_row_groups<G>(C, u, pitch, ent, U2, S);
  uint32_t x[G][3], bal[G];
  if (T < 12) {
    const Transpose32 tr(lane);
    dvbt2_columns<G>(tr, S, q, T, x);
#pragma unroll
    for (int f = 0; f < G; f++) {
      uint32_t carry = 0;
#pragma unroll
      for (int A = 0; A < 3; A++) {
        if (32 * A >= q) break;
        uint32_t v = x[f][A];
        v ^= v << 1;
        v ^= v << 2;
        v ^= v << 4;
        v ^= v << 8;
        v ^= v << 16;
        x[f][A] = v ^ carry;
        carry = (uint32_t)((int)x[f][A] >> 31);  // the last word's upper bits repeat its last parity
      }
      bal[f] = __ballot_sync(0xffffffffu, carry & 1u);
      if (lane == 0) tot[12 * f + T] = bal[f];
    }
  }
  __syncthreads();
  if (T < 12) {
    const int t = 32 * T + lane;
#pragma unroll
    for (int f = 0; f < G; f++) {
      const uint32_t before = lane < T ? (uint32_t)__popc(tot[12 * f + lane]) & 1u : 0u;
      const uint32_t flip =
          0u - ((__popc(__ballot_sync(0xffffffffu, before)) ^ __popc(bal[f] & ((1u << lane) - 1u))) & 1u);
#pragma unroll
      for (int A = 0; A < 3; A++) {
        const int nb = q - 32 * A;
        if (nb > 0) x[f][A] = (x[f][A] ^ flip) & (nb < 32 ? (1u << nb) - 1u : ~0u);
      }
      if (t < 360) dvbt2_or_bits(x[f], q, t, P + f * wp);
    }
  }
  __syncthreads();
}

// Shared memory of the DVB-T2 path: block copies and row-group words (G frames),
// entries, parity and scan scratch, and before them G messages of 2 words_k words.
static __host__ __device__ inline int dvbt2_scratch_words(int nblk, int q, int m, int entries, int G) {
  return (kBlkWords * nblk + kRowWords * q + (m + 31) / 32 + 1 + 12) * G + entries;
}
template <int G>
struct DvbScratch {
  Words<G>*U2, *S;
  uint32_t *ent, *P, *tot;
};
template <int G>
__device__ __forceinline__ DvbScratch<G> dvbt2_carve(const DevCode& C, uint32_t* scratch) {
  DvbScratch<G> D;
  D.U2 = (Words<G>*)scratch;
  D.S = D.U2 + kBlkWords * (C.k / 360);
  D.ent = (uint32_t*)(D.S + kRowWords * C.enc_q);
  D.P = D.ent + C.enc_rg_total;
  D.tot = D.P + ((C.m + 31) / 32 + 1) * G;
  return D;
}

// Encodes the message bits u (k bits, u32 words in shared memory) into the
// codeword cw (n bits, u32 words in shared memory); scratch as encode_smem sizes
// it, with the DVB-T2 entries in place.
__device__ void encode_frame(const DevCode& C, const uint32_t* u, uint32_t* cw, uint32_t* scratch) {
  const int n = C.n, k = C.k, m = C.m;
  const int wn = (n + 31) >> 5;
  if (C.enc_kind == 0) {
    const DvbScratch<1> D = dvbt2_carve<1>(C, scratch);
    dvbt2_parity<1>(C, u, 0, D.ent, D.U2, D.S, D.P, D.tot);
    for (int w = threadIdx.x; w < wn; w += blockDim.x) cw[w] = dvbt2_code_word(u, D.P, k, n, w);
    __syncthreads();
  } else {
    // parity word j (64 bits) = XOR over message bits i of P[i][j]
    const int Wm = C.words_m;
    uint64_t* par64 = (uint64_t*)scratch;  // Wm words (scratch sized for it)
    for (int j = threadIdx.x; j < Wm; j += blockDim.x) {
      uint64_t acc = 0;
      for (int i = 0; i < k; i++)
        if (getbit(u, i)) acc ^= __ldg(&C.enc_p[(size_t)i * Wm + j]);
      par64[j] = acc;
    }
    for (int w = threadIdx.x; w < wn; w += blockDim.x) cw[w] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < k; i += blockDim.x)
      if (getbit(u, i)) {
        const int c = __ldg(&C.enc_msg_cols[i]);
        atomicOr(&cw[c >> 5], 1u << (c & 31));
      }
    for (int j = threadIdx.x; j < m; j += blockDim.x)
      if ((par64[j >> 6] >> (j & 63)) & 1ull) {
        const int c = __ldg(&C.enc_par_cols[j]);
        atomicOr(&cw[c >> 5], 1u << (c & 31));
      }
    __syncthreads();
  }
}

// shared memory: u (wk32) + cw (wn32) + scratch
static size_t encode_smem(const DevCode& C) {
  const int wn = (C.n + 31) / 32, wm = (C.m + 31) / 32;
  const int scratch = C.enc_kind == 0 ? dvbt2_scratch_words(C.k / 360, C.enc_q, C.m, C.enc_rg_total, 1)
                                      : std::max(wm + 64, 2 * C.words_m);
  return (size_t)(((2 * C.words_k + 3) & ~3) + ((wn + 3) & ~3) + scratch + 4) * 4;
}

// DVB-T2 encoder, G frames per CTA at a time.  See launch_encode for what
// bounds it and the figures.
template <int G>
__global__ void __launch_bounds__(kEncodeThreads, G == 1 ? 3 : 2) encode_dvb_kernel(const DevCode* __restrict__ Cp,
                                                                    const uint64_t* __restrict__ msg,
                                                                    long long frames, uint64_t* __restrict__ cw) {
  extern __shared__ __align__(16) uint32_t sm[];
  const DevCode C = *Cp;
  const int pitch = 2 * C.words_k;  // words per message in shared memory
  uint32_t* u = sm;
  const DvbScratch<G> D = dvbt2_carve<G>(C, sm + ((G * pitch + 3) & ~3));
  dvbt2_build_entries(C, D.ent);
  const int whole = C.k >> 6, wp = ((C.m + 31) >> 5) + 1;
  for (long long f0 = (long long)blockIdx.x * G; f0 < frames; f0 += (long long)gridDim.x * G) {
    // the messages, into shared memory and straight into the codewords' whole
    // message words; frames beyond the batch are zero
    const int wk = C.words_k, real = (int)min((long long)G, frames - f0) * wk;  // words of the batch's frames
    const uint2* mi = (const uint2*)(msg + f0 * wk);
    for (int base = threadIdx.x; base < G * wk; base += 4 * kEncodeThreads) {
      uint2 x[4];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int i = base + r * kEncodeThreads;
        x[r] = i < real ? __ldcs(&mi[i]) : make_uint2(0u, 0u);
      }
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int i = base + r * kEncodeThreads;
        if (i >= G * wk) continue;
        const int f = G == 1 ? 0 : i / wk, w = i - f * wk, rem = C.k - 64 * w;
        if (rem < 64) {
          x[r].x &= rem >= 32 ? ~0u : (1u << rem) - 1u;
          x[r].y &= rem > 32 ? (1u << (rem - 32)) - 1u : 0u;
        } else if (i < real) {
          __stcs((uint2*)(cw + (f0 + f) * (long long)C.words_n) + w, x[r]);
        }
        ((uint2*)u)[i] = x[r];
      }
    }
    // the next frames' messages into L2 meanwhile (whole 16-byte pieces of the batch)
    if (threadIdx.x == 0) {
      const long long fn = f0 + (long long)gridDim.x * G;
      if (fn < frames) {
        const uintptr_t a = ((uintptr_t)(msg + fn * wk) + 15) & ~(uintptr_t)15;
        const uintptr_t e = (uintptr_t)(msg + min(fn + G, frames) * wk) & ~(uintptr_t)15;
        if (e > a)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(e - a)) : "memory");
      }
    }
    __syncthreads();
    dvbt2_parity<G>(C, u, pitch, D.ent, D.U2, D.S, D.P, D.tot);
    const int tail = C.words_n - whole;
    for (int i = threadIdx.x; i < G * tail; i += kEncodeThreads) {
      const int f = i / tail, w = whole + i - f * tail;
      if (f0 + f < frames)
        __stcs((uint2*)(cw + (f0 + f) * (long long)C.words_n) + w,
               make_uint2(dvbt2_code_word(u + f * pitch, D.P + f * wp, C.k, C.n, 2 * w),
                          dvbt2_code_word(u + f * pitch, D.P + f * wp, C.k, C.n, 2 * w + 1)));
    }
    __syncthreads();
  }
}

// Encoder with a dense generator block (codes other than DVB-T2).
__global__ void __launch_bounds__(256) encode_kernel(const DevCode* __restrict__ Cp, const uint64_t* __restrict__ msg,
                                                     long long frames, uint64_t* __restrict__ cw) {
  extern __shared__ __align__(16) uint32_t sm[];
  const DevCode C = *Cp;
  const int wn = (C.n + 31) / 32, wk = (C.k + 31) / 32;
  uint32_t* u = sm;
  uint32_t* c = sm + ((wk + 3) & ~3);  // 16-byte aligned carve-up (scratch holds u64 words)
  uint32_t* scratch = c + ((wn + 3) & ~3);
  for (long long f = blockIdx.x; f < frames; f += gridDim.x) {
    const uint32_t* mi = (const uint32_t*)(msg + f * (long long)C.words_k);
    for (int w = threadIdx.x; w < wk; w += blockDim.x) {
      uint32_t x = mi[w];
      const int rem = C.k - 32 * w;
      if (rem < 32) x &= (1u << rem) - 1u;
      u[w] = x;
    }
    __syncthreads();
    encode_frame(C, u, c, scratch);
    uint32_t* co = (uint32_t*)(cw + f * (long long)C.words_n);
    for (int w = threadIdx.x; w < 2 * C.words_n; w += blockDim.x) co[w] = w < wn ? c[w] : 0u;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) syndrome_kernel(const DevCode* __restrict__ Cp,
                                                       const uint64_t* __restrict__ cw, long long frames,
                                                       uint64_t* __restrict__ synd, int32_t* __restrict__ weight) {
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ int s_w;
  const DevCode C = *Cp;
  const int wn = (C.n + 31) / 32;
  DvbScratch<1> D{};
  if (C.enc_kind == 0) {
    D = dvbt2_carve<1>(C, sm + wn);
    dvbt2_build_entries(C, D.ent);
  }
  for (long long f = blockIdx.x; f < frames; f += gridDim.x) {
    const uint32_t* ci = (const uint32_t*)(cw + f * (long long)C.words_n);
    for (int w = threadIdx.x; w < wn; w += blockDim.x) sm[w] = ci[w];
    if (threadIdx.x == 0) s_w = 0;
    __syncthreads();
    uint32_t* so = synd ? (uint32_t*)(synd + f * (long long)C.words_m) : nullptr;
    int cnt = 0;
    if (C.enc_kind == 0) {
      // s_p = (info syndrome of check p) ^ c[k + p] ^ c[k + p - 1], natural order
      const int k = C.k, m = C.m, wm = (m + 31) >> 5;
      uint32_t* nat = D.P;
      for (int w = threadIdx.x; w <= wm; w += blockDim.x) nat[w] = 0u;
      dvbt2_row_groups<1>(C, sm, 0, D.ent, D.U2, D.S);
      const Transpose32 tr(threadIdx.x & 31);
      for (int T = threadIdx.x >> 5; T < 12; T += blockDim.x >> 5) {
        uint32_t x[1][3];
        dvbt2_columns<1>(tr, D.S, C.enc_q, T, x);
        const int t = 32 * T + (threadIdx.x & 31);
        if (t < 360) dvbt2_or_bits(x[0], C.enc_q, t, nat);
      }
      __syncthreads();
      auto par_word = [&](int w) -> uint32_t {  // codeword bits k + 32 w .. + 31
        const int pos = k + 32 * w, i = pos >> 5;
        return __funnelshift_r(sm[i], i + 1 < wn ? sm[i + 1] : 0u, pos & 31);
      };
      for (int w = threadIdx.x; w < 2 * C.words_m; w += blockDim.x) {
        uint32_t x = 0;
        if (w < wm) {
          const uint32_t pw = par_word(w), prev = w > 0 ? par_word(w - 1) : 0u;
          x = nat[w] ^ pw ^ ((pw << 1) | (prev >> 31));
          if (w == wm - 1 && (m & 31)) x &= (1u << (m & 31)) - 1u;
        }
        cnt += __popc(x);
        if (so) so[w] = x;
      }
      atomicAdd(&s_w, cnt);
      __syncthreads();
      if (threadIdx.x == 0 && weight) weight[f] = s_w;
      __syncthreads();
      continue;
    }
    for (int base = 0; base < 32 * 2 * C.words_m; base += blockDim.x) {
      const int p = base + threadIdx.x;
      uint32_t s = 0;
      if (p < C.m) {
        const int e1 = __ldg(&C.csr_ptr[p + 1]);
        for (int e = __ldg(&C.csr_ptr[p]); e < e1; e++) s ^= getbit(sm, __ldg(&C.csr_idx[e]));
      }
      cnt += s;
      const uint32_t b = __ballot_sync(0xffffffffu, s);
      // a frame owns 2 * words_m 32-bit words; base is a multiple of 32, so lane
      // 0 bounds the whole warp's word
      if ((threadIdx.x & 31) == 0 && so && p < 64 * C.words_m) so[p >> 5] = b;
    }
    atomicAdd(&s_w, cnt);
    __syncthreads();
    if (threadIdx.x == 0 && weight) weight[f] = s_w;
    __syncthreads();
  }
}

// LLRs of one frame with codeword bits c.  Not inlined: the loop is bound by FP64
// arithmetic and wants the registers that the encoder in front of it would hold
// (3000 normal 3/5 frames: 1.51 ms inlined, 1.41 ms).
__device__ __noinline__ void channel_llrs(const uint32_t* c, int n, uint32_t fr, uint2 key, double s2, float* lo) {
  const double sigma = __dsqrt_rn(s2);
  for (int pair = threadIdx.x; 2 * pair < n; pair += blockDim.x) {
    const uint4 r = philox4x32_10(make_uint4((uint32_t)pair, fr, 2u, 0u), key);
    const unsigned long long a = (((unsigned long long)r.x << 32) | r.y) >> 11;
    const unsigned long long b = (((unsigned long long)r.z << 32) | r.w) >> 11;
    const double u1 = __dmul_rn((double)(a + 1ull), 1.1102230246251565404e-16);
    const double u2 = __dmul_rn((double)b, 1.1102230246251565404e-16);
    const double rad = __dsqrt_rn(__dmul_rn(-2.0, log_d(u1)));
    double sn, cs;
    sincos_2pi_d(u2, &sn, &cs);
    const double z[2] = {__dmul_rn(rad, cs), __dmul_rn(rad, sn)};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = 2 * pair + h;
      if (i < n) {
        const double sym = getbit(c, i) ? -1.0 : 1.0;
        const double y = __dadd_rn(sym, __dmul_rn(sigma, z[h]));
        lo[i] = __double2float_rn(__ddiv_rn(__dmul_rn(2.0, y), s2));
      }
    }
  }
}

__global__ void __launch_bounds__(kEncThreads) channel_kernel(const DevCode* __restrict__ Cp, uint2 key,
                                                              unsigned long long frame0, long long frames,
                                                              const double* __restrict__ sigma2,
                                                              uint64_t* __restrict__ info,
                                                              uint64_t* __restrict__ cwo, float* __restrict__ llr) {
  extern __shared__ __align__(16) uint32_t sm[];
  const DevCode C = *Cp;
  const int wn = (C.n + 31) / 32, wk = (C.k + 31) / 32;
  uint32_t* u = sm;
  uint32_t* c = sm + ((wk + 3) & ~3);  // 16-byte aligned carve-up (scratch holds u64 words)
  uint32_t* scratch = c + ((wn + 3) & ~3);
  if (C.enc_kind == 0) dvbt2_build_entries(C, dvbt2_carve<1>(C, scratch).ent);
  for (long long f = blockIdx.x; f < frames; f += gridDim.x) {
    const uint32_t fr = (uint32_t)(frame0 + (unsigned long long)f);
    // info bits: 128 per Philox call, counter (block, frame, 1, 0)
    for (int blk = threadIdx.x; blk * 128 < C.k; blk += blockDim.x) {
      const uint4 r = philox4x32_10(make_uint4((uint32_t)blk, fr, 1u, 0u), key);
      const uint32_t wv[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int w = blk * 4 + q;
        if (w < wk) {
          uint32_t x = wv[q];
          const int rem = C.k - 32 * w;
          if (rem < 32) x &= (1u << rem) - 1u;
          u[w] = x;
        }
      }
    }
    __syncthreads();
    encode_frame(C, u, c, scratch);
    if (info) {
      uint32_t* io = (uint32_t*)(info + f * (long long)C.words_k);
      for (int w = threadIdx.x; w < 2 * C.words_k; w += blockDim.x) io[w] = w < wk ? u[w] : 0u;
    }
    if (cwo) {
      uint32_t* co = (uint32_t*)(cwo + f * (long long)C.words_n);
      for (int w = threadIdx.x; w < 2 * C.words_n; w += blockDim.x) co[w] = w < wn ? c[w] : 0u;
    }
    if (llr) channel_llrs(c, C.n, fr, key, sigma2[f], llr + f * (long long)C.n);
    __syncthreads();
  }
}

// Bit and frame errors between two packed bit batches (the FER / BER counters
// of a Monte Carlo point; the reference's counterpart is the uncoded runner
// SimulationRunner, crates/gf2-coding/src/simulation.rs:140-193).
// totals[0] += frames with at least one error, totals[1] += bit errors.
__global__ void __launch_bounds__(256) count_errors_kernel(const uint64_t* __restrict__ a,
                                                           const uint64_t* __restrict__ b, long long frames,
                                                           int words, int32_t* __restrict__ per_frame,
                                                           unsigned long long* __restrict__ totals) {
  __shared__ unsigned long long s_bits, s_frames;
  if (threadIdx.x == 0) {
    s_bits = 0;
    s_frames = 0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  for (long long f = (long long)blockIdx.x * nwarp + warp; f < frames; f += (long long)gridDim.x * nwarp) {
    int e = 0;
    for (int w = lane; w < words; w += 32) e += __popcll(a[f * words + w] ^ b[f * words + w]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) {
      if (per_frame) per_frame[f] = e;
      if (e) {
        atomicAdd(&s_bits, (unsigned long long)e);
        atomicAdd(&s_frames, 1ull);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_frames) atomicAdd(&totals[0], s_frames);
    if (s_bits) atomicAdd(&totals[1], s_bits);
  }
}

int launch_count_errors(const uint64_t* a, const uint64_t* b, long long frames, int words, int32_t* per_frame,
                        unsigned long long* totals, cudaStream_t st) {
  if (frames <= 0) return GF2C_OK;
  int grid = (int)std::min<long long>((frames + 7) / 8, 148 * 8);
  count_errors_kernel<<<grid, 256, 0, st>>>(a, b, frames, words, per_frame, totals);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

static int grid_for(long long frames) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long g = std::min<long long>(frames, (long long)sms * 2);
  return (int)std::max<long long>(g, 1);
}

template <int G>
static int launch_encode_dvb(const DevCode* dcode, const DevCode& h, const uint64_t* msg, long long frames,
                             uint64_t* cw, int sms, cudaStream_t st) {
  const size_t smem =
      (size_t)(((2 * h.words_k * G + 3) & ~3) + dvbt2_scratch_words(h.k / 360, h.enc_q, h.m, h.enc_rg_total, G)) * 4;
  int per_sm = 1;
  GF2C_CUDA(allow_smem((const void*)encode_dvb_kernel<G>, smem));
  GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_dvb_kernel<G>, kEncodeThreads, smem));
  const long long grid = std::min<long long>((frames + G - 1) / G, (long long)sms * std::max(per_sm, 1));
  encode_dvb_kernel<G><<<(int)grid, kEncodeThreads, smem, st>>>(dcode, msg, frames, cw);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

int launch_encode(const DevCode* dcode, const DevCode& h, const uint64_t* msg, long long frames,
                  uint64_t* cw, cudaStream_t st) {
  if (frames <= 0) return GF2C_OK;
  int dev = 0, sms = 148, per_sm = 1;
  GF2C_CUDA(cudaGetDevice(&dev));
  GF2C_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // DVB-T2: bound by instruction issue and the latency between the six short
  // phases of a frame (two CTAs of 12 warps per SM, issue slots 46 % busy).  Four
  // frames per CTA share the table entries, the addresses and the barriers: 5.5
  // K warp instructions per normal 3/5 frame (one frame per CTA: 7.2 K; before,
  // with a division and a modulo per word and address, a prefix pass over the
  // words and a shift-and-mask transpose: 13.7 K).  65536 normal 3/5 frames:
  // 1.27 ms before, 0.84 ms one frame at a time, 0.72 ms four, 0.65 ms with the
  // messages loaded together and the next ones prefetched.  Batches that would
  // leave SMs without a CTA of four frames take one frame at a time.
  if (h.enc_kind == 0)
    return frames >= 8ll * sms ? launch_encode_dvb<4>(dcode, h, msg, frames, cw, sms, st)
                               : launch_encode_dvb<1>(dcode, h, msg, frames, cw, sms, st);
  size_t smem = encode_smem(h);
  GF2C_CUDA(allow_smem((const void*)encode_kernel, smem));
  GF2C_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_kernel, 256, smem));
  const long long grid = std::max<long long>(1, std::min<long long>(frames, (long long)sms * std::max(per_sm, 1)));
  encode_kernel<<<(int)grid, 256, smem, st>>>(dcode, msg, frames, cw);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

int launch_syndrome(const DevCode* dcode, const DevCode& h, const uint64_t* cw, long long frames,
                    uint64_t* synd, int32_t* weight, cudaStream_t st) {
  if (frames <= 0) return GF2C_OK;
  size_t smem = (size_t)((h.n + 31) / 32) * 4;
  if (h.enc_kind == 0) smem += (size_t)dvbt2_scratch_words(h.k / 360, h.enc_q, h.m, h.enc_rg_total, 1) * 4;
  GF2C_CUDA(allow_smem((const void*)syndrome_kernel, smem));
  syndrome_kernel<<<grid_for(frames), 256, smem, st>>>(dcode, cw, frames, synd, weight);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

int launch_channel(const DevCode* dcode, const DevCode& h, uint64_t seed, uint64_t frame0,
                   long long frames, const double* sigma2, uint64_t* info, uint64_t* cw, float* llr,
                   cudaStream_t st) {
  if (frames <= 0) return GF2C_OK;
  size_t smem = encode_smem(h);
  GF2C_CUDA(allow_smem((const void*)channel_kernel, smem));
  uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  channel_kernel<<<grid_for(frames), kEncThreads, smem, st>>>(dcode, key, frame0, frames, sigma2, info, cw, llr);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

}  // namespace gf2c
