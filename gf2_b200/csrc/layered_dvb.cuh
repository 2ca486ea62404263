// gf2cuda layered decoder of the DVB-T2 codes (sm_100a): the kernels of
// layered_impl.cuh specialised to row groups of 360 checks.
//
// Same schedule, arithmetic and update order as layered_iterations, so results
// are bit-identical; what differs is the work around the arithmetic.  The
// kernel is bound by instruction issue and the ALU pipe as much as by the
// latency of the posterior gathers (see bp_layered_dvb_kernel for the figures):
//   - the circulant size is a constant, so message addresses are
//     immediate offsets of one base;
//   - the posteriors' memory space is a template parameter (PL_GLOBAL: the
//     CTA's workspace, PL_SHARED: short frames), not a generic pointer;
//   - slot descriptors and row-group records are in shared memory (the streams
//     of posteriors evict them from L1 between two uses by one CTA);
//   - sign masks come from sign bits by funnel shifts.  LLRs enter as llr +
//     0.0f (-0 becomes +0, a NaN the positive canonical one) and every later
//     posterior and v2c is the result of an addition of which not both terms
//     are -0, so the sign bit is the comparison x < 0;
//   - the syndrome test reads the hard-decision bitmap 32 checks at a time (a
//     slot of a row group is a rotated run of 360 bits).
// Row groups with repeated variables, and the first row group (its first
// check lacks one edge, the staircase's corner), take the SLOW row variants.
#pragma once
#include "layered_impl.cuh"

namespace gf2c {

constexpr int kDvbZ = 360;
enum { PL_GLOBAL = 0, PL_SHARED = 1 };

// Row groups of at most D slots; irregular short codes have as few as this.
__host__ __device__ constexpr int dvb_min_slots(int D) { return D == 7 ? 4 : D == 13 ? 9 : D == 19 ? 16 : D; }

// Row-group records and slot descriptors in shared memory.
struct DvbTab {
  const int4* cg;    // per row group {slots, first message, first descriptor, sync bits}
  const int2* desc;  // {start, wrap}
};
__host__ __device__ constexpr size_t dvb_tab_bytes(int ncg, int ndesc) { return (size_t)ncg * 16 + (size_t)ndesc * 8; }

__device__ __forceinline__ int dvb_u(const int2 S, int t) { return S.x + t - (t >= S.y ? kDvbZ : 0); }

// One check's slots: variables and posteriors (slots >= d of an irregular row
// group and the corner's missing slot read `neutral`).
template <int D, bool PART, bool SLOW>
__device__ __forceinline__ void dvb_load(const int2* sd, int t, const float* app, int d, bool corner, float neutral,
                                         int (&u)[D], float (&ap)[D]) {
#pragma unroll
  for (int i = 0; i < D; i++) {
    u[i] = 0;
    ap[i] = neutral;
    if (!PART || i < dvb_min_slots(D) || i < d) {
      u[i] = dvb_u(sd[i], t);
      ap[i] = app[u[i]];
    }
    if (SLOW) ap[i] = (corner && i == (PART ? d : D) - 2) ? neutral : ap[i];
  }
}

// Toggle the bitmap bits of the slots set in m (slot i at bit D - 1 - i): rare
// after the first iterations.
template <int D>
__device__ __forceinline__ void dvb_flips(uint32_t m, const int2* sd, int t, const LayerSmem& S) {
  while (m) {
    const int b = __ffs(m) - 1;
    m &= m - 1;
    flip_var(dvb_u(sd[D - 1 - b], t), S);
  }
}

// Stores the new posterior of slot i, or (a slot inside a run of one block,
// SLOW) its delta for phase B; rank counts the run slots so far.
template <bool SLOW>
__device__ __forceinline__ void dvb_put(float* app, int u, float ap, float delta, float nw, bool run, bool skip, int t,
                                        int& rank, float* dbuf, uint32_t& newneg) {
  if (SLOW && run) {
    dbuf[rank * kDvbZ + t] = delta;
    rank++;
    newneg = __funnelshift_l(__float_as_uint(ap), newneg, 1);  // unchanged until phase B
  } else {
    if (!(SLOW && skip)) app[u] = nw;
    newneg = __funnelshift_l(__float_as_uint(nw), newneg, 1);
  }
}

// Compressed states of the min-sum family (see StateOld): slot i's sign at bit
// 31 - i, the argmin slot in the low five bits.
struct DvbState {
  float r1, r2;
  uint32_t w;
};
template <int MSG16>
__device__ __forceinline__ DvbState dvb_load_state(const void* cst, int ci) {
  if constexpr (MSG16) {
    const uint2 v = __ldcs((const uint2*)cst + ci);
    return DvbState{__half2float(__ushort_as_half((unsigned short)(v.x & 0xffffu))),
                    __half2float(__ushort_as_half((unsigned short)(v.x >> 16))), v.y};
  } else {
    const uint4 v = __ldcs((const uint4*)cst + ci);
    return DvbState{__uint_as_float(v.x), __uint_as_float(v.y), v.z};
  }
}
template <int MSG16>
__device__ __forceinline__ void dvb_store_state(void* cst, int ci, float r1, float r2, uint32_t w) {
  if constexpr (MSG16) {
    const uint32_t h1 = __half_as_ushort(__float2half_rn(r1)), h2 = __half_as_ushort(__float2half_rn(r2));
    __stcs((uint2*)cst + ci, make_uint2(h1 | (h2 << 16), w));
  } else {
    __stcs((uint4*)cst + ci, make_uint4(__float_as_uint(r1), __float_as_uint(r2), w, 0u));
  }
}

// Normalised / offset min-sum update of check t (the arithmetic of ms_row /
// ms_rep_a).  A slot whose magnitude equals the minimum gets the second one:
// where several do, the two are equal.
template <int MSG16, int D, bool PART, bool SLOW>
__device__ __forceinline__ void dvb_ms_row(const int2* sd, int t, int ci, float* app, void* cst, bool first, float al,
                                           float be, uint32_t sync, bool corner, float* dbuf, const LayerSmem& S,
                                           int d) {
  typedef MsgIO<MSG16> IO;
  const float inf = __int_as_float(0x7f800000);
  // Registers: many slots recompute the old message and the address instead of
  // keeping them
  constexpr bool KEEP_O = D <= 11, KEEP_U = D <= 14;
  int u[D];
  float ap[D], o[KEEP_O ? D : 1], w[D];
  const DvbState st = first ? DvbState{0.0f, 0.0f, 0u} : dvb_load_state<MSG16>(cst, ci);
  dvb_load<D, PART, SLOW>(sd, t, app, d, corner, inf, u, ap);
  const int i0 = (int)(st.w & 31u);
  auto old_of = [&](int i) {
    return __uint_as_float(__float_as_uint(i == i0 ? st.r2 : st.r1) ^ ((st.w << i) & 0x80000000u));
  };
  float m1 = inf, m2 = inf;
  uint32_t neg = 0, oldneg = 0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const float oi = old_of(i);
    if constexpr (KEEP_O) o[i] = oi;
    w[i] = __fsub_rn(ap[i], oi);
    const float ax = fabsf(w[i]);
    m2 = fmaxf(m1, fminf(m2, ax));
    m1 = fminf(m1, ax);
    neg = __funnelshift_l(__float_as_uint(w[i]), neg, 1);
    oldneg = __funnelshift_l(__float_as_uint(ap[i]), oldneg, 1);
  }
  const float d1 = __fsub_rn(m1, be), d2 = __fsub_rn(m2, be);
  const float r1 = IO::rt(__fmul_rn(al, d1 > 0.0f ? d1 : 0.0f)), r2 = IO::rt(__fmul_rn(al, d2 > 0.0f ? d2 : 0.0f));
  const uint32_t par = (uint32_t)__popc(neg) << 31;  // bit 31: parity of the signs
  const uint32_t q1 = __float_as_uint(r1) ^ par, q2 = __float_as_uint(r2) ^ par;
  const uint32_t rep = sync | (sync << 1);
  int rank = 0;
  uint32_t newneg = 0, i1 = 31u;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const bool mn = fabsf(w[i]) == m1;
    i1 = mn ? (uint32_t)i : i1;
    const float out = __uint_as_float((mn ? q2 : q1) ^ (__float_as_uint(w[i]) & 0x80000000u));
    const float delta = __fsub_rn(out, KEEP_O ? o[KEEP_O ? i : 0] : old_of(i));
    const float nw = __fadd_rn(ap[i], delta);
    if (!PART || i < dvb_min_slots(D) || i < d)
      dvb_put<SLOW>(app, KEEP_U ? u[i] : dvb_u(sd[i], t), ap[i], delta, nw, (rep >> i) & 1u,
                    corner && i == (PART ? d : D) - 2, t, rank, dbuf, newneg);
    else
      newneg <<= 1;
  }
  // sign bits slot 0 first; the slots below the lowest stay within bits 31..10
  const uint32_t sgn = (neg ^ (0u - (par >> 31))) << (32 - D);
  dvb_store_state<MSG16>(cst, ci, r1, r2, (sgn & ~31u) | i1);
  dvb_flips<D>(oldneg ^ newneg, sd, t, S);
}

// Old messages of one check in a sum-product row group (slot i at a constant
// offset), read into registers before anything waits; binary16 messages stay
// packed in pairs, since rows with repeated variables need them twice.
template <int MSG16, int D>
struct DvbOld {
  uint32_t w[MSG16 ? (D + 1) / 2 : D];
  __device__ __forceinline__ float get(int i) const {
    if constexpr (MSG16) return __half2float(__ushort_as_half((unsigned short)(w[i >> 1] >> (16 * (i & 1)))));
    else return __uint_as_float(w[i]);
  }
  // raw(i): the stored bits of slot i; slots >= d hold nothing
  template <class F>
  __device__ __forceinline__ void load(F raw, bool part, int least, int d) {
#pragma unroll
    for (int i = 0; i < (MSG16 ? (D + 1) / 2 : D); i++) {
      if constexpr (MSG16) {
        const int a = 2 * i, b = 2 * i + 1;
        const uint32_t lo = (!part || a < least || a < d) ? raw(a) : 0u;
        const uint32_t hi = b < D && (!part || b < least || b < d) ? raw(b) : 0u;
        w[i] = lo | (hi << 16);
      } else {
        w[i] = (!part || i < least || i < d) ? raw(i) : 0u;
      }
    }
  }
};

// Sum-product (SFU) update of check t (the arithmetic of spa_fast_row /
// spa_fast_rep_a): the posterior is v2c + c2v_new in plain row groups and
// APP + (c2v_new - c2v_old) in those with repeated variables.
template <int MSG16, int D, bool PART, bool SLOW>
__device__ __forceinline__ void dvb_spa_row(const int2* sd, int t, float* app, typename MsgIO<MSG16>::T* msg, bool first, uint32_t sync, bool corner, float* dbuf,
                                            const LayerSmem& S, int d) {
  const float big = 3.402823466e38f;
  constexpr bool KEEP_U = D <= 14;
  int u[D];
  float x[D], e[D];
  DvbOld<MSG16, D> old;
  if (!first)
    old.load(
        [&](int i) -> uint32_t {
          if constexpr (MSG16) return __ldcs((const unsigned short*)msg + i * kDvbZ);
          else return __ldcs((const uint32_t*)msg + i * kDvbZ);
        },
        PART, dvb_min_slots(D), d);
  else
    old.load([](int) -> uint32_t { return 0u; }, PART, dvb_min_slots(D), d);
  dvb_load<D, PART, SLOW>(sd, t, app, d, corner, big, u, x);
  uint32_t neg = 0, oldneg = 0;
  float N = 1.0f, Dp = 1.0f;
#pragma unroll
  for (int i = 0; i < D; i++) {
    oldneg = __funnelshift_l(__float_as_uint(x[i]), oldneg, 1);
    // the first iteration's old messages are +0 (x - 0 = x)
    if (!PART || i < dvb_min_slots(D) || i < d) x[i] = __fsub_rn(x[i], old.get(i));
    if (SLOW) x[i] = (corner && i == (PART ? d : D) - 2) ? big : x[i];
    neg = __funnelshift_l(__float_as_uint(x[i]), neg, 1);
    e[i] = ex2_approx(fabsf(x[i]) * -1.4426950408889634f);
    N *= fmaxf(1.0f - e[i], 5.9604645e-08f);
    Dp = __fmaf_rn(Dp, e[i], Dp);
  }
  const uint32_t par = (uint32_t)__popc(neg) << 31;
  auto message = [&](int i) {
    const float ni = fmaxf(1.0f - e[i], 5.9604645e-08f), di = 1.0f + e[i];
    const float num = __fmaf_rn(Dp, ni, N * di);
    const float den = fmaxf(__fmaf_rn(Dp, ni, -N * di), num * 5.9604645e-08f);
    const float mag = fminf(0.69314718055994531f * lg2_approx(num * rcp_approx(den)), 16.635532f);
    return __uint_as_float(__float_as_uint(mag) ^ ((__float_as_uint(x[i]) ^ par) & 0x80000000u));
  };
  uint32_t newneg = 0;
  if (SLOW && sync) {
    // posteriors re-read a few at a time, ahead of the stores they may not alias
    const uint32_t rep = sync | (sync << 1);
    int rank = 0;
#pragma unroll
    for (int i0 = 0; i0 < D; i0 += 4) {
      float ap[4];
      int v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int i = i0 + q;
        ap[q] = big;
        v[q] = 0;
        if (i < D && (!PART || i < dvb_min_slots(D) || i < d)) {
          v[q] = KEEP_U ? u[i < D ? i : 0] : dvb_u(sd[i], t);
          ap[q] = app[v[q]];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int i = i0 + q;
        if (i >= D) continue;
        if (PART && i >= dvb_min_slots(D) && i >= d) {
          newneg <<= 1;
          continue;
        }
        const float out = put_capped_msg<MSG16>(msg, i * kDvbZ, message(i));
        const bool skip = corner && i == (PART ? d : D) - 2;
        const float a = skip ? big : ap[q], delta = out - old.get(i);
        dvb_put<SLOW>(app, v[q], a, delta, __fadd_rn(a, delta), (rep >> i) & 1u, skip, t, rank, dbuf, newneg);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < D; i++) {
      if (PART && i >= dvb_min_slots(D) && i >= d) {
        newneg <<= 1;
        continue;
      }
      const float out = put_capped_msg<MSG16>(msg, i * kDvbZ, message(i));
      const float nw = x[i] + out;
      if (!(SLOW && corner && i == (PART ? d : D) - 2)) app[KEEP_U ? u[i] : dvb_u(sd[i], t)] = nw;
      newneg = __funnelshift_l(__float_as_uint(nw), newneg, 1);
    }
  }
  dvb_flips<D>(oldneg ^ newneg, sd, t, S);
}

// Phase B of a row group with repeated variables: the thread of each run's
// first slot adds the run's deltas to its variable in slot order.
__device__ __forceinline__ void dvb_rep_b(const int2* sd, int t, float* app, uint32_t sync, const float* dbuf,
                                          const LayerSmem& S) {
  const uint32_t rep = sync | (sync << 1);
  for (uint32_t heads = sync & ~(sync << 1); heads; heads &= heads - 1) {
    const int i = __ffs(heads) - 1;
    int k = __popc(rep & ((1u << i) - 1u));
    const int v = dvb_u(sd[i], t);
    const float ov = app[v];
    float nw = __fadd_rn(ov, dbuf[k * kDvbZ + t]);
    for (int j = i + 1; (sync >> (j - 1)) & 1u; j++) {
      k++;
      int tj = v - sd[j].x;  // the check of slot j that holds v
      if (tj < 0) tj += kDvbZ;
      nw = __fadd_rn(nw, dbuf[k * kDvbZ + tj]);
    }
    app[v] = nw;
    if ((__float_as_uint(ov) ^ __float_as_uint(nw)) >> 31) flip_var(v, S);
  }
}

// Syndrome of the hard decisions in the bitmap, 32 checks per task: bit t of a
// slot's run is block bit (t + shift) mod 360, a window of the bitmap.  Passes
// of blockDim tasks, each ending at a barrier, stop at the first one with an
// unsatisfied check.
__device__ __forceinline__ uint32_t bit_window(const uint32_t* w, int pos) {
  return __funnelshift_r(w[pos >> 5], w[(pos >> 5) + 1], pos & 31);
}
__device__ __forceinline__ bool dvb_syndrome_zero(const DvbTab T, int ncg, uint32_t absent0, const uint32_t* bitmap) {
  const int tasks = ncg * 12;
  for (int base = 0; base < tasks; base += blockDim.x) {
    const int k = base + threadIdx.x;
    uint32_t p = 0;
    if (k < tasks) {
      const int g = k / 12, w = k - 12 * g;
      const int4 G = T.cg[g];
      for (int i = 0; i < G.x; i++) {
        const int2 D = T.desc[G.z + i];
        const int blk = D.x + D.y - kDvbZ;  // the block's first variable (start - shift)
        int s = 32 * w + kDvbZ - D.y;
        if (s >= kDvbZ) s -= kDvbZ;
        uint32_t x = bit_window(bitmap, blk + s);
        const int left = kDvbZ - s;  // bits before the block wraps
        if (left < 32) x = (x & ((1u << left) - 1u)) | (bit_window(bitmap, blk) << left);
        if (k == 0 && ((absent0 >> i) & 1u)) x &= ~1u;
        p ^= x;
      }
      if (w == 11) p &= 0xffu;
    }
    if (__syncthreads_or(p != 0u)) return false;
  }
  return true;
}

// Iterations of one frame; the counterpart of layered_iterations.
template <int ALGO, int MSG16, int D, bool PART, bool MULTI>
__device__ __forceinline__ void dvb_iterations(const DecodeArgs& a, const DevCode& C, const DvbTab T, float* app,
                                               typename MsgIO<MSG16>::T* __restrict__ c2v, const LayerSmem& S,
                                               int maxit, bool prefetch, int& it, int& converged) {
  const int tid = threadIdx.x, ncg = C.ncg;
  const int NT = MULTI ? (int)blockDim.x : (1 << 30);
  constexpr bool MS = ALGO == L_NMS || ALGO == L_MS;
  const uint32_t absent0 = __ldg(&C.sp_absent[0]);
  it = 0;
  converged = 0;
  for (;;) {
    const int tw = (a.nms_iters > 0) ? min(it, a.nms_iters - 1) : 0;
    const bool first = (it == 0);
    for (int g = 0; g < ncg; g++) {
      const int4 G = T.cg[g];
      const int d = G.x;
      const uint32_t sync = (uint32_t)G.w;
      const int2* sd = T.desc + G.z;
      if constexpr (!MS) {
        // the next row group's old messages into L2, and (posteriors in the
        // workspace) slot i's variable group by lane i of the last warp, which
        // has the fewest checks: 2048 normal 3/5 frames 57.8 -> 56.5 ms,
        // 8192 frames of the twelve codes mixed 27.2 -> 26.5 ms
        if (tid >= (int)blockDim.x - 32) {
          const int lane = tid & 31, gn = (g + 1 < ncg) ? g + 1 : 0;
          const int4 Gn = T.cg[gn];
          if (prefetch && lane < Gn.x) {
            const int2 P = T.desc[Gn.z + lane];
            prefetch_l2(app + (P.x + P.y - kDvbZ), (uint32_t)kDvbZ * 4u);
          }
          if (lane == 31 && !first) prefetch_l2(c2v + Gn.y, (uint32_t)(Gn.x * kDvbZ * (MSG16 ? 2 : 4)));
        }
      }
      if constexpr (MS && MULTI) {
        // lane i of the last warp: slot i's variable group of the next row
        // group into L2 (lane 31: its compressed states)
        if (prefetch && (tid >> 5) == ((int)blockDim.x >> 5) - 1) {
          const int lane = tid & 31, gn = (g + 1 < ncg) ? g + 1 : 0;
          const int4 Gn = T.cg[gn];
          if (lane < Gn.x) {
            const int2 P = T.desc[Gn.z + lane];
            prefetch_l2(app + (P.x + P.y - kDvbZ), (uint32_t)kDvbZ * 4u);
          } else if (lane == 31) {
            prefetch_l2((const char*)c2v + (size_t)gn * kDvbZ * (MSG16 ? 8 : 16), (uint32_t)kDvbZ * (MSG16 ? 8u : 16u));
          }
        }
      }
      float al = 1.0f, be = 0.0f;
      if constexpr (MS) {
        const int lay = (a.nms_L == ncg) ? g : 0;
        al = __ldg(&a.alpha[tw * a.nms_L + lay]);
        be = __ldg(&a.beta[tw * a.nms_L + lay]);
      }
      const bool slow = sync != 0 || (g == 0 && absent0 != 0);
      for (int t = tid; t < kDvbZ; t += NT) {
        const bool corner = g == 0 && t == 0 && absent0 != 0;
        if constexpr (MS) {
          const int ci = g * kDvbZ + t;
          if (!slow)
            dvb_ms_row<MSG16, D, PART, false>(sd, t, ci, app, c2v, first, al, be, 0u, false, nullptr, S, d);
          else
            dvb_ms_row<MSG16, D, PART, true>(sd, t, ci, app, c2v, first, al, be, sync, corner, S.dbuf, S, d);
        } else {
          typename MsgIO<MSG16>::T* msg = c2v + G.y + t;
          if (!slow)
            dvb_spa_row<MSG16, D, PART, false>(sd, t, app, msg, first, 0u, false, nullptr, S, d);
          else
            dvb_spa_row<MSG16, D, PART, true>(sd, t, app, msg, first, sync, corner, S.dbuf, S, d);
        }
      }
      if (sync) {
        __syncthreads();
        for (int t = tid; t < kDvbZ; t += NT) dvb_rep_b(sd, t, app, sync, S.dbuf, S);
      }
      __syncthreads();
    }
    ++it;
    if ((a.early_stop || it >= maxit) && dvb_syndrome_zero(T, ncg, absent0, S.bitmap)) {
      converged = 1;
      break;
    }
    if (it >= maxit) break;
  }
}

// Persistent decoder of DVB-T2 frames.  Bound by issue slots (56 % busy for the
// min-sum family on normal frames, 60 % for the sum-product, 79 % on short
// frames) next to the latency of the posterior gathers (long scoreboard 3.4 /
// 1.5 / below 0.6 stalls per issue).  Against the general kernel, per
// frame-iteration: normal 2/3 min-sum 423 -> 288 K warp instructions, normal
// 3/5 sum-product 744 -> 591 K.  Old messages are read into registers before
// the posteriors, and rows with repeated variables re-read posteriors four at a
// time: with either load inside the slot loop each slot waited for L2 (mixed
// batch, normal 5/6: 16.7 against 3.3 ms).  Not staged in shared memory by TMA:
// the stage's L1 and proxy fences cost what it hid (2048 normal 3/5 frames 59.0
// against 57.7 ms, short 3/4 5.2 against 4.5 ms).  8192 normal 2/3 frames,
// min-sum: 43.5 -> 26.1 ms; 2048 normal 3/5, sum-product: 82.4 -> 57.7 ms (56.5
// with the L2 prefetch); 4096 short 3/4, sum-product: 7.3 -> 4.5 ms.  Three CTAs of 384 threads per SM
// (56 registers) spill: 57.7 -> 84 ms.  D = 0: a mixed batch, each frame with
// its own code's slot count (PL then is where short frames live, normal ones
// are in the workspace).
template <int ALGO, int MSG16, int D, int MAXT, int MINB, int PL, bool PART>
__global__ void __launch_bounds__(MAXT, MINB) bp_layered_dvb_kernel(const DecodeArgs a) {
  typedef typename MsgIO<MSG16>::T MsgT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long s_frame;
  __shared__ DevCode C;
  uint32_t* bitmap = (uint32_t*)smem_raw;
  float* smem_app = (float*)(smem_raw + ((a.bitmap_words * 4 + 15) & ~15));
  char* work = a.work + (long long)blockIdx.x * a.work_stride;
  MsgT* __restrict__ c2v = (MsgT*)work;
  float* gapp = (float*)(work + a.app_offset);
  constexpr bool MULTI = MAXT < 384;
  const int tid = threadIdx.x, NT = blockDim.x;
  const LayerSmem S{bitmap, a.lay_dbuf_floats ? (float*)(smem_raw + a.lay_dbuf_off) : nullptr};
  int tab_code = -1;

  for (;;) {
    if (tid == 0) {
      const long long q = (long long)atomicAdd(a.queue, 1ull);
      const long long nq = a.frames_dev ? *a.frames_dev : a.frames;  // queue entries
      s_frame = (q < nq) ? (a.order != nullptr ? a.order[q] : q) : -1;
    }
    __syncthreads();
    const long long f = s_frame;
    if (f < 0 || f >= a.frames) break;
    const int cid = a.code_id ? a.code_id[f] : 0;
    if (cid < 0 || cid >= a.ncodes) {
      if (tid == 0) {
        atomicExch(a.status, 1);
        if (a.iters) a.iters[f] = -1;
      }
      __syncthreads();
      continue;
    }
    if (tab_code != cid) {
      if (tid == 0) C = a.codes[cid];
      __syncthreads();
    }
    const int n = C.n, k = C.k, ncg = C.ncg;
    int4* tcg = (int4*)(smem_raw + a.lay_tab_off);
    int2* tdesc = (int2*)(tcg + ncg);
    const DvbTab T{tcg, tdesc};
    if (tab_code != cid) {
      for (int i = tid; i < ncg; i += NT) {
        const int4 G = __ldg(&C.cg[i]);
        tcg[i] = make_int4(G.z, G.w, __ldg(&C.sp_cg[i]).w, (int)__ldg(&C.cg_sync[i]));
      }
      for (int i = tid; i < C.sp_ndesc; i += NT) tdesc[i] = __ldg(&C.sp_desc[i]);
      tab_code = cid;
    }
    const float* __restrict__ llr = a.llr + (a.llr_off ? a.llr_off[f] : f * (long long)n);
    const int maxit = a.max_iter_arr ? a.max_iter_arr[f] : a.max_iter;
    const bool shared_app = PL == PL_SHARED && (D != 0 || n <= a.smem_app_floats);
    float* app = shared_app ? smem_app : gapp;
    uint64_t* mo = a.msg ? a.msg + (a.msg_off ? a.msg_off[f] : f * (long long)C.words_k) : nullptr;
    float* bo = a.beliefs ? a.beliefs + (a.llr_off ? a.llr_off[f] : f * (long long)n) : nullptr;

    if (maxit <= 0) {
      if (mo)
        for (int w = tid; w < C.words_k; w += NT) mo[w] = 0ull;
      if (bo)
        for (int v = tid; v < n; v += NT) bo[v] = 0.0f;
      if (tid == 0) {
        if (a.iters) a.iters[f] = 0;
        if (a.conv) a.conv[f] = 0;
        if (a.synd_ok) a.synd_ok[f] = 1;
      }
      __syncthreads();
      continue;
    }

    // APP = llr (u order: parity bit k + a + q t at k + 360 a + t) and the hard
    // decisions, eight loads in flight per thread
    const int q = ncg;
    for (int base = 0; base < n; base += 8 * NT) {
      float x[8];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int u = base + r * NT + tid;
        int v = u;
        if (u >= k) {
          const int p = u - k, row = p / kDvbZ;
          v = k + row + q * (p - row * kDvbZ);
        }
        x[r] = u < n ? __ldcs(llr + v) + 0.0f : 0.0f;
      }
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int u = base + r * NT + tid;
        if (u < n) app[u] = x[r];
        const unsigned b = __ballot_sync(0xffffffffu, u < n && x[r] < 0.0f);
        if ((tid & 31) == 0 && u < n) bitmap[u >> 5] = b;
      }
    }
    __syncthreads();
    int it = 0, converged = 0;
    if constexpr (D > 0) {
      dvb_iterations<ALGO, MSG16, D, PART, MULTI>(a, C, T, PL == PL_SHARED ? smem_app : gapp, c2v, S, maxit,
                                                  PL == PL_GLOBAL, it, converged);
    } else {
#define GF2C_DVB(DD, P, APP, PF) \
  dvb_iterations<ALGO, MSG16, DD, P, MULTI>(a, C, T, APP, c2v, S, maxit, PF, it, converged)
      if (PL == PL_SHARED && shared_app) {
        switch (C.lay_bucket) {
          case 7: GF2C_DVB(7, true, smem_app, false); break;
          case 9: GF2C_DVB(9, false, smem_app, false); break;
          case 10: GF2C_DVB(10, false, smem_app, false); break;
          case 13: GF2C_DVB(13, true, smem_app, false); break;
          default: GF2C_DVB(19, true, smem_app, false); break;
        }
      } else if (PL == PL_GLOBAL && n <= 16200) {  // short frames in the workspace too
        switch (C.lay_bucket) {
          case 7: GF2C_DVB(7, true, gapp, true); break;
          case 9: GF2C_DVB(9, false, gapp, true); break;
          case 10: GF2C_DVB(10, false, gapp, true); break;
          case 13: GF2C_DVB(13, true, gapp, true); break;
          default: GF2C_DVB(19, true, gapp, true); break;
        }
      } else {
        switch (C.lay_bucket) {
          case 7: GF2C_DVB(7, false, gapp, true); break;
          case 10: GF2C_DVB(10, false, gapp, true); break;
          case 11: GF2C_DVB(11, false, gapp, true); break;
          case 14: GF2C_DVB(14, false, gapp, true); break;
          case 18: GF2C_DVB(18, false, gapp, true); break;
          default: GF2C_DVB(22, false, gapp, true); break;
        }
      }
#undef GF2C_DVB
    }
    if (mo) {
      const int wn = (n + 31) >> 5;
      for (int w = tid; w < C.words_k; w += NT) {
        const uint32_t lo = bitmap[2 * w];
        const uint32_t hi = (2 * w + 1 < wn) ? bitmap[2 * w + 1] : 0u;
        unsigned long long word = (unsigned long long)lo | ((unsigned long long)hi << 32);
        const int rem = k - 64 * w;
        if (rem < 64) word &= (1ull << rem) - 1ull;
        mo[w] = word;
      }
    }
    if (bo)
      for (int u = tid; u < n; u += NT) {
        int v = u;
        if (u >= k) {
          const int p = u - k, row = p / kDvbZ;
          v = k + row + q * (p - row * kDvbZ);
        }
        bo[v] = app[u];
      }
    if (tid == 0) {
      if (a.iters) a.iters[f] = it + a.iters_add;
      if (a.conv) a.conv[f] = (uint8_t)converged;
      if (a.synd_ok) a.synd_ok[f] = (uint8_t)converged;
    }
    __syncthreads();
  }
}

// Kernel of one DVB-T2 code: slot bucket and placement as the twelve codes
// have them (short frames' posteriors in shared memory, normal ones' in the
// workspace); D = 0: mixed batches.
template <int ALGO, int MSG16, int MAXT, int MINB>
static const void* dvb_exact(int D, bool shared_app) {
  if (shared_app) {
    switch (D) {
      case 7: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 7, MAXT, MINB, PL_SHARED, true>;
      case 9: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 9, MAXT, MINB, PL_SHARED, false>;
      case 10: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 10, MAXT, MINB, PL_SHARED, false>;
      case 13: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 13, MAXT, MINB, PL_SHARED, true>;
      case 19: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 19, MAXT, MINB, PL_SHARED, true>;
    }
    return nullptr;
  }
  switch (D) {
    case 7: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 7, MAXT, MINB, PL_GLOBAL, false>;
    case 10: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 10, MAXT, MINB, PL_GLOBAL, false>;
    case 11: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 11, MAXT, MINB, PL_GLOBAL, false>;
    case 14: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 14, MAXT, MINB, PL_GLOBAL, false>;
    case 18: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 18, MAXT, MINB, PL_GLOBAL, false>;
    case 22: return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 22, MAXT, MINB, PL_GLOBAL, false>;
  }
  return nullptr;
}

// threads 384: one check per thread; 192 / 128: two / three (FP16 messages).
template <int ALGO, int MSG16>
static const void* dvb_t(int D, bool shared_app, int threads) {
  if (D == 0) {
    if constexpr (ALGO == L_SPA_FAST) {
      if (threads == 384) return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 0, 384, 2, PL_SHARED, false>;
      if constexpr (MSG16)
        if (threads == 192) return (const void*)bp_layered_dvb_kernel<ALGO, MSG16, 0, 192, 4, PL_GLOBAL, false>;
    }
    return nullptr;
  }
  if (threads == 384) return dvb_exact<ALGO, MSG16, 384, 2>(D, shared_app);
  if constexpr (MSG16) {
    if (threads == 192) return dvb_exact<ALGO, MSG16, 192, 4>(D, shared_app);
    if (threads == 128) return dvb_exact<ALGO, MSG16, 128, 6>(D, shared_app);
  }
  return nullptr;
}

}  // namespace gf2c
