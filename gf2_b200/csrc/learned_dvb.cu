// gf2cuda learned min-sum, layered training on the DVB-T2 codes (sm_100a).
//
// The layered forward and backward of learned.cu (same arithmetic, same order
// of every sum, so losses and gradients are bit-identical) with the row
// structure of layered_dvb.cuh: unrolled slots, descriptors in shared memory,
// posteriors in u order (parity bit k + a + q t at k + 360 a + t).
//
// What the forward saves.  A check's backward needs its two smallest
// magnitudes, their slots and the signs of its inputs, no input itself: one
// 16-byte record per check and iteration {m1, m2, signs | i1 | i2} instead of
// 4 bytes per edge.  The record of iteration t - 1 with that iteration's weights
// is also the check's old messages of iteration t, so the forward keeps no
// message array.  Only the two minimum slots receive a gradient, so a row group
// without repeated variables updates dL/dA with no barrier before it.
//
// Bound by latency: one CTA per frame and one frame's row groups in order (60
// of normal 2/3, ten iterations, both ways), so what counts is the chain of a
// row group: the gathers of a check are in flight together, and the sums of a
// row group's weight-gradient terms are done a row group later, by a warp that
// rotates; the copy engine brings the next row group's records and message
// gradients, which come from DRAM, into L2 meanwhile.  256 normal 2/3 frames,
// T = 10, one loss_grad call: 19.1 ms with per-edge activations and run-time
// slot loops (issue slots 20 % busy, long scoreboard 18 to 20 stalls per
// issue), 4.07 ms with this structure (47 % / 36 %, 4.7 / 8.1), 3.53 ms with the
// prefetch.
#include <algorithm>

#include "layered_dvb.cuh"

namespace gf2c {

static constexpr int kTrainThreads = 384;

__device__ __forceinline__ float train_warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// u-order position of natural variable v.
__device__ __forceinline__ int dvb_u_of(int v, int k, int q) {
  const int p = v - k, t = p / q;
  return v < k ? v : k + (p - t * q) * kDvbZ + t;
}

// Record word: sign of slot i at bit 31 - i, i1 at bits 9..5, i2 at bits 4..0.
__device__ __forceinline__ uint32_t slot_sign(uint32_t w, int i) { return (w << i) & 0x80000000u; }

struct TrainTab {
  DvbTab T;
  float* dbuf;
};

// Tables of the code in dynamic shared memory, behind the run buffer.
__device__ __forceinline__ TrainTab train_tables(const DevCode& C, unsigned char* smem) {
  float* dbuf = (float*)smem;
  int4* tcg = (int4*)(dbuf + C.lay_runs * kDvbZ);
  int2* tdesc = (int2*)(tcg + C.ncg);
  for (int i = threadIdx.x; i < C.ncg; i += blockDim.x) {
    const int4 G = __ldg(&C.cg[i]);
    tcg[i] = make_int4(G.z, G.w, __ldg(&C.sp_cg[i]).w, (int)__ldg(&C.cg_sync[i]));
  }
  for (int i = threadIdx.x; i < C.sp_ndesc; i += blockDim.x) tdesc[i] = __ldg(&C.sp_desc[i]);
  __syncthreads();
  return TrainTab{DvbTab{tcg, tdesc}, dbuf};
}
static size_t train_smem(const DevCode& h) {
  return (size_t)h.lay_runs * kDvbZ * 4 + dvb_tab_bytes(h.ncg, h.sp_ndesc);
}

// Adds the runs' buffered terms to their variables in slot order.
__device__ __forceinline__ void train_runs(const int2* sd, int t, float* a, uint32_t sync, const float* dbuf) {
  const uint32_t rep = sync | (sync << 1);
  for (uint32_t heads = sync & ~(sync << 1); heads; heads &= heads - 1) {
    const int i = __ffs(heads) - 1;
    int k = __popc(rep & ((1u << i) - 1u));
    const int v = dvb_u(sd[i], t);
    float x = __fadd_rn(a[v], dbuf[k * kDvbZ + t]);
    for (int j = i + 1; (sync >> (j - 1)) & 1u; j++) {
      k++;
      int tj = v - sd[j].x;
      if (tj < 0) tj += kDvbZ;
      x = __fadd_rn(x, dbuf[k * kDvbZ + tj]);
    }
    a[v] = x;
  }
}

// Forward of check t: old messages from the record `old` under the weights
// (alp, bep) of the previous iteration, new ones under (al, be).
template <int D, bool PART, bool SLOW>
__device__ __forceinline__ uint4 train_forward_row(const int2* sd, int t, float* app, const uint4 old, float al,
                                                   float be, float alp, float bep, uint32_t sync, bool corner,
                                                   float* dbuf, int d) {
  constexpr bool KEEP_U = D <= 14;
  const float inf = __int_as_float(0x7f800000);
  const float e1 = __fsub_rn(__uint_as_float(old.x), bep), e2 = __fsub_rn(__uint_as_float(old.y), bep);
  const uint32_t o1 = __float_as_uint(__fmul_rn(alp, e1 > 0.0f ? e1 : 0.0f));
  const uint32_t o2 = __float_as_uint(__fmul_rn(alp, e2 > 0.0f ? e2 : 0.0f));
  const int oi1 = (int)((old.z >> 5) & 31u);
  const uint32_t osg = __popc(old.z >> 10) & 1u ? ~old.z : old.z;  // sign of each old message
  auto old_of = [&](int i) { return __uint_as_float((i == oi1 ? o2 : o1) ^ slot_sign(osg, i)); };
  int u[D];
  float ap[D], o[D];
  dvb_load<D, PART, SLOW>(sd, t, app, d, corner, inf, u, ap);
  float m1 = inf, m2 = inf;
  uint32_t i1 = 31u, i2 = 31u, neg = 0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    o[i] = old_of(i);
    const float x = __fsub_rn(ap[i], o[i]);
    const float ax = fabsf(x);
    const bool lt1 = ax < m1, lt2 = ax < m2;
    i2 = lt1 ? i1 : (lt2 ? (uint32_t)i : i2);
    i1 = lt1 ? (uint32_t)i : i1;
    m2 = fmaxf(m1, fminf(m2, ax));
    m1 = fminf(m1, ax);
    neg = __funnelshift_l(__float_as_uint(x), neg, 1);
  }
  const uint32_t word = (neg << (32 - D)) | (i1 << 5) | i2;
  const float d1 = __fsub_rn(m1, be), d2 = __fsub_rn(m2, be);
  const uint32_t par = (uint32_t)__popc(neg) << 31;
  const uint32_t r1 = __float_as_uint(__fmul_rn(al, d1 > 0.0f ? d1 : 0.0f)) ^ par;
  const uint32_t r2 = __float_as_uint(__fmul_rn(al, d2 > 0.0f ? d2 : 0.0f)) ^ par;
  const uint32_t rep = sync | (sync << 1);
  int rank = 0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    if (PART && i >= dvb_min_slots(D) && i >= d) continue;
    const float out = __uint_as_float((i == (int)i1 ? r2 : r1) ^ slot_sign(word, i));
    const float delta = __fsub_rn(out, o[i]);
    if (SLOW && ((rep >> i) & 1u)) {
      dbuf[rank * kDvbZ + t] = delta;
      rank++;
    } else if (!(SLOW && corner && i == (PART ? d : D) - 2)) {
      app[KEEP_U ? u[i] : dvb_u(sd[i], t)] = __fadd_rn(ap[i], delta);
    }
  }
  return make_uint4(__float_as_uint(m1), __float_as_uint(m2), word, 0u);
}

template <int D, bool PART>
__global__ void __launch_bounds__(kTrainThreads, 2) nms_dvb_forward_kernel(
    const DevCode* __restrict__ Cp, int T, int L, const float* __restrict__ llr, const uint64_t* __restrict__ cw,
    long long frames, const float* __restrict__ alpha, const float* __restrict__ beta, uint4* __restrict__ X,
    float* __restrict__ Bout, char* __restrict__ work, long long work_stride, float* __restrict__ pf) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_part[kTrainThreads / 32];
  __shared__ DevCode C;
  const int tid = threadIdx.x, NT = blockDim.x;
  if (tid == 0) C = *Cp;
  __syncthreads();
  const TrainTab S = train_tables(C, smem);
  const int n = C.n, k = C.k, m = C.m, ncg = C.ncg;
  const uint32_t absent0 = __ldg(&C.sp_absent[0]);
  float* app = (float*)(work + (long long)blockIdx.x * work_stride);
  const float scale = 1.0f / ((float)frames * (float)n);
  const int t = min(tid, kDvbZ - 1);
  const bool act = tid < kDvbZ;
  for (long long f = blockIdx.x; f < frames; f += gridDim.x) {
    const float* lf = llr + f * (long long)n;
    for (int base = tid; base < n; base += 8 * NT) {
      float x[8];
#pragma unroll
      for (int r = 0; r < 8; r++) x[r] = base + r * NT < n ? lf[base + r * NT] + 0.0f : 0.0f;
#pragma unroll
      for (int r = 0; r < 8; r++)
        if (base + r * NT < n) app[dvb_u_of(base + r * NT, k, ncg)] = x[r];
    }
    __syncthreads();
    for (int it = 0; it < T; it++) {
      uint4* Xt = X + (f * T + it) * (long long)m;
      for (int g = 0; g < ncg; g++) {
        const int4 G = S.T.cg[g];
        const uint32_t sync = (uint32_t)G.w;
        const int2* sd = S.T.desc + G.z;
        const int lay = (L == ncg) ? g : 0, pt = it > 0 ? it - 1 : 0;
        const float al = __ldg(&alpha[it * L + lay]), be = __ldg(&beta[it * L + lay]);
        const float alp = __ldg(&alpha[pt * L + lay]), bep = __ldg(&beta[pt * L + lay]);
        const bool slow = sync != 0 || (g == 0 && absent0 != 0);
        // the next row group's records
        if (tid == kTrainThreads - 1 && it > 0 && g + 1 < ncg) prefetch_l2(Xt + (g + 1) * kDvbZ - m, kDvbZ * 16);
        if (act) {
          // before the first iteration: two zero magnitudes under the offset
          const uint4 old = it > 0 ? __ldcs(&Xt[g * kDvbZ + t - m]) : make_uint4(0u, 0u, 0u, 0u);
          const float op = it > 0 ? alp : 0.0f, ob = it > 0 ? bep : 0.0f;
          uint4 rec;
          if (!slow)
            rec = train_forward_row<D, PART, false>(sd, t, app, old, al, be, op, ob, 0u, false, nullptr, G.x);
          else
            rec = train_forward_row<D, PART, true>(sd, t, app, old, al, be, op, ob, sync,
                                                   g == 0 && t == 0 && absent0 != 0, S.dbuf, G.x);
          Xt[g * kDvbZ + t] = rec;
        }
        if (sync) {
          __syncthreads();
          if (act) train_runs(sd, t, app, sync, S.dbuf);
        }
        __syncthreads();
      }
    }
    float part = 0.0f;
    const uint64_t* cf = cw + f * (long long)C.words_n;
    for (int base = tid; base < n; base += 4 * NT) {
      float b[4];
#pragma unroll
      for (int r = 0; r < 4; r++) b[r] = base + r * NT < n ? app[dvb_u_of(base + r * NT, k, ncg)] : 0.0f;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int v = base + r * NT;
        if (v >= n) continue;
        Bout[f * (long long)n + v] = b[r];
        const float sv = ((cf[v >> 6] >> (v & 63)) & 1ull) ? -1.0f : 1.0f;
        const float z = -sv * b[r];
        part += (z > 0.0f ? z + log1pf(expf(-z)) : log1pf(expf(z))) * scale;
      }
    }
    part = train_warp_sum(part);
    if ((tid & 31) == 0) s_part[tid >> 5] = part;
    __syncthreads();
    if (tid == 0) {
      float sum = 0.0f;
      for (int w = 0; w < NT >> 5; w++) sum = __fadd_rn(sum, s_part[w]);
      pf[f * (2LL * T * L + 1) + 2 * T * L] = sum;
    }
    __syncthreads();
  }
}

// Backward of check t from its record: returns its alpha / beta gradient terms.
template <int D, bool PART, bool SLOW>
__device__ __forceinline__ float2 train_backward_row(const int2* sd, int t, float* Gv, float* __restrict__ P,
                                                     bool last, const uint4 rec, float al, float be, uint32_t sync,
                                                     bool corner, float* dbuf, int d) {
  constexpr bool KEEP_U = D <= 14;
  int u[D];
  float gv[D], gc[D];
#pragma unroll
  for (int i = 0; i < D; i++)
    gc[i] = (last || (PART && i >= dvb_min_slots(D) && i >= d)) ? 0.0f : __ldcs(&P[i * kDvbZ]);
  dvb_load<D, PART, SLOW>(sd, t, Gv, d, corner, 0.0f, u, gv);
  const float m1 = __uint_as_float(rec.x), m2 = __uint_as_float(rec.y);
  const int i1 = (int)((rec.z >> 5) & 31u), i2 = (int)(rec.z & 31u);
  const uint32_t par = (uint32_t)__popc(rec.z >> 10) << 31;
  const float u1 = m1 - be, u2 = m2 - be;
  float gA = 0.0f, gB = 0.0f, g1 = 0.0f, g2 = 0.0f;
#pragma unroll
  for (int i = 0; i < D; i++) {
    float c = __fadd_rn(gv[i], gc[i]);
    if (SLOW) c = (corner && i == (PART ? d : D) - 2) ? 0.0f : c;
    const bool first = i == i1;
    const float uu = first ? u2 : u1;
    if (uu > 0.0f) {
      const float gs = __uint_as_float(__float_as_uint(c) ^ slot_sign(rec.z, i) ^ par);
      gA += gs * uu;
      const float gm = gs * al;
      gB -= gm;
      if (first) g2 += gm;
      else g1 += gm;
    }
  }
  const float dx1 = __uint_as_float(__float_as_uint(g1) ^ slot_sign(rec.z, i1));
  const float dx2 = __uint_as_float(__float_as_uint(g2) ^ slot_sign(rec.z, i2));
  const uint32_t rep = sync | (sync << 1);
  int rank = 0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    if (PART && i >= dvb_min_slots(D) && i >= d) continue;
    const float dx = i == i1 ? dx1 : (i == i2 ? dx2 : 0.0f);
    __stcs(&P[i * kDvbZ], -gv[i] - dx);
    if (SLOW && ((rep >> i) & 1u)) {
      dbuf[rank * kDvbZ + t] = dx;
      rank++;
    } else if (dx != 0.0f && !(SLOW && corner && i == (PART ? d : D) - 2)) {
      Gv[KEEP_U ? u[i] : dvb_u(sd[i], t)] = __fadd_rn(gv[i], dx);
    }
  }
  return make_float2(gA, gB);
}

template <int D, bool PART>
__global__ void __launch_bounds__(kTrainThreads, 2) nms_dvb_backward_kernel(
    const DevCode* __restrict__ Cp, int T, int L, const uint64_t* __restrict__ cw, long long frames,
    const float* __restrict__ alpha, const float* __restrict__ beta, const uint4* __restrict__ X,
    const float* __restrict__ Bin, char* __restrict__ work, long long work_stride, float* __restrict__ pf) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_g[2][2][kTrainThreads];  // [row group parity][alpha / beta][check]
  __shared__ DevCode C;
  const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = NT >> 5;
  if (tid == 0) C = *Cp;
  __syncthreads();
  const TrainTab S = train_tables(C, smem);
  const int n = C.n, k = C.k, m = C.m, ncg = C.ncg;
  const uint32_t absent0 = __ldg(&C.sp_absent[0]);
  float* Gv = (float*)(work + (long long)blockIdx.x * work_stride);
  float* P = Gv + ((n + 63) & ~63);
  const float scale = 1.0f / ((float)frames * (float)n);
  const int t = min(tid, kDvbZ - 1);
  const bool act = tid < kDvbZ;
  for (long long f = blockIdx.x; f < frames; f += gridDim.x) {
    const uint64_t* cf = cw + f * (long long)C.words_n;
    for (int base = tid; base < n; base += 4 * NT) {
      float b[4];
#pragma unroll
      for (int r = 0; r < 4; r++) b[r] = base + r * NT < n ? Bin[f * (long long)n + base + r * NT] : 0.0f;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int v = base + r * NT;
        if (v >= n) continue;
        const float sv = ((cf[v >> 6] >> (v & 63)) & 1ull) ? -1.0f : 1.0f;
        const float z = -sv * b[r];
        Gv[dvb_u_of(v, k, ncg)] = scale * (1.0f / (1.0f + expf(-z))) * (-sv);
      }
    }
    __syncthreads();
    float* row = pf + f * (2LL * T * L + 1);
    // Sums of row group g of iteration it, its terms in buffer b (one warp, a
    // fixed order); L == 1: row groups added in descending order.
    auto reduce = [&](int it, int g, int b) {
      float sa = 0.0f, sb = 0.0f;
      for (int c = lane; c < kDvbZ; c += 32) {
        sa = __fadd_rn(sa, s_g[b][0][c]);
        sb = __fadd_rn(sb, s_g[b][1][c]);
      }
      sa = train_warp_sum(sa);
      sb = train_warp_sum(sb);
      if (lane == 0) {
        const int at = it * L + (L == ncg ? g : 0);
        const bool add = L != ncg && g != ncg - 1;
        row[at] = add ? __fadd_rn(row[at], sa) : sa;
        row[T * L + at] = add ? __fadd_rn(row[T * L + at], sb) : sb;
      }
    };
    int done = 0, pit = 0, pg = 0;  // row groups done, the last one
    for (int it = T - 1; it >= 0; it--) {
      const uint4* Xt = X + (f * T + it) * (long long)m;
      for (int g = ncg - 1; g >= 0; g--) {
        const int4 G = S.T.cg[g];
        const uint32_t sync = (uint32_t)G.w;
        const int2* sd = S.T.desc + G.z;
        const int lay = (L == ncg) ? g : 0;
        const float al = __ldg(&alpha[it * L + lay]), be = __ldg(&beta[it * L + lay]);
        const bool slow = sync != 0 || (g == 0 && absent0 != 0);
        if (tid == kTrainThreads - 1) {  // the next row group's records and message gradients
          const bool wrap = g == 0;
          if (!wrap || it > 0) {
            const int gn = wrap ? ncg - 1 : g - 1;
            const int4 Gn = S.T.cg[gn];
            prefetch_l2(Xt + gn * kDvbZ - (wrap ? m : 0), kDvbZ * 16);
            if (wrap || it < T - 1) prefetch_l2(P + Gn.y, (uint32_t)(Gn.x * kDvbZ * 4));
          }
        }
        if (act) {
          const uint4 rec = __ldcs(&Xt[g * kDvbZ + t]);
          float* Pg = P + G.y + t;
          float2 ga;
          if (!slow)
            ga = train_backward_row<D, PART, false>(sd, t, Gv, Pg, it == T - 1, rec, al, be, 0u, false, nullptr, G.x);
          else
            ga = train_backward_row<D, PART, true>(sd, t, Gv, Pg, it == T - 1, rec, al, be, sync,
                                                   g == 0 && t == 0 && absent0 != 0, S.dbuf, G.x);
          s_g[done & 1][0][t] = ga.x;
          s_g[done & 1][1][t] = ga.y;
        }
        if (done > 0 && warp == done % nw) reduce(pit, pg, (done - 1) & 1);
        if (sync) {
          __syncthreads();
          if (act) train_runs(sd, t, Gv, sync, S.dbuf);
        }
        __syncthreads();
        done++;
        pit = it;
        pg = g;
      }
    }
    if (warp == 0) reduce(pit, pg, (done - 1) & 1);
    __syncthreads();
  }
}

template <int D, bool PART>
static int launch_dvb(const DevCode* dcode, const DevCode& h, int T, int L, const float* llr, const uint64_t* cw,
                      long long frames, const float* alpha, const float* beta, float* X, float* B, char* work,
                      long long work_stride, int grid, float* pf, cudaStream_t st) {
  const size_t smem = train_smem(h);
  GF2C_CUDA(allow_smem((const void*)nms_dvb_forward_kernel<D, PART>, smem));
  GF2C_CUDA(allow_smem((const void*)nms_dvb_backward_kernel<D, PART>, smem));
  nms_dvb_forward_kernel<D, PART><<<grid, kTrainThreads, smem, st>>>(dcode, T, L, llr, cw, frames, alpha, beta, (uint4*)X,
                                                                     B, work, work_stride, pf);
  GF2C_CUDA(cudaGetLastError());
  nms_dvb_backward_kernel<D, PART><<<grid, kTrainThreads, smem, st>>>(dcode, T, L, cw, frames, alpha, beta,
                                                                      (const uint4*)X, B, work, work_stride, pf);
  GF2C_CUDA(cudaGetLastError());
  return GF2C_OK;
}

// Forward and backward of the layered schedule on a DVB-T2 code (h.lay_dvb).
int launch_nms_layered_dvb(const DevCode* dcode, const DevCode& h, int T, int L, const float* llr, const uint64_t* cw,
                           long long frames, const float* alpha, const float* beta, float* X, float* B, char* work,
                           long long work_stride, int grid, float* pf, cudaStream_t st) {
#define GF2C_TRAIN(D, PART) \
  return launch_dvb<D, PART>(dcode, h, T, L, llr, cw, frames, alpha, beta, X, B, work, work_stride, grid, pf, st)
  switch (h.lay_dvb) {
    case 7: GF2C_TRAIN(7, true);
    case 9: GF2C_TRAIN(9, false);
    case 10: GF2C_TRAIN(10, false);
    case 11: GF2C_TRAIN(11, false);
    case 13: GF2C_TRAIN(13, true);
    case 14: GF2C_TRAIN(14, false);
    case 18: GF2C_TRAIN(18, false);
    case 19: GF2C_TRAIN(19, true);
    case 22: GF2C_TRAIN(22, false);
  }
#undef GF2C_TRAIN
  return set_error(GF2C_ERR_UNSUPPORTED, "no layered training kernel for this code");
}

}  // namespace gf2c
