// gf2cuda flooding sum-product decoder of the DVB-T2 codes (sm_100a).
//
// The schedule and arithmetic of bp_decode_kernel (decode.cu): one message per
// edge, v2c = belief - c2v formed in the check node, 2 atanh of the extrinsic
// tanh products by prefix / suffix products (exact) or the SFU form, belief =
// llr + sum of c2v in ascending original check index, the syndrome of iteration
// t evaluated in the check pass of t + 1 -- the same results bit for bit.  The
// passes are those of the check-state kernel (state_flood.cu): row groups and
// variable groups in chunks of 32, descriptors in shared memory, u order,
// rotated edge lists (here offsets of messages), teams of CTAs per frame.
//
// Bound by issue slots (the exact check node is about a hundred separately
// rounded operations per edge), so its divisions are own code (spa_math.cuh).
#include <cuda_fp16.h>

#include <algorithm>

#include "flood_common.cuh"
#include "numeric.cuh"
#include "spa_math.cuh"

namespace gf2c {

static constexpr int kSpaThreads = 512;

__device__ __forceinline__ float sf_ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sf_lg2(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Check-node update of one check with D slots: posteriors ap, messages at
// msg[i * kZ]; writes the new messages and returns a word whose bit 31 is the
// parity of the hard decisions.  The corner's missing slot (posterior +inf) is
// neutral: tanh 1, e = 0.
constexpr int kZ = 360;
template <bool FAST, int MSG16, int D>
__device__ __forceinline__ uint32_t spa_check(const float (&ap)[D], bool first, typename MsgIO<MSG16>::T* msg) {
  typedef MsgIO<MSG16> IO;
  uint32_t hp = 0;
  float x[D];
#pragma unroll
  for (int i = 0; i < D; i++) x[i] = first ? 0.0f : IO::ld(msg, i * kZ);
#pragma unroll
  for (int i = 0; i < D; i++) {
    hp ^= __float_as_uint(ap[i]);
    x[i] = __fsub_rn(ap[i], x[i]);  // v2c
  }
  if constexpr (FAST) {
    uint32_t neg = 0;
    float N = 1.0f, Dp = 1.0f, e[D];
#pragma unroll
    for (int i = 0; i < D; i++) {
      neg ^= __float_as_uint(x[i]);
      e[i] = sf_ex2(fabsf(x[i]) * -1.4426950408889634f);
      N *= fmaxf(1.0f - e[i], 5.9604645e-08f);
      Dp = __fmaf_rn(Dp, e[i], Dp);
    }
#pragma unroll
    for (int i = 0; i < D; i++) {
      const float ni = fmaxf(1.0f - e[i], 5.9604645e-08f), di = 1.0f + e[i];
      const float num = __fmaf_rn(Dp, ni, N * di);
      const float den = fmaxf(__fmaf_rn(Dp, ni, -N * di), num * 5.9604645e-08f);
      const float mag = fminf(0.69314718055994531f * sf_lg2(num * sf_rcp(den)), 16.635532f);
      IO::st(msg, i * kZ, __uint_as_float(__float_as_uint(mag) ^ ((neg ^ __float_as_uint(x[i])) & 0x80000000u)));
    }
  } else {
    // tanh products; the sign of a product is the XOR of its factors' signs
    float suf[D];
#pragma unroll
    for (int i = 0; i < D; i++)
      x[i] = __uint_as_float(__float_as_uint(tanh_half_abs(fabsf(x[i]))) | (__float_as_uint(x[i]) & 0x80000000u));
    suf[D - 1] = 1.0f;
#pragma unroll
    for (int i = D - 2; i >= 0; i--) suf[i] = __fmul_rn(x[i + 1], suf[i + 1]);
    float pre = 1.0f;
#pragma unroll
    for (int i = 0; i < D; i++) {
      const float p = __fmul_rn(pre, suf[i]);
      const float mag = fabsf(p);
      const float out = two_atanh_abs(mag > GF2C_SPA_PMAX ? GF2C_SPA_PMAX : mag);  // a NaN stays one
      IO::st(msg, i * kZ, __uint_as_float(__float_as_uint(out) | (__float_as_uint(p) & 0x80000000u)));
      pre = (i == 0) ? x[0] : __fmul_rn(pre, x[i]);
    }
  }
  return hp;
}

template <bool FAST, int MSG16, int DCMAX>
__device__ __forceinline__ int spa_check_pass(const Team team, const DevCode& C, const FastTab T, const float* P,
                                              typename MsgIO<MSG16>::T* c2v, bool first) {
  const int lane = threadIdx.x & 31, ncc = C.sp_ncchunk, n = C.n;
  const bool has_corner = __ldg(&C.sp_absent[0]) != 0u;
  uint32_t par = 0;
  for (int ch = team.warp; ch < ncc; ch += team.nwarps) {
    const int g = ch / 12, t = (ch - 12 * g) * 32 + lane;
    if (t >= kZ) continue;
    const int2 G = T.cg[g];
    const bool corner = g == 0 && t == 0 && has_corner;
    typename MsgIO<MSG16>::T* msg = c2v + (long long)G.y * kZ + t;  // a row group's messages: slots x checks
    switch (DCMAX - G.x) {
#define GF2C_SPA_CASE(R)                                                        \
  case R:                                                                       \
    if constexpr (DCMAX - R >= 4 && (R == 0 || DCMAX == 7 || DCMAX == 13 || DCMAX == 19)) { \
      float ap[DCMAX - R];                                                      \
      load_check<DCMAX - R>(T.desc + G.y, t, kZ, P, corner, n, ap);             \
      par |= spa_check<FAST, MSG16, DCMAX - R>(ap, first, msg);                 \
    }                                                                           \
    break;
      GF2C_SPA_CASE(0)
      GF2C_SPA_CASE(1)
      GF2C_SPA_CASE(2)
      GF2C_SPA_CASE(3)
      GF2C_SPA_CASE(4)
#undef GF2C_SPA_CASE
    }
  }
  return (int)(par >> 31);
}

// belief = llr + sum of c2v, two chunks of variables at a time.
template <int MSG16>
__device__ __forceinline__ void spa_var_pass(const Team team, const DevCode& C, const FastTab T, const int* ve,
                                             const typename MsgIO<MSG16>::T* c2v, float* P, const float* lu) {
  typedef MsgIO<MSG16> IO;
  const int lane = threadIdx.x & 31, nvc = C.sp_nvchunk;
  const uint8_t* __restrict__ rot = C.sp_rot;
  for (int ch = team.warp; ch < nvc; ch += 2 * team.nwarps) {
    int u[2], dv[2];
    const int* L[2];
    float b[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int c = min(ch + r * team.nwarps, nvc - 1), h = c / 12, j = (c - 12 * h) * 32 + lane;
      const bool on = j < kZ && ch + r * team.nwarps < nvc;
      u[r] = h * kZ + min(j, kZ - 1);
      const int2 V = T.vh[h];
      const int rr = __ldg(&rot[u[r]]);
      L[r] = ve + V.y + (rr & 127);
      dv[r] = on ? V.x - (rr >> 7) : -1;
      b[r] = __ldcs(&lu[u[r]]);
    }
    const int dm = max(dv[0], dv[1]);
    for (int i = 0; i < dm; i += 4) {
      float m[2][4];
#pragma unroll
      for (int r = 0; r < 2; r++)
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (i + q < dv[r]) m[r][q] = IO::ld(c2v, L[r][i + q] + u[r]);
#pragma unroll
      for (int r = 0; r < 2; r++)
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (i + q < dv[r]) b[r] = __fadd_rn(b[r], m[r][q]);
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
      if (dv[r] >= 0) P[u[r]] = b[r];
  }
}

// Parity of the hard decisions over all checks (this thread's part).
__device__ __forceinline__ int spa_syndrome(const Team team, const DevCode& C, const FastTab T, const float* P) {
  const int lane = threadIdx.x & 31, ncc = C.sp_ncchunk;
  const bool has_corner = __ldg(&C.sp_absent[0]) != 0u;
  uint32_t par = 0;
  for (int ch = team.warp; ch < ncc; ch += team.nwarps) {
    const int g = ch / 12, t = (ch - 12 * g) * 32 + lane;
    if (t >= kZ) continue;
    const int2 G = T.cg[g];
    uint32_t p = 0;
    for (int i = 0; i < G.x; i++) {
      const int2 S = T.desc[G.y + i];
      if (g == 0 && t == 0 && has_corner && i == G.x - 2) continue;
      p ^= __float_as_uint(P[S.x + t - (t >= S.y ? kZ : 0)]);
    }
    par |= p;
  }
  return (int)(par >> 31);
}

// Up to 11 slots two CTAs fit an SM at 64 registers; more slots need more.
template <bool FAST, int MSG16, int DCMAX>
__global__ void __launch_bounds__(kSpaThreads, DCMAX <= 11 ? 2 : 1) bp_spa_flood_kernel(const DecodeArgs a) {
  typedef typename MsgIO<MSG16>::T MsgT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_frame[2];
  __shared__ int s_vote[3];
  __shared__ DevCode C;
  const Team team = Team::make(true);
  const int tid = team.rank * (int)blockDim.x + (int)threadIdx.x, NT = team.size * (int)blockDim.x;
  const int lane = threadIdx.x & 31, ltid = threadIdx.x;
  char* work = a.work + (long long)(blockIdx.x / (unsigned)team.size) * a.work_stride;
  float* llr_u = (float*)(work + a.sf_llr_off);
  MsgT* c2v = (MsgT*)(work + a.sf_st_off);
  float* P = (float*)(work + a.sf_app_off);
  int tab_code = -1;
  if (team.size > 1) team.sync();  // every CTA of the team runs before the first remote store
  for (;;) {
    if (tid == 0) {
      const long long q = (long long)atomicAdd(a.queue, 1ull);
      const long long nq = a.frames_dev ? *a.frames_dev : a.frames;  // queue entries
      const long long f = (q < nq) ? (a.order != nullptr ? a.order[q] : q) : -1;
      team.put(&s_frame[0], (int)(f & 0xffffffffll));
      team.put(&s_frame[1], (int)(f >> 32));
    }
    if (ltid < 3) s_vote[ltid] = 0;
    team.sync();
    const long long f = (long long)s_frame[1] << 32 | (unsigned)s_frame[0];
    if (f < 0 || f >= a.frames) break;
    const int cid = a.code_id ? a.code_id[f] : 0;
    if (cid < 0 || cid >= a.ncodes) {
      if (tid == 0) {
        atomicExch(a.status, 1);
        if (a.iters) a.iters[f] = -1;
      }
      team.sync();
      continue;
    }
    if (ltid == 0) C = a.codes[cid];
    __syncthreads();
    const int n = C.n, k = C.k, q = C.ncg;
    const float* __restrict__ llr = a.llr + (a.llr_off ? a.llr_off[f] : f * (long long)n);
    const int maxit = a.max_iter_arr ? a.max_iter_arr[f] : a.max_iter;
    uint64_t* mo = a.msg ? a.msg + (a.msg_off ? a.msg_off[f] : f * (long long)C.words_k) : nullptr;
    float* bo = a.beliefs ? a.beliefs + (a.llr_off ? a.llr_off[f] : f * (long long)n) : nullptr;
    if (maxit <= 0) {  // a fresh reference decoder: all-zero beliefs, valid word
      if (mo)
        for (int w = tid; w < C.words_k; w += NT) mo[w] = 0ull;
      if (bo)
        for (int v = tid; v < n; v += NT) bo[v] = 0.0f;
      if (tid == 0) {
        if (a.iters) a.iters[f] = 0;
        if (a.conv) a.conv[f] = 0;
        if (a.synd_ok) a.synd_ok[f] = 1;
      }
      team.sync();
      continue;
    }
    // natural index of u-order variable u
    auto nat = [&](int u) {
      const int p = u - k, row = p / kZ;
      return u < k ? u : k + row + q * (p - row * kZ);
    };
    for (int base = tid; base < n; base += 4 * NT) {
      float x[4];
#pragma unroll
      for (int r = 0; r < 4; r++) x[r] = base + r * NT < n ? llr[nat(base + r * NT)] + 0.0f : 0.0f;
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (base + r * NT < n) {
          llr_u[base + r * NT] = x[r];
          P[base + r * NT] = x[r];
        }
    }
    if (tid == 0) P[n] = __int_as_float(0x7f800000);
    const FastTab T = stage_tables(C, (int2*)smem_raw, tab_code != cid);
    int* ve = (int*)(T.vd + C.sp_nvd);
    if (tab_code != cid)
      for (int i = ltid; i < C.sp_nvd; i += blockDim.x) ve[i] = __ldg(&C.sp_ve[i]);
    tab_code = cid;
    team.sync();

    int it = 0, converged = 0, synd = 1;
    for (;;) {
      int par = spa_check_pass<FAST, MSG16, DCMAX>(team, C, T, P, c2v, it == 0);
      par = team.any(par, &s_vote[it & 1]);
      if (ltid == 0) s_vote[(it + 1) & 1] = 0;  // used after the next barrier
      if (it > 0 && a.early_stop && !par) {
        converged = 1;
        synd = 0;
        break;
      }
      spa_var_pass<MSG16>(team, C, T, ve, c2v, P, llr_u);
      team.sync();
      ++it;
      if (it >= maxit) break;
    }
    if (!converged) {
      synd = team.any(spa_syndrome(team, C, T, P), &s_vote[2]);
      converged = !synd;
    }
    if (mo) {  // message bits: the first k variables (identical in u order)
      uint32_t* mo32 = (uint32_t*)mo;
      const int wk = C.words_k;
      for (int base = 0; base < 64 * wk; base += NT) {
        const int u = base + tid;
        const unsigned bits = __ballot_sync(0xffffffffu, u < k && P[u < n ? u : 0] < 0.0f);
        if (lane == 0 && u < 64 * wk) mo32[u >> 5] = bits;
      }
    }
    if (bo)
      for (int u = tid; u < n; u += NT) bo[nat(u)] = P[u];
    if (tid == 0) {
      if (a.iters) a.iters[f] = it;
      if (a.conv) a.conv[f] = (uint8_t)converged;
      if (a.synd_ok) a.synd_ok[f] = (uint8_t)(!synd);
    }
    team.sync();
  }
}

int spa_flood_threads() { return kSpaThreads; }

// Workspace of a team and shared memory for the tables of the largest code.
StateFloodLayout spa_flood_layout(const std::vector<const HostCode*>& codes, int msg_bytes) {
  size_t n = 0, e = 0, tab = 0;
  for (const HostCode* h : codes) {
    n = std::max(n, (size_t)h->n);
    e = std::max(e, (size_t)h->e_slots);
    tab = std::max(tab, 8 * (h->sp_desc.size() + h->cg.size() + h->sp_vh.size() + h->sp_vd.size()) + 4 * h->sp_vd.size());
  }
  auto al = [](size_t x) { return (long long)((x + 255) / 256 * 256); };
  StateFloodLayout L{};
  L.smem = tab;
  L.llr_off = 0;
  L.st_off = al(n * 4);
  L.app_off = L.st_off + al(e * msg_bytes);
  L.work_stride = L.app_off + al(n * 4 + 16);
  return L;
}

template <bool FAST, int MSG16>
static const void* spa_kernel(int D) {
  switch (D) {
    case 7: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 7>;
    case 9: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 9>;
    case 10: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 10>;
    case 11: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 11>;
    case 13: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 13>;
    case 14: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 14>;
    case 18: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 18>;
    case 19: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 19>;
    case 22: return (const void*)bp_spa_flood_kernel<FAST, MSG16, 22>;
  }
  return nullptr;
}
const void* spa_flood_kernel_ptr(int algo, int msg16, int D) {
  if (algo == GF2C_ALGO_SPA) return msg16 ? spa_kernel<false, 1>(D) : spa_kernel<false, 0>(D);
  if (algo == GF2C_ALGO_SPA_FAST) return msg16 ? spa_kernel<true, 1>(D) : spa_kernel<true, 0>(D);
  return nullptr;
}

}  // namespace gf2c
