// gf2cuda flooding min-sum decoder on compressed check states (sm_100a).
//
// For min-sum every message leaving a check is determined by four numbers: the
// smallest and second-smallest |v2c| (min1, min2), the slot of min1 and the
// final sign of each slot's message (the parity of the other inputs' signs):
//     c2v_i = sign_i * (i == argmin ? min2 : min1)
// (Llr::boxplus_minsum_n, crates/gf2-coding/src/llr.rs:246-284, over the other
// edges of the check).  A 16-byte state {min1, min2, sign bits, argmin} per
// check therefore reproduces every message bit for bit while moving 16 B per
// check instead of 4 B per edge, and the check-node pass writes nothing per
// edge.
//
// Schedule and arithmetic are the reference's flooding loop
// (ldpc/core.rs:889-938): v2c = belief - c2v (formed in the check node, the
// same IEEE subtraction), belief = llr + sum of c2v in ascending original check
// index, the syndrome of the hard decisions of iteration t evaluated in the
// check-node pass of iteration t + 1.  Normalised / offset min-sum transforms
// the two magnitudes; FP16 message storage rounds them to binary16 (the
// rounding is odd-symmetric, so the messages equal those of a decoder that
// stores each message in binary16).
//
// Sign conventions.  The sign bits of a state are kept with slot i at bit
// 31 - i, so that a shift by the slot brings its sign to bit 31.  The frame's
// LLRs enter as llr + 0.0f, which turns -0 into +0 and any NaN into the
// positive canonical one; every later v2c is the result of an addition, so a
// v2c is never -0 or a negative NaN and its sign bit is the comparison x < 0.
//
// Work decomposition.  One CTA of 1024 threads (fewer where several frames fit
// on an SM) decodes one frame at a time (persistent, frames from an atomic queue).  Each warp takes chunks of 32
// consecutive checks of one row group (check pass) or 32 consecutive
// variables of one variable group (variable pass), so the degree, the slot
// descriptors and the loop trip counts are warp-uniform.  The posteriors are
// kept in "u order" (DVB-T2 parity bit k + a + q t at k + a Z + t), in which
// every slot of every row group reads a contiguous, rotated run of Z
// posteriors and every variable group reads contiguous check states.
//
// Batches that leave SMs idle, or would in their last wave: a cluster of 2 to 16
// CTAs takes a frame (struct Team), with the frame state in the workspace.  Which
// size, if any, is estimated per batch (team_of in capi.cu).
//
// Placement.  The check states (m x 16 B) and the posteriors (n x 4 B) live in
// shared memory when they fit together (DVB-T2 short frames, ALL_SMEM);
// otherwise both live in the CTA's global workspace slice, which the L1 and the
// 126 MB L2 cache for the frames in flight.  The u-order copy of the channel
// LLRs (read once per iteration) is in the workspace.
#include <cuda_fp16.h>

#include <algorithm>

#include "flood_common.cuh"
#include "numeric.cuh"

namespace gf2c {

static constexpr int kStateThreads = 1024;

// c2v of slot i from a check state {min1, min2, sign bits, argmin}
__device__ __forceinline__ float state_c2v(const uint4 s, int i) {
  const uint32_t mag = (i == (int)s.w) ? s.y : s.x;
  return __uint_as_float(mag | ((s.z << i) & 0x80000000u));
}

__device__ __forceinline__ float round_mag16(float v) {
  return __half2float(__float2half_rn(v > 65504.0f ? 65504.0f : v));
}

// Posteriors in u order (shared memory or the CTA workspace).
template <bool ALL_SMEM>
struct Post {
  float* p;
  __device__ __forceinline__ float* at(int u) const { return p + u; }
  __device__ __forceinline__ float* run(int) const { return p; }
};

struct SlotTables {
  const int2* desc;      // DevCode::sp_desc
  const uint32_t* absent;
  const int* slot_var;
};

// Posteriors of the slots of check t of row group g (slot i in ap[i]); returns
// the mask of the slots that hold an edge.  Every address is valid, so the
// loads are issued unconditionally, back to back.
template <int DCMAX, bool ALL_SMEM>
__device__ __forceinline__ uint32_t load_slots(const SlotTables T, int g, const int4 G, int t, uint32_t dmask,
                                               const Post<ALL_SMEM> P, float (&ap)[DCMAX]) {
  if (T.desc) {
    const int2* __restrict__ sd = T.desc + G.w;
#pragma unroll
    for (int i = 0; i < DCMAX; i++) {
      if (i < G.z) {
        const int2 D = __ldg(&sd[i]);
        ap[i] = P.run(D.x)[D.x + t - (t >= D.y ? G.y : 0)];
      }
    }
    return t == 0 ? dmask & ~__ldg(&T.absent[g]) : dmask;
  }
  const int* __restrict__ sv = T.slot_var + G.w + t;
  uint32_t real = 0;
#pragma unroll
  for (int i = 0; i < DCMAX; i++) {
    if (i < G.z) {
      const int u = __ldg(&sv[i * G.y]);
      real |= (uint32_t)(u >= 0) << i;
      ap[i] = *P.at(u < 0 ? 0 : u);
    }
  }
  return real;
}

// Check-node update from the slot posteriors ap[] and the old state `so`:
// writes the new state and returns the parity of the hard decisions of the
// posteriors.  ALLREAL: every slot below d holds an edge; FIRST: the old
// messages are all zero.
template <int DCMAX, bool FIRST, bool ALLREAL>
__device__ __forceinline__ int check_node(const float (&ap)[DCMAX], uint32_t real, int d, const uint4 so,
                                          uint4* st_cc, bool nms, float al, float be, bool msg16) {
  float m1 = __int_as_float(0x7f800000), m2 = m1;
  uint32_t i1 = 0xffu, neg = 0u;
  int hp = 0;
#pragma unroll
  for (int i = 0; i < DCMAX; i++) {
    if (i < d && (ALLREAL || ((real >> i) & 1u))) {
      hp ^= (int)(ap[i] < 0.0f);
      const float x = FIRST ? ap[i] : __fsub_rn(ap[i], state_c2v(so, i));
      const float ax = fabsf(x);
      const bool lt1 = ax < m1, lt2 = ax < m2;
      m2 = lt1 ? m1 : (lt2 ? ax : m2);
      m1 = lt1 ? ax : m1;
      i1 = lt1 ? (uint32_t)i : i1;
      neg |= (uint32_t)(x < 0.0f) << (31 - i);
    }
  }
  const bool single = ALLREAL ? d == 1 : __popc(real) == 1;
  float mag1 = single ? 0.0f : m1, mag2 = single ? 0.0f : m2;
  if (nms) {  // normalised / offset min-sum
    const float d1 = __fsub_rn(mag1, be), d2 = __fsub_rn(mag2, be);
    mag1 = __fmul_rn(al, d1 > 0.0f ? d1 : 0.0f);
    mag2 = __fmul_rn(al, d2 > 0.0f ? d2 : 0.0f);
  }
  if (msg16) {
    mag1 = round_mag16(mag1);
    mag2 = round_mag16(mag2);
  }
  const uint32_t sgn = (__popc(neg) & 1) ? ~neg : neg;
  *st_cc = make_uint4(__float_as_uint(mag1), __float_as_uint(mag2), sgn, i1);
  return hp;
}

// ---------------------------------------------------------------------------
// Structured passes (QC / DVB-T2 codes, DevCode::sp_mode): the slot and edge
// descriptors live in shared memory, every lane of a warp reads the same ones,
// and no index table is read per edge.
//
// Bound by instruction issue with the frame state on chip (short 1/2: issue
// slots 71 % busy) and by the latency of the gathers with it in the workspace
// (normal 3/5: 49 %, long scoreboard 7.5 stalls per issue), so the instructions
// per edge and the loads in flight count.  Against per-edge index tables and
// sign masks built from comparisons: 165 -> 111 K warp instructions per short
// 1/2 iteration and 704 -> 470 K per normal 3/5 iteration; 256 short 1/2
// frames 3.14 -> 1.92 ms, 1000 normal 3/5 frames 51.2 -> 31.7 ms (of that
// 37.5 -> 31.7 ms by loading the next variables' LLRs ahead, taking two
// degree-3 variables at a time and reading the LLRs evict-first).
// ---------------------------------------------------------------------------
// Check-node update of check t of a row group whose D slots all hold an edge.
// `corner` (the staircase's first check): the slot before the last holds none
// and reads the +inf posterior at index n, which leaves minima and signs as
// they are.  Returns a word whose bit 31 is the parity of the hard decisions.
template <int D>
__device__ __forceinline__ uint32_t update_check(const float (&ap)[D], const uint4 so, uint4* st_cc, bool nms, float al,
                                                 float be, bool msg16) {
  float m1 = __int_as_float(0x7f800000), m2 = m1;
  uint32_t i1 = 0xffu, neg = 0u, hp = 0u;
#pragma unroll
  for (int i = 0; i < D; i++) {
    hp ^= __float_as_uint(ap[i]);
    const float x = __fsub_rn(ap[i], state_c2v(so, i));
    const float ax = fabsf(x);
    i1 = ax < m1 ? (uint32_t)i : i1;
    m2 = fmaxf(m1, fminf(m2, ax));
    m1 = fminf(m1, ax);
    neg = __funnelshift_l(__float_as_uint(x), neg, 1);  // slot i at bit D - 1 - i
  }
  float mag1 = m1, mag2 = m2;
  if (nms) {
    const float d1 = __fsub_rn(mag1, be), d2 = __fsub_rn(mag2, be);
    mag1 = __fmul_rn(al, d1 > 0.0f ? d1 : 0.0f);
    mag2 = __fmul_rn(al, d2 > 0.0f ? d2 : 0.0f);
  }
  if (msg16) {
    mag1 = round_mag16(mag1);
    mag2 = round_mag16(mag2);
  }
  const uint32_t sgn = ((__popc(neg) & 1) ? ~neg : neg) << (32 - D);
  *st_cc = make_uint4(__float_as_uint(mag1), __float_as_uint(mag2), sgn, i1);
  return hp;
}
template <int D>
__device__ __forceinline__ uint32_t fast_check(const int2* sd, int t, int Z, const float* P, bool corner, int n,
                                               const uint4 so, uint4* st_cc, bool nms, float al, float be,
                                               bool msg16) {
  float ap[D];
  load_check<D>(sd, t, Z, P, corner, n, ap);
  return update_check<D>(ap, so, st_cc, nms, al, be, msg16);
}

// The code descriptor of the frame a CTA is decoding (shared by the passes).
__shared__ DevCode sf_code;

// Check-node pass: every check reads its slot posteriors and its old state and
// writes its new state.  Returns this thread's part of the parity of the hard
// decisions over all checks (the syndrome of the previous iteration).  NMS
// weights of this iteration start at alpha / beta + nms_row, one per row group
// when per_layer, else one for the whole code.
template <int DCMAX, bool ALL_SMEM>
__device__ __forceinline__ int sf_check_pass(const Team team, uint4* st, const Post<ALL_SMEM> P, bool first, bool nms, bool msg16,
                                             const float* alpha, const float* beta, int nms_row, bool per_layer) {
  const DevCode& C = sf_code;
  const int lane = threadIdx.x & 31, nwarps = team.nwarps;
  const SlotTables T{C.sp_desc, C.sp_absent, C.slot_var};
  const int2* __restrict__ cch = C.sp_cchunk;
  const int4* __restrict__ spcg = C.sp_cg;
  const int ncc = C.sp_ncchunk;
  int par = 0;
  for (int ch = team.warp; ch < ncc; ch += nwarps) {
    const int2 CH = cch[ch];
    const int4 G = spcg[CH.x];
    const int t = CH.y + lane;
    if (t >= G.y) continue;
    const int cc = G.x + t;
    const uint32_t dmask = G.z >= 32 ? 0xffffffffu : (1u << G.z) - 1u;
    float ap[DCMAX];
    const uint32_t real = load_slots<DCMAX, ALL_SMEM>(T, CH.x, G, t, dmask, P, ap);
    float al = 1.0f, be = 0.0f;
    if (nms) {
      const int idx = nms_row + (per_layer ? CH.x : 0);
      al = __ldg(&alpha[idx]);
      be = __ldg(&beta[idx]);
    }
    if (real == dmask) {
      if (first)
        par |= check_node<DCMAX, true, true>(ap, real, G.z, make_uint4(0u, 0u, 0u, 0xffu), st + cc, nms, al, be,
                                             msg16);
      else
        par |= check_node<DCMAX, false, true>(ap, real, G.z, st[cc], st + cc, nms, al, be, msg16);
    } else {
      const uint4 so = first ? make_uint4(0u, 0u, 0u, 0xffu) : st[cc];
      par |= check_node<DCMAX, false, false>(ap, real, G.z, so, st + cc, nms, al, be, msg16);
    }
  }
  return par;
}

// Check-node pass over the structured tables; chunks of 32 checks of one row
// group, so the slot count is warp-uniform.  Row groups up to three slots
// short of DCMAX (the irregular short codes) have their own unrolled body.
template <int DCMAX>
__device__ __forceinline__ int sf_check_fast(const Team team, const FastTab T, uint4* st, const float* P, bool first, bool nms,
                                             bool msg16, const float* alpha, const float* beta, int nms_row,
                                             bool per_layer) {
  const DevCode& C = sf_code;
  const int lane = threadIdx.x & 31, nwarps = team.nwarps;
  const int Z = C.vgs, n = C.n, ncc = C.sp_ncchunk, cpg = (Z + 31) >> 5;
  const uint32_t magic = 0xffffffffu / (uint32_t)cpg + 1u;  // ch / cpg as a multiply (cpg > 1)
  const bool has_corner = __ldg(&C.sp_absent[0]) != 0u;
  uint32_t par = 0;
  for (int ch = team.warp; ch < ncc; ch += nwarps) {
    const int g = cpg > 1 ? (int)__umulhi((uint32_t)ch, magic) : ch;
    const int t = (ch - g * cpg) * 32 + lane;
    if (t >= Z) continue;
    const int2 G = T.cg[g];
    const int cc = g * Z + t;
    const int2* sd = T.desc + G.y;
    const bool corner = cc == 0 && has_corner;
    float al = 1.0f, be = 0.0f;
    if (nms) {
      const int idx = nms_row + (per_layer ? g : 0);
      al = __ldg(&alpha[idx]);
      be = __ldg(&beta[idx]);
    }
    const uint4 so = first ? make_uint4(0u, 0u, 0u, 0xffu) : st[cc];
    switch (DCMAX - G.x) {
#define GF2C_SF_CASE(R)                                                                                       \
  case R:                                                                                                     \
    if constexpr (DCMAX - R >= 2) par |= fast_check<DCMAX - R>(sd, t, Z, P, corner, n, so, st + cc, nms, al, be, msg16); \
    break;
      GF2C_SF_CASE(0)
      GF2C_SF_CASE(1)
      GF2C_SF_CASE(2)
      GF2C_SF_CASE(3)
#undef GF2C_SF_CASE
      default: {
        float ap[DCMAX];
#pragma unroll
        for (int i = 0; i < DCMAX; i++)
          if (i < G.x) {
            const int2 S = sd[i];
            ap[i] = P[S.x + t - (t >= S.y ? Z : 0)];
          }
        uint32_t real = (1u << G.x) - 1u;
        if (corner) real &= ~(1u << (G.x - 2));
        par |= (uint32_t)check_node<DCMAX, false, false>(ap, real, G.x, so, st + cc, nms, al, be, msg16) << 31;
      }
    }
  }
  return (int)(par >> 31);
}

// State of list entry e for variable j of its group.
template <bool WRAP>
__device__ __forceinline__ uint4 state_at(const int2 e, int j, int Z, const uint4* st) {
  int off = e.x + 16 * j;
  if (WRAP) off -= j >= (e.y >> 8) ? 16 * Z : 0;
  return *(const uint4*)((const char*)st + off);
}

// N edges of one variable: the states are gathered together, then added in
// list order.  WRAP: the list entries carry their wrap position.
template <int N, bool WRAP>
__device__ __forceinline__ float add_edges(float b, const int2* L, int j, int Z, const uint4* st) {
  int2 e[N];
  uint4 s[N];
#pragma unroll
  for (int q = 0; q < N; q++) e[q] = L[q];
#pragma unroll
  for (int q = 0; q < N; q++) s[q] = state_at<WRAP>(e[q], j, Z, st);
#pragma unroll
  for (int q = 0; q < N; q++) b = __fadd_rn(b, state_c2v(s[q], WRAP ? e[q].y & 0xff : e[q].y));
  return b;
}

// Variable-node pass over the structured edge lists.
template <bool WRAP>
__device__ __forceinline__ void sf_var_fast(const Team team, const FastTab T, const uint4* st, float* P, const float* lu) {
  const DevCode& C = sf_code;
  const int lane = threadIdx.x & 31, nwarps = team.nwarps;
  const int Z = C.vgs, nvc = C.sp_nvchunk, cpg = (Z + 31) >> 5;
  const uint32_t magic = 0xffffffffu / (uint32_t)cpg + 1u;
  const uint8_t* __restrict__ rot = C.sp_rot;
  auto var_of = [&](int ch, int& h, int& j) {
    h = cpg > 1 ? (int)__umulhi((uint32_t)ch, magic) : ch;
    j = (ch - h * cpg) * 32 + lane;
    return h * Z + min(j, Z - 1);
  };
  // Two chunks at a time, so that the gathers of two degree-3 variables (most
  // of a DVB-T2 code) are in flight together; LLRs and list starts of the next
  // pair are loaded meanwhile.
  struct Var {
    int h, j, u, r;
    float l;
  };
  auto fetch = [&](int ch) {
    Var v{0, Z, 0, 0, 0.0f};
    if (ch < nvc) {
      v.u = var_of(ch, v.h, v.j);
      v.l = __ldcs(&lu[v.u]);
      if (!WRAP) v.r = __ldg(&rot[v.u]);
    }
    return v;
  };
  auto one = [&](const Var& v) {
    if (v.j >= Z) return;
    const int2 V = T.vh[v.h];
    float b = v.l + 0.0f;
    const int2* L = T.vd + V.y + (v.r & 127);
    int dv = V.x - (v.r >> 7);
    for (; dv >= 4; dv -= 4, L += 4) b = add_edges<4, WRAP>(b, L, v.j, Z, st);
    if (dv == 3) b = add_edges<3, WRAP>(b, L, v.j, Z, st);
    else if (dv == 2) b = add_edges<2, WRAP>(b, L, v.j, Z, st);
    else if (dv == 1) b = add_edges<1, WRAP>(b, L, v.j, Z, st);
    P[v.u] = b;
  };
  int ch = team.warp;
  Var v0 = fetch(ch), v1 = fetch(ch + nwarps);
  for (; ch < nvc; ch += 2 * nwarps) {
    const Var n0 = fetch(ch + 2 * nwarps), n1 = fetch(ch + 3 * nwarps);
    const int2 V0 = T.vh[v0.h], V1 = T.vh[v1.h];
    if (V0.x == 3 && V1.x == 3 && ch + nwarps < nvc) {
      const int2* L0 = T.vd + V0.y + (v0.r & 127);
      const int2* L1 = T.vd + V1.y + (v1.r & 127);
      const int j0 = min(v0.j, Z - 1), j1 = min(v1.j, Z - 1);
      int2 e[6];
      uint4 s[6];
#pragma unroll
      for (int q = 0; q < 3; q++) {
        e[q] = L0[q];
        e[3 + q] = L1[q];
      }
#pragma unroll
      for (int q = 0; q < 6; q++) s[q] = state_at<WRAP>(e[q], q < 3 ? j0 : j1, Z, st);
      float b0 = v0.l + 0.0f, b1 = v1.l + 0.0f;
#pragma unroll
      for (int q = 0; q < 3; q++) {
        b0 = __fadd_rn(b0, state_c2v(s[q], WRAP ? e[q].y & 0xff : e[q].y));
        b1 = __fadd_rn(b1, state_c2v(s[3 + q], WRAP ? e[3 + q].y & 0xff : e[3 + q].y));
      }
      if (v0.j < Z) P[v0.u] = b0;
      if (v1.j < Z) P[v1.u] = b1;
    } else {
      one(v0);
      one(v1);
    }
    v0 = n0;
    v1 = n1;
  }
}

// Variable-node pass: belief = llr + sum of c2v in ascending original check index.
template <bool ALL_SMEM>
__device__ __forceinline__ void sf_var_pass(const Team team, const uint4* st, const Post<ALL_SMEM> P, const float* lu) {
  const DevCode& C = sf_code;
  const int lane = threadIdx.x & 31, nwarps = team.nwarps;
  const int nvc = C.sp_nvchunk, vgs = C.vgs, n = C.n;
  const int2* __restrict__ vch = C.sp_vchunk;
  const int2* __restrict__ svg = C.sp_vg;
  const int* __restrict__ sci = C.sp_ci;
  for (int ch = team.warp; ch < nvc; ch += nwarps) {
    const int2 CH = vch[ch];
    const int2 V = svg[CH.x];
    const int j = CH.y + lane;
    const int u = CH.x * vgs + j;
    if (j >= vgs || u >= n) continue;
    float b = lu[u] + 0.0f;
    const int* __restrict__ ci = sci + V.y + j;
    // batches of 4 edges, the last one partial: the edge-table loads of a
    // batch, then its state gathers, are in flight together (two dependent
    // round trips per batch, whatever the degree)
    for (int i = 0; i < V.x; i += 4) {
      int e[4];
      uint4 s[4];
#pragma unroll
      for (int q = 0; q < 4; q++) e[q] = i + q < V.x ? __ldg(&ci[(i + q) * vgs]) : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) s[q] = st[e[q] < 0 ? 0 : (e[q] & 0xffffff)];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (e[q] >= 0) b = __fadd_rn(b, state_c2v(s[q], e[q] >> 24));
    }
    *P.at(u) = b;
  }
}

// Parity of the hard decisions over all checks (this thread's part).
template <int DCMAX, bool ALL_SMEM>
__device__ __forceinline__ int sf_syndrome_pass(const Team team, const Post<ALL_SMEM> P) {
  const DevCode& C = sf_code;
  const int lane = threadIdx.x & 31, nwarps = team.nwarps;
  const SlotTables T{C.sp_desc, C.sp_absent, C.slot_var};
  int p = 0;
  for (int ch = team.warp; ch < C.sp_ncchunk; ch += nwarps) {
    const int2 CH = C.sp_cchunk[ch];
    const int4 G = C.sp_cg[CH.x];
    const int t = CH.y + lane;
    if (t >= G.y) continue;
    float ap[DCMAX];
    const uint32_t real =
        load_slots<DCMAX, ALL_SMEM>(T, CH.x, G, t, G.z >= 32 ? 0xffffffffu : (1u << G.z) - 1u, P, ap);
#pragma unroll
    for (int i = 0; i < DCMAX; i++)
      if (i < G.z && ((real >> i) & 1u)) p ^= (int)(ap[i] < 0.0f);
  }
  return p;
}

// PASSES: StateFloodLayout::passes; TEAM: clusters of CTAs.  A kernel of its own
// for each, since a CTA of 1024 threads has 64 registers per thread, and passes
// that do not run or a team of one cost spills: 2000 frames of QC codes with the
// state in the workspace, Z = 1024 without structured tables 10.6 -> 10.3 ms, 46 x
// 68 blocks of Z = 384 9.79 -> 7.92 ms; 148 normal 1/2 frames 1.89 -> 1.68 ms.
template <int DCMAX, bool ALL_SMEM, int PASSES, bool TEAM>
__global__ void __launch_bounds__(kStateThreads, 1) bp_state_flood_kernel(const DecodeArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_frame[2];  // the frame (low, high word)
  __shared__ int s_vote[3];   // team votes: alternating iterations, final syndrome
  const DevCode& C = sf_code;
  const Team team = Team::make(TEAM);
  // thread index and count of the team
  const int tid = team.rank * (int)blockDim.x + (int)threadIdx.x, NT = team.size * (int)blockDim.x;
  const int lane = threadIdx.x & 31, ltid = threadIdx.x, LT = blockDim.x;
  char* work = a.work + (long long)(blockIdx.x / (unsigned)team.size) * a.work_stride;
  uint4* st = ALL_SMEM ? (uint4*)smem_raw : (uint4*)(work + a.sf_st_off);
  const Post<ALL_SMEM> P{ALL_SMEM ? (float*)(smem_raw + a.sf_app_soff) : (float*)(work + a.sf_app_off)};
  int tab_code = -1;  // code whose tables are in shared memory
  if (team.size > 1) team.sync();  // every CTA of the team runs before the first remote store
  for (;;) {
    if (tid == 0) {
      const long long q = (long long)atomicAdd(a.queue, 1ull);
      const long long nq = a.frames_dev ? *a.frames_dev : a.frames;  // queue entries
      const long long f = (q < nq) ? (a.order != nullptr ? a.order[q] : q) : -1;
      if (TEAM) {
        team.put(&s_frame[0], (int)(f & 0xffffffffll));
        team.put(&s_frame[1], (int)(f >> 32));
      } else {
        s_frame[0] = (int)(f & 0xffffffffll);
        s_frame[1] = (int)(f >> 32);
      }
    }
    if (TEAM && ltid < 3) s_vote[ltid] = 0;
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
    if (ltid == 0) sf_code = a.codes[cid];
    __syncthreads();
    const int n = C.n;
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
    const int* __restrict__ u2v = C.sp_u2v;
    float* llr_u = (float*)(work + a.sf_llr_off);
    for (int base = tid; base < n; base += 4 * NT) {  // four loads in flight per thread
      float x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int u = base + q * NT;
        x[q] = u < n ? llr[u2v ? __ldg(&u2v[u]) : u] + 0.0f : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int u = base + q * NT;
        if (u < n) {
          if (u2v) llr_u[u] = x[q];
          *P.at(u) = x[q];
        }
      }
    }
    const bool fast = PASSES == kStructured || (PASSES == kBothPasses && a.sf_tab_off >= 0 && C.sp_mode != 0);
    FastTab T{};
    if (fast) {
      T = stage_tables(C, (int2*)(smem_raw + a.sf_tab_off), tab_code != cid);
      tab_code = cid;
      if (tid == 0) P.p[n] = __int_as_float(0x7f800000);  // what the staircase corner reads
    }
    const float* lu = u2v ? llr_u : llr;
    team.sync();

    const bool nms = a.nms_iters > 0;
    int it = 0, converged = 0, synd = 1;
    for (;;) {
      const int nms_row = nms ? min(it, a.nms_iters - 1) * a.nms_L : 0;
      int par = PASSES != kTables && fast
                    ? sf_check_fast<DCMAX>(team, T, st, P.p, it == 0, nms, a.sf_msg16 != 0, a.alpha, a.beta, nms_row,
                                           a.nms_L == C.ncg)
                    : sf_check_pass<DCMAX, ALL_SMEM>(team, st, P, it == 0, nms, a.sf_msg16 != 0, a.alpha, a.beta, nms_row,
                                                     a.nms_L == C.ncg);
      par = team.any(par, &s_vote[it & 1]);
      if (TEAM && ltid == 0) s_vote[(it + 1) & 1] = 0;  // used after the next barrier
      if (it > 0 && a.early_stop && !par) {
        converged = 1;
        synd = 0;
        break;
      }
      if (PASSES == kTables || !fast) sf_var_pass<ALL_SMEM>(team, st, P, lu);
      else if (C.sp_mode == 1) sf_var_fast<false>(team, T, st, P.p, lu);
      else sf_var_fast<true>(team, T, st, P.p, lu);
      team.sync();
      ++it;
      if (it >= maxit) break;
    }
    if (!converged) {
      synd = team.any(sf_syndrome_pass<DCMAX, ALL_SMEM>(team, P), &s_vote[2]);
      converged = !synd;
    }
    if (mo) {  // message bits: the first k variables (identical in u order)
      uint32_t* mo32 = (uint32_t*)mo;
      const int k = C.k, wk = C.words_k;
      for (int base = 0; base < 64 * wk; base += NT) {
        const int u = base + tid;
        const unsigned bits = __ballot_sync(0xffffffffu, u < k && *P.at(u < n ? u : 0) < 0.0f);
        if (lane == 0 && u < 64 * wk) mo32[u >> 5] = bits;
      }
    }
    if (bo)
      for (int u = tid; u < n; u += NT) bo[u2v ? __ldg(&u2v[u]) : u] = *P.at(u);
    if (tid == 0) {
      if (a.iters) a.iters[f] = it;
      if (a.conv) a.conv[f] = (uint8_t)converged;
      if (a.synd_ok) a.synd_ok[f] = (uint8_t)(!synd);
    }
    team.sync();
  }
}

int state_flood_threads() { return kStateThreads; }

int state_dcmax_bucket(int max_dc) {
  static const int buckets[] = {7, 9, 10, 11, 13, 14, 18, 19, 22, 26, 32};
  for (int b : buckets)
    if (max_dc <= b) return b;
  return -1;
}

template <bool ALL_SMEM, int PASSES, bool TEAM>
static const void* state_kernel(int dcmax) {
  switch (dcmax) {
    case 7: return (const void*)bp_state_flood_kernel<7, ALL_SMEM, PASSES, TEAM>;
    case 9: return (const void*)bp_state_flood_kernel<9, ALL_SMEM, PASSES, TEAM>;
    case 10: return (const void*)bp_state_flood_kernel<10, ALL_SMEM, PASSES, TEAM>;
    case 11: return (const void*)bp_state_flood_kernel<11, ALL_SMEM, PASSES, TEAM>;
    case 13: return (const void*)bp_state_flood_kernel<13, ALL_SMEM, PASSES, TEAM>;
    case 14: return (const void*)bp_state_flood_kernel<14, ALL_SMEM, PASSES, TEAM>;
    case 18: return (const void*)bp_state_flood_kernel<18, ALL_SMEM, PASSES, TEAM>;
    case 19: return (const void*)bp_state_flood_kernel<19, ALL_SMEM, PASSES, TEAM>;
    case 22: return (const void*)bp_state_flood_kernel<22, ALL_SMEM, PASSES, TEAM>;
    case 26: return (const void*)bp_state_flood_kernel<26, ALL_SMEM, PASSES, TEAM>;
    case 32: return (const void*)bp_state_flood_kernel<32, ALL_SMEM, PASSES, TEAM>;
  }
  return nullptr;
}

StateFloodLayout state_flood_layout(const std::vector<const HostCode*>& codes, bool on_chip) {
  size_t max_m = 0, max_n = 0, tab = 0;
  bool any_perm = false, any_fast = false, all_fast = true;
  for (const HostCode* h : codes) {
    max_m = std::max(max_m, (size_t)h->m);
    max_n = std::max(max_n, (size_t)h->n);
    any_perm = any_perm || !h->sp_u2v.empty();
    all_fast = all_fast && h->sp_mode != 0;
    if (h->sp_mode) {
      any_fast = true;
      tab = std::max(tab, 8 * (h->sp_desc.size() + h->cg.size() + h->sp_vh.size() + h->sp_vd.size()));
    }
  }
  // Either the whole frame state is on chip, or all of it is in the workspace:
  // keeping only part of it in shared memory (measured on normal 3/5 frames)
  // shrinks L1, which caches the workspace, by more than it saves in L2 traffic.
  // The tables go beside it up to the most a CTA may have (1 KB left for the
  // static part), and up to 48 KB, so that most of L1 stays a cache.
  const size_t st_bytes = max_m * 16;
  StateFloodLayout L{};
  L.all_smem = on_chip && st_bytes + max_n * 4 <= 224 * 1024;
  size_t app_bytes = (max_n * 4 + 4 + 15) / 16 * 16;  // one more posterior: the corner's
  const size_t state = L.all_smem ? st_bytes + app_bytes : 0;
  const bool fits = any_fast && tab <= 48 * 1024 && state + tab <= 226 * 1024;
  if (!fits) app_bytes = max_n * 4;
  L.app_soff = (int)st_bytes;
  L.tab_off = fits ? (int)state : -1;
  // (In the workspace the kernel with both kinds of passes serves the structured
  // ones alone too: 148 normal 3/5 frames 1.82 ms, 2.08 ms without the others.)
  L.passes = !fits ? kTables : all_fast && L.all_smem ? kStructured : kBothPasses;
  L.smem = fits ? state + tab : (L.all_smem ? st_bytes + max_n * 4 : 0);
  auto al = [](size_t x) { return (long long)((x + 255) / 256 * 256); };
  long long off = 0;
  L.llr_off = off;
  off += any_perm ? al(app_bytes) : 0;
  L.st_off = off;
  off += L.all_smem ? 0 : al(st_bytes);
  L.app_off = off;
  off += L.all_smem ? 0 : al(app_bytes);
  L.work_stride = off;
  return L;
}

const void* state_flood_kernel_ptr(int dcmax, const StateFloodLayout& L, bool team) {
  if (team)
    return L.passes == kTables ? state_kernel<false, kTables, true>(dcmax) : state_kernel<false, kBothPasses, true>(dcmax);
  if (!L.all_smem)
    return L.passes == kTables ? state_kernel<false, kTables, false>(dcmax)
                               : state_kernel<false, kBothPasses, false>(dcmax);
  return L.passes == kTables       ? state_kernel<true, kTables, false>(dcmax)
         : L.passes == kStructured ? state_kernel<true, kStructured, false>(dcmax)
                                   : state_kernel<true, kBothPasses, false>(dcmax);
}

}  // namespace gf2c
