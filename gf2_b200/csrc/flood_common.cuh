// gf2cuda flooding decoders, shared device code (sm_100a): teams of CTAs per
// frame and the structured code tables in shared memory.
#pragma once
#include "internal.h"

namespace gf2c {

// A frame may be decoded by a cluster of CTAs (frame state in the workspace,
// shared by the cluster): warps of all its CTAs take the chunks, and the frame's
// barriers are cluster barriers, whose release / acquire makes one CTA's writes
// visible to the others.
struct Team {
  int size, rank;     // CTAs, this CTA
  int warp, nwarps;   // this warp among all warps of the team
  static __device__ __forceinline__ Team make(bool clusters) {
    Team t{1, 0, 0, 0};
    if (clusters) {
      asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(t.size));
      asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(t.rank));
    }
    t.warp = t.rank * ((int)blockDim.x >> 5) + ((int)threadIdx.x >> 5);
    t.nwarps = t.size * ((int)blockDim.x >> 5);
    return t;
  }
  __device__ __forceinline__ void sync() const {
    if (size == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
    }
  }
  // Stores v to the shared variable at p in every CTA of the team.
  __device__ __forceinline__ void put(int* p, int v) const {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    for (int r = 0; r < size; r++)
      asm volatile("{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %0, %1;\n st.shared::cluster.u32 [ra], %2;\n}" ::"r"(a),
                   "r"(r), "r"(v)
                   : "memory");
  }
  // Barrier that returns whether any thread of the team passes p != 0; flag is
  // zero when the first thread arrives (every CTA has its own copy).
  __device__ __forceinline__ int any(int p, int* flag) const {
    if (size == 1) return __syncthreads_or(p);
    if (__any_sync(0xffffffffu, p) && (threadIdx.x & 31) == 0) put(flag, 1);
    sync();
    return *(volatile int*)flag;
  }
};

// Structured tables of the code (DevCode::sp_mode) in shared memory.
struct FastTab {
  const int2* desc;  // slot descriptors {start, wrap}
  const int2* cg;    // per row group {slots, first descriptor}
  const int2* vh;    // per var group {edges, first list entry}
  const int2* vd;    // edge lists
};

// Fills (or, with `load` false, only addresses) the tables at `tab`: desc, cg, vh, vd.
__device__ __forceinline__ FastTab stage_tables(const DevCode& C, int2* tab, bool load) {
  const int nd = C.sp_ndesc, ncg = C.ncg, nvg = C.n / C.vgs, nvd = C.sp_nvd;
  if (load) {
    for (int i = threadIdx.x; i < nd; i += blockDim.x) tab[i] = __ldg(&C.sp_desc[i]);
    for (int i = threadIdx.x; i < ncg; i += blockDim.x)
      tab[nd + i] = make_int2(__ldg(&C.sp_cg[i]).z, __ldg(&C.sp_cg[i]).w);
    for (int i = threadIdx.x; i < nvg; i += blockDim.x) tab[nd + ncg + i] = __ldg(&C.sp_vh[i]);
    for (int i = threadIdx.x; i < nvd; i += blockDim.x) tab[nd + ncg + nvg + i] = __ldg(&C.sp_vd[i]);
  }
  return FastTab{tab, tab + nd, tab + nd + ncg, tab + nd + ncg + nvg};
}

// Posteriors of the D slots of check t of a row group.  `corner` (the
// staircase's first check): the slot before the last holds no edge and reads
// the +inf posterior at index n.
template <int D>
__device__ __forceinline__ void load_check(const int2* sd, int t, int Z, const float* P, bool corner, int n,
                                           float (&ap)[D]) {
#pragma unroll
  for (int i = 0; i < D; i++) {
    const int2 S = sd[i];
    int u = S.x + t - (t >= S.y ? Z : 0);
    if (i == D - 2) u = corner ? n : u;
    ap[i] = P[u];
  }
}
}  // namespace gf2c
