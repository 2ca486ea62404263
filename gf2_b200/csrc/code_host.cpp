// gf2cuda host side: building the parity-check matrix exactly as the reference
// does, and planning its device layout.
//
// Sparse structure (the reference's, so that neighbour orders match):
//   LdpcCode::from_edges -> SpBitMatrixDual::from_coo      ldpc/core.rs:96-104
//   SpBitMatrix::from_coo: rows sorted, odd multiplicity kept  gf2-core/src/sparse.rs:166-203
//   SpBitMatrix::transpose: stable, CSC rows ascending         gf2-core/src/sparse.rs:297-328
//   build_dvb_edges: (x + j q) mod m, staircase p / p-1       ldpc/dvb_t2/builder.rs:74-118
//   QuasiCyclicLdpc::to_edges: row i -> col (i + s) mod Z     ldpc/core.rs:436-447, 578-605
#include <algorithm>
#include <atomic>
#include <cstring>

#include "dvbt2_tables.h"
#include "internal.h"

namespace gf2c {

static void finish_sparse(HostCode& c, std::vector<std::vector<int64_t>>& per_row) {
  c.row_ptr.assign(1, 0);
  c.row_idx.clear();
  for (auto& row : per_row) {
    std::sort(row.begin(), row.end());
    size_t i = 0;
    while (i < row.size()) {
      size_t cnt = 1;
      while (i + cnt < row.size() && row[i + cnt] == row[i]) cnt++;
      if (cnt & 1) c.row_idx.push_back(row[i]);
      i += cnt;
    }
    c.row_ptr.push_back((int64_t)c.row_idx.size());
  }
  std::vector<int64_t> cnt(c.n + 1, 0);
  for (int64_t v : c.row_idx) cnt[v + 1]++;
  c.col_ptr.assign(c.n + 1, 0);
  for (int64_t v = 0; v < c.n; v++) c.col_ptr[v + 1] = c.col_ptr[v] + cnt[v + 1];
  c.col_idx.assign(c.row_idx.size(), 0);
  c.col_edge.assign(c.row_idx.size(), 0);
  std::vector<int64_t> next(c.col_ptr.begin(), c.col_ptr.end() - 1);
  for (int64_t r = 0; r < c.m; r++)
    for (int64_t e = c.row_ptr[r]; e < c.row_ptr[r + 1]; e++) {
      int64_t v = c.row_idx[e];
      c.col_idx[next[v]] = r;
      c.col_edge[next[v]] = e;
      next[v]++;
    }
  c.k = c.n > c.m ? c.n - c.m : 0;
}

uint64_t next_code_serial() {
  static std::atomic<uint64_t> counter{0};
  return ++counter;
}

static uint32_t pack_desc(int type, int base, int shift_or_q) {
  return (uint32_t)base | ((uint32_t)shift_or_q << 20) | ((uint32_t)type << 30);
}

// Edge of (check, var) in CSR, -1 if absent.
static int64_t find_edge(const HostCode& c, int64_t p, int64_t v) {
  auto b = c.row_idx.begin() + c.row_ptr[p], e = c.row_idx.begin() + c.row_ptr[p + 1];
  auto it = std::lower_bound(b, e, v);
  if (it == e || *it != v) return -1;
  return it - c.row_idx.begin();
}

// Builds the VG tables and validates the CG plan against the CSR.  Returns
// false if the plan does not cover every edge exactly once.
static bool finish_plan(HostCode& c) {
  const int64_t E = (int64_t)c.row_idx.size();
  std::vector<int> edge_slot(E, -1);
  int64_t flat = 0;
  for (size_t g = 0; g < c.cg.size(); g++) {
    int4 G = c.cg[g];
    for (int t = 0; t < G.y; t++, flat++) {
      int64_t p = c.cg_checks[flat];
      int real = 0;
      for (int i = 0; i < G.z; i++) {
        int s = G.w + i * G.y + t;
        int v = c.slot_var[s];
        if (v < 0) continue;
        int64_t e = find_edge(c, p, v);
        if (e < 0 || edge_slot[e] >= 0) return false;
        edge_slot[e] = s;
        real++;
      }
      if (real != c.row_ptr[p + 1] - c.row_ptr[p]) return false;
    }
  }
  if (flat != c.m) return false;
  c.chk_cg.assign(c.m, 0);
  flat = 0;
  for (size_t g = 0; g < c.cg.size(); g++)
    for (int t = 0; t < c.cg[g].y; t++) c.chk_cg[flat++] = (uint16_t)g;
  c.max_dc = 0;
  c.max_nchk = 0;
  for (auto& G : c.cg) {
    c.max_dc = std::max(c.max_dc, G.z);
    c.max_nchk = std::max(c.max_nchk, G.y);
  }
  // variable groups
  int nvg = (int)((c.n + c.vgs - 1) / c.vgs);
  c.vg.assign(nvg, int2{0, 0});
  c.vg_slot.clear();
  c.vg_chk.clear();
  c.vg_ci.clear();
  std::vector<int> slot_cc(c.e_slots, -1), slot_i(c.e_slots, -1);
  for (size_t g = 0; g < c.cg.size(); g++) {
    int4 G = c.cg[g];
    for (int i = 0; i < G.z; i++)
      for (int t = 0; t < G.y; t++) {
        slot_cc[(size_t)G.w + (size_t)i * G.y + t] = G.x + t;
        slot_i[(size_t)G.w + (size_t)i * G.y + t] = i;
      }
  }
  c.max_dv = 0;
  for (int h = 0; h < nvg; h++) {
    int dv = 0;
    for (int j = 0; j < c.vgs; j++) {
      int64_t v = (int64_t)h * c.vgs + j;
      if (v >= c.n) break;
      dv = std::max(dv, (int)(c.col_ptr[v + 1] - c.col_ptr[v]));
    }
    c.vg[h] = int2{dv, (int)c.vg_slot.size()};
    size_t base = c.vg_slot.size();
    c.vg_slot.resize(base + (size_t)dv * c.vgs, -1);
    c.vg_chk.resize(base + (size_t)dv * c.vgs, -1);
    c.vg_ci.resize(base + (size_t)dv * c.vgs, -1);
    for (int j = 0; j < c.vgs; j++) {
      int64_t v = (int64_t)h * c.vgs + j;
      if (v >= c.n) break;
      int i = 0;
      for (int64_t s = c.col_ptr[v]; s < c.col_ptr[v + 1]; s++, i++) {
        const int sl = edge_slot[c.col_edge[s]];
        c.vg_slot[base + (size_t)i * c.vgs + j] = sl;
        c.vg_chk[base + (size_t)i * c.vgs + j] = slot_cc[sl];
        c.vg_ci[base + (size_t)i * c.vgs + j] = slot_cc[sl] | (slot_i[sl] << 24);
      }
    }
    c.max_dv = std::max(c.max_dv, dv);
  }
  return true;
}

// Structured variable edge lists of a code whose check slots all fit the
// descriptors (see DevCode::sp_mode); checked entry by entry against the edge
// table, which stays in use when any variable does not match.
static void plan_structured(HostCode& c) {
  c.sp_mode = 0;
  c.sp_vh.clear();
  c.sp_vd.clear();
  c.sp_rot.clear();
  c.sp_ve.clear();
  const int Z = c.z;
  if (c.sp_desc.empty() || Z <= 0 || c.vgs != Z || c.n % Z != 0 || c.m * 16 >= (1ll << 31)) return;
  for (size_t g = 0; g < c.cg.size(); g++) {
    const uint32_t ab = c.sp_absent[g];
    const int d = c.cg[g].z;
    // the one slot without an edge: the staircase corner (first check, last slot but one)
    if (c.cg[g].y != Z || c.cg[g].x != (int)g * Z || (ab && !(g == 0 && d >= 2 && ab == 1u << (d - 2)))) return;
  }
  const int nvg = (int)(c.n / Z);
  struct Circ {
    int g, slot, tau;
  };
  std::vector<std::vector<Circ>> of(nvg);
  for (size_t g = 0; g < c.sp_cg.size(); g++)
    for (int i = 0; i < c.sp_cg[g].z; i++) {
      const int2 D = c.sp_desc[(size_t)c.sp_cg[g].w + i];
      const int base = D.x - (Z - D.y);  // first variable of the circulant's block
      if (base % Z != 0) return;
      of[base / Z].push_back(Circ{(int)g, i, D.y % Z});
    }
  const bool rot = c.kind == 2;
  if (rot) c.sp_rot.assign((size_t)c.n, 0);
  for (int h = 0; h < nvg; h++) {
    auto& L = of[h];
    const int dv = (int)L.size();
    if (rot)
      std::sort(L.begin(), L.end(), [](const Circ& x, const Circ& y) { return x.tau != y.tau ? x.tau < y.tau : x.g < y.g; });
    if (dv > 63) return;
    c.sp_vh.push_back(int2{dv, (int)c.sp_vd.size()});
    if (rot) {
      for (int pass = 0; pass < 2; pass++)
        for (const Circ& e : L) {
          const int t0 = e.tau - (pass == 0 ? Z : 0);
          c.sp_vd.push_back(int2{16 * (e.g * Z + t0), e.slot});
          c.sp_ve.push_back(c.cg[e.g].w + e.slot * Z + t0 - h * Z);
        }
    } else {
      for (const Circ& e : L) c.sp_vd.push_back(int2{16 * (e.g * Z + e.tau), e.slot | (Z - e.tau) << 8});
    }
    for (int j = 0; j < Z; j++) {
      int s = 0, cnt = dv;
      if (rot) {
        s = dv;  // the first circulant that wraps
        for (int i = dv - 1; i >= 0 && j + L[i].tau >= Z; i--) s = i;
        // the staircase corner: its wrapped entry has no edge (it is the first of the list)
        if (s < dv && L[s].g == 0 && c.sp_absent[0] == 1u << L[s].slot && j + L[s].tau == Z) {
          s++;
          cnt--;
        }
        c.sp_rot[(size_t)h * Z + j] = (uint8_t)(s | (cnt < dv ? 128 : 0));
      }
      const int2 V = c.sp_vg[h];
      for (int i = 0; i < V.x; i++) {
        const int want = c.sp_ci[(size_t)V.y + (size_t)i * Z + j];
        int have = -1;
        if (i < cnt) {
          const int2 e = c.sp_vd[(size_t)c.sp_vh[h].y + s + i];
          const int wrap = rot ? Z : e.y >> 8;
          have = (e.x / 16 + j - (j >= wrap ? Z : 0)) | (e.y & 0xff) << 24;
        }
        if (have != want) return;
      }
      if (cnt > V.x) return;
    }
  }
  c.sp_mode = rot ? 1 : 2;
}

// Check-state flooding plan.  DVB-T2 parity bits are stored transposed (u order,
// see DevCode); every other code keeps the natural order.  For codes with slot
// descriptors each (CG, slot) is refitted in u order as base + (t + shift) mod Z
// with an optional missing t = 0 (the staircase corner); if any slot does not
// fit, the plan falls back to the natural order and the slot table.  A slot
// with shift s is stored as {start = base + s, wrap = Z - s}; the variable of a
// missing t = 0 entry is start itself (a valid index, masked by sp_absent).
void plan_state(HostCode& c) {
  const int64_t n = c.n;
  std::vector<int> u_of(n), v_of(n);
  for (int64_t v = 0; v < n; v++) u_of[v] = (int)v;
  if (c.kind == 2) {
    const int64_t k = c.k, q = c.q, Z = c.z;
    for (int64_t p = 0; p < c.m; p++) u_of[k + p] = (int)(k + (p % q) * Z + p / q);
  }
  c.sp_desc.clear();
  c.sp_absent.clear();
  c.sp_cg.clear();
  bool structured = !c.slot_desc.empty() && n < (1 << 30);
  for (size_t g = 0; g < c.cg.size() && structured; g++) {
    const int4 G = c.cg[g];
    const int Z = G.y;
    if (G.z > 32) structured = false;
    uint32_t absent = 0;
    for (int i = 0; i < G.z && structured; i++) {
      std::vector<int> u(Z);
      int base = INT32_MAX, t1 = -1;
      for (int t = 0; t < Z; t++) {
        const int v = c.slot_var[(size_t)G.w + (size_t)i * Z + t];
        u[t] = v < 0 ? -1 : u_of[v];
        if (u[t] >= 0) {
          base = std::min(base, u[t]);
          if (t1 < 0) t1 = t;
        } else if (t > 0) {
          structured = false;
        }
      }
      if (!structured || t1 < 0) {
        structured = false;
        break;
      }
      const int sh = (int)((((int64_t)u[t1] - base - t1) % Z + Z) % Z);
      if ((int64_t)base + Z > n) structured = false;  // every start + t must be a valid index
      for (int t = 0; t < Z && structured; t++)
        if (u[t] >= 0 && u[t] != base + (t + sh) % Z) structured = false;
      c.sp_desc.push_back(int2{base + sh, Z - sh});
      if (u[0] < 0) absent |= 1u << i;
    }
    c.sp_absent.push_back(absent);
  }
  if (!structured) {
    c.sp_desc.clear();
    c.sp_absent.clear();
    for (int64_t v = 0; v < n; v++) u_of[v] = (int)v;
  }
  bool identity = true;
  for (int64_t v = 0; v < n; v++) {
    v_of[u_of[v]] = (int)v;
    identity = identity && u_of[v] == v;
  }
  c.sp_u2v.clear();
  if (!identity) c.sp_u2v = v_of;
  int desc_off = 0;
  c.sp_cchunk.clear();
  for (size_t g = 0; g < c.cg.size(); g++) {
    const int4 G = c.cg[g];
    c.sp_cg.push_back(int4{G.x, G.y, G.z, structured ? desc_off : G.w});
    desc_off += G.z;
    for (int t0 = 0; t0 < G.y; t0 += 32) c.sp_cchunk.push_back(int2{(int)g, t0});
  }
  // u-order var groups of vgs variables; edge lists copied from the natural ones
  const int vgs = c.vgs;
  const int nvg = (int)((n + vgs - 1) / vgs);
  std::vector<int2> vg2(nvg, int2{0, 0});
  c.sp_ci.clear();
  c.sp_vchunk.clear();
  for (int h = 0; h < nvg; h++) {
    int dv = 0;
    for (int j = 0; j < vgs && (int64_t)h * vgs + j < n; j++) {
      const int v = v_of[(size_t)h * vgs + j];
      dv = std::max(dv, (int)(c.col_ptr[v + 1] - c.col_ptr[v]));
    }
    const size_t off = c.sp_ci.size();
    vg2[h] = int2{dv, (int)off};
    c.sp_ci.resize(off + (size_t)dv * vgs, -1);
    for (int j = 0; j < vgs && (int64_t)h * vgs + j < n; j++) {
      const int v = v_of[(size_t)h * vgs + j];
      const int hv = v / vgs, jv = v - hv * vgs;
      const int2 V = c.vg[hv];
      const int deg = (int)(c.col_ptr[v + 1] - c.col_ptr[v]);
      for (int i = 0; i < deg; i++) c.sp_ci[off + (size_t)i * vgs + j] = c.vg_ci[(size_t)V.y + (size_t)i * vgs + jv];
    }
    for (int j0 = 0; j0 < vgs && (int64_t)h * vgs + j0 < n; j0 += 32) c.sp_vchunk.push_back(int2{h, j0});
  }
  c.sp_vg = vg2;
  plan_structured(c);
  if (!c.sp_mode) {
    c.sp_vh.clear();
    c.sp_vd.clear();
    c.sp_rot.clear();
    c.sp_ve.clear();
  }
}

// Generic plan: CGs of up to 256 consecutive checks, slots in CSR order.
static void plan_generic(HostCode& c) {
  c.cg.clear();
  c.cg_sync.clear();
  c.slot_var.clear();
  c.cg_checks.clear();
  const int G = 256;
  int edge0 = 0;
  for (int64_t r0 = 0; r0 < c.m; r0 += G) {
    int nchk = (int)std::min<int64_t>(G, c.m - r0);
    int dc = 0;
    for (int t = 0; t < nchk; t++) dc = std::max(dc, (int)(c.row_ptr[r0 + t + 1] - c.row_ptr[r0 + t]));
    c.cg.push_back(int4{(int)r0, nchk, dc, edge0});
    c.cg_sync.push_back(0);
    c.slot_var.resize((size_t)edge0 + (size_t)dc * nchk, -1);
    for (int t = 0; t < nchk; t++) {
      int64_t r = r0 + t;
      c.cg_checks.push_back(r);
      int i = 0;
      for (int64_t e = c.row_ptr[r]; e < c.row_ptr[r + 1]; e++, i++)
        c.slot_var[(size_t)edge0 + (size_t)i * nchk + t] = (int)c.row_idx[e];
    }
    edge0 += dc * nchk;
  }
  c.e_slots = edge0;
  c.vgs = 256;
  c.layered_ok = 0;
  finish_plan(c);
}

int build_edges(int64_t m, int64_t n, const int64_t* pairs, int64_t count, HostCode& c) {
  if (m < 0 || n < 0 || count < 0 || (count > 0 && !pairs))
    return set_error(GF2C_ERR_INVALID_ARG, "invalid dimensions or pairs");
  if (n > (int64_t)1 << 30 || m > 65535LL * 256 || count > (int64_t)1 << 31)
    return set_error(GF2C_ERR_UNSUPPORTED, "code too large");
  c.m = m;
  c.n = n;
  std::vector<std::vector<int64_t>> per_row(m);
  for (int64_t i = 0; i < count; i++) {
    int64_t r = pairs[2 * i], col = pairs[2 * i + 1];
    if (r < 0 || r >= m || col < 0 || col >= n)
      return set_error(GF2C_ERR_INVALID_ARG, "edge index out of bounds");
    per_row[r].push_back(col);
  }
  finish_sparse(c, per_row);
  c.kind = 0;
  plan_generic(c);
  plan_state(c);
  return GF2C_OK;
}

int build_qc(const int32_t* base, int mb, int nb, int z, HostCode& c) {
  if (!base || mb <= 0 || nb <= 0) return set_error(GF2C_ERR_INVALID_ARG, "base matrix must be non-empty");
  if (z <= 0) return set_error(GF2C_ERR_INVALID_ARG, "expansion factor must be positive");
  if ((int64_t)mb * z > 65535LL * 256 || (int64_t)nb * z > (int64_t)1 << 30)
    return set_error(GF2C_ERR_UNSUPPORTED, "code too large");
  c.m = (int64_t)mb * z;
  c.n = (int64_t)nb * z;
  std::vector<std::vector<int64_t>> per_row(c.m);
  for (int r = 0; r < mb; r++)
    for (int cb = 0; cb < nb; cb++) {
      int s = base[r * nb + cb];
      if (s == -1) continue;
      if (s < 0 || s >= z) return set_error(GF2C_ERR_INVALID_ARG, "shift must be -1 or in [0, Z)");
      for (int i = 0; i < z; i++) per_row[(int64_t)r * z + i].push_back((int64_t)cb * z + (i + s) % z);
    }
  finish_sparse(c, per_row);
  c.kind = 1;
  c.z = z;
  c.mb = mb;
  c.nb = nb;
  c.qc_base.assign(base, base + (size_t)mb * nb);
  // QC plan: one CG per base row, slots in ascending base column.
  c.cg.clear();
  c.cg_sync.clear();
  c.slot_var.clear();
  c.cg_checks.clear();
  int edge0 = 0;
  for (int r = 0; r < mb; r++) {
    std::vector<std::pair<int, int>> circ;
    for (int cb = 0; cb < nb; cb++)
      if (base[r * nb + cb] >= 0) circ.push_back({cb, base[r * nb + cb]});
    int dc = (int)circ.size();
    c.cg.push_back(int4{r * z, z, dc, edge0});
    c.cg_sync.push_back(0);
    for (int i = 0; i < dc; i++) c.slot_desc.push_back(pack_desc(0, circ[i].first * z, circ[i].second));
    c.cg_ninfo.push_back(dc);
    c.slot_var.resize((size_t)edge0 + (size_t)dc * z, -1);
    for (int t = 0; t < z; t++) {
      c.cg_checks.push_back((int64_t)r * z + t);
      for (int i = 0; i < dc; i++)
        c.slot_var[(size_t)edge0 + (size_t)i * z + t] = circ[i].first * z + (t + circ[i].second) % z;
    }
    edge0 += dc * z;
  }
  c.e_slots = edge0;
  c.vgs = z <= 1024 ? z : 256;
  c.layered_ok = (z <= 1023 && c.n < (1 << 20)) ? 1 : 0;
  if (!c.layered_ok) c.slot_desc.clear();
  if (!finish_plan(c)) {
    c.slot_desc.clear();
    plan_generic(c);
  }
  plan_state(c);
  return GF2C_OK;
}

int build_dvbt2(int frame, int rate, HostCode& c) {
  if (frame < 0 || frame > 1 || rate < 0 || rate > 5)
    return set_error(GF2C_ERR_INVALID_ARG, "DVB-T2 frame size must be 0/1 and rate 0..5");
  const gf2_dvbt2_table_t& T = gf2_dvbt2_tables[frame * 6 + rate];
  const int64_t n = T.n, k = T.k, m = n - k, q = T.q, Z = 360;
  c.m = m;
  c.n = n;
  std::vector<std::vector<int64_t>> per_row(m);
  for (auto& row : per_row) row.reserve(24);
  for (int b = 0; b < T.rows; b++)
    for (int a = T.row_ptr[b]; a < T.row_ptr[b + 1]; a++) {
      int64_t x = T.addr[a];
      for (int64_t j = 0; j < Z; j++) {
        per_row[x].push_back(b * Z + j);
        x += q;
        if (x >= m) x -= m;
      }
    }
  for (int64_t p = 0; p < m; p++) {
    per_row[p].push_back(k + p);
    if (p > 0) per_row[p].push_back(k + p - 1);
  }
  finish_sparse(c, per_row);
  c.kind = 2;
  c.z = (int)Z;
  c.q = (int)q;
  // encoder lists: address x of block b lies in row group x mod q and rotates
  // the block's 360 bits by x div q; repeated addresses cancel (XOR)
  {
    std::vector<std::vector<int>> rg(q);
    for (int b = 0; b < T.rows; b++) {
      std::vector<int64_t> xs(T.addr + T.row_ptr[b], T.addr + T.row_ptr[b + 1]);
      std::sort(xs.begin(), xs.end());
      for (size_t i = 0; i < xs.size();) {
        size_t j = i;
        while (j < xs.size() && xs[j] == xs[i]) j++;
        if ((j - i) & 1) rg[xs[i] % q].push_back((b << 16) | (int)(xs[i] / q));
        i = j;
      }
    }
    c.enc_rg_ptr.assign(1, 0);
    c.enc_rg_ent.clear();
    for (const auto& v : rg) {
      c.enc_rg_ent.insert(c.enc_rg_ent.end(), v.begin(), v.end());
      c.enc_rg_ptr.push_back((int)c.enc_rg_ent.size());
    }
  }
  c.dvb_index = frame * 6 + rate;
  // Row group a = checks p = a + q t (t = 0..359).  An address x lies in row
  // group x mod q and, for info block b, links check t to bit b*360 + (t - x div q) mod 360:
  // one 360x360 circulant.  Slots: circulants sorted by (block, shift), then the
  // staircase sub-diagonal (k + p - 1, absent for p = 0) and diagonal (k + p).
  c.cg.clear();
  c.cg_sync.clear();
  c.slot_var.clear();
  c.cg_checks.clear();
  std::vector<std::vector<std::pair<int, int>>> circ(q);
  for (int b = 0; b < T.rows; b++)
    for (int a = T.row_ptr[b]; a < T.row_ptr[b + 1]; a++) {
      int x = T.addr[a];
      circ[x % q].push_back({b, x / (int)q});
    }
  int edge0 = 0;
  for (int a = 0; a < q; a++) {
    auto& cl = circ[a];
    std::sort(cl.begin(), cl.end());
    int ninfo = (int)cl.size();
    int dc = ninfo + 2;
    c.cg.push_back(int4{(int)(a * Z), (int)Z, dc, edge0});
    uint32_t sync = 0;
    for (int i = 0; i + 1 < ninfo; i++)
      if (cl[i].first == cl[i + 1].first) sync |= 1u << i;
    c.cg_sync.push_back(sync);
    for (int i = 0; i < ninfo; i++)
      c.slot_desc.push_back(pack_desc(0, cl[i].first * (int)Z, (int)((Z - cl[i].second) % Z)));
    c.slot_desc.push_back(pack_desc(1, (int)(k + a), (int)q));
    c.slot_desc.push_back(pack_desc(2, (int)(k + a), (int)q));
    c.cg_ninfo.push_back(ninfo);
    c.slot_var.resize((size_t)edge0 + (size_t)dc * Z, -1);
    for (int t = 0; t < Z; t++) {
      int64_t p = a + q * t;
      c.cg_checks.push_back(p);
      for (int i = 0; i < ninfo; i++)
        c.slot_var[(size_t)edge0 + (size_t)i * Z + t] =
            (int)(cl[i].first * Z + ((t - cl[i].second) % Z + Z) % Z);
      c.slot_var[(size_t)edge0 + (size_t)ninfo * Z + t] = p > 0 ? (int)(k + p - 1) : -1;
      c.slot_var[(size_t)edge0 + (size_t)(ninfo + 1) * Z + t] = (int)(k + p);
    }
    edge0 += dc * (int)Z;
  }
  c.e_slots = edge0;
  c.vgs = (int)Z;
  c.layered_ok = 1;
  if (!finish_plan(c)) {
    c.slot_desc.clear();
    plan_generic(c);
  }
  // cross-check the descriptors against the slot table
  for (size_t g = 0; g < c.cg.size() && !c.slot_desc.empty(); g++) {
    const int4 G = c.cg[g];
    for (int i = 0; i < G.z; i++) {
      const uint32_t D = c.slot_desc[G.w / G.y + i];
      const int type = (int)(D >> 30), sh = (int)((D >> 20) & 1023u), base = (int)(D & 0xFFFFFu);
      for (int t = 0; t < G.y; t++) {
        int v;
        if (type == 0) v = base + (t + sh) % G.y;
        else if (type == 1) v = (g == 0 && t == 0) ? -1 : base + sh * t - 1;
        else v = base + sh * t;
        if (v != c.slot_var[(size_t)G.w + (size_t)i * G.y + t])
          return set_error(GF2C_ERR_KERNEL, "internal: DVB-T2 slot descriptor mismatch");
      }
    }
  }
  plan_state(c);
  return GF2C_OK;
}

// Right-to-left pivot search (RuEncodingMatrices::compute_generator_matrix with
// rref(h, pivot_from_right = true), richardson_urbanke.rs:158-243 and
// gf2-core/src/alg/rref.rs:67-130): parity columns = greedy right-most basis of
// the column space, message columns = the rest in ascending order, and
// P[i][j] = reduced H[pivot row of parity column j][message column i].
int prepare_encoder(HostCode& c) {
  if (c.enc_ready) return c.enc_status;
  c.enc_ready = true;
  if (c.kind == 2) {
    c.enc_kind = 0;
    c.enc_status = GF2C_OK;
    return GF2C_OK;
  }
  c.enc_kind = 1;
  const int64_t m = c.m, n = c.n;
  if (m == 0 || n == 0 || m >= n) {
    c.enc_status = set_error(GF2C_ERR_INVALID_ARG, "encoding needs 0 < m < n");
    return c.enc_status;
  }
  const int64_t W = (n + 63) / 64;
  if ((double)m * (double)W * 8.0 > 4e9) {
    c.enc_status = set_error(GF2C_ERR_UNSUPPORTED, "generic encoder: matrix too large");
    return c.enc_status;
  }
  std::vector<uint64_t> rows((size_t)m * W, 0);
  for (int64_t r = 0; r < m; r++)
    for (int64_t e = c.row_ptr[r]; e < c.row_ptr[r + 1]; e++)
      rows[(size_t)r * W + (c.row_idx[e] >> 6)] |= 1ull << (c.row_idx[e] & 63);
  std::vector<char> used(m, 0), is_piv(n, 0);
  std::vector<int64_t> piv_row;
  c.enc_par_cols.clear();
  for (int64_t col = n - 1; col >= 0 && (int64_t)piv_row.size() < m; col--) {
    int64_t pr = -1;
    for (int64_t r = 0; r < m; r++)
      if (!used[r] && ((rows[(size_t)r * W + (col >> 6)] >> (col & 63)) & 1)) {
        pr = r;
        break;
      }
    if (pr < 0) continue;
    used[pr] = 1;
    const uint64_t* src = &rows[(size_t)pr * W];
    for (int64_t r = 0; r < m; r++)
      if (r != pr && ((rows[(size_t)r * W + (col >> 6)] >> (col & 63)) & 1)) {
        uint64_t* dst = &rows[(size_t)r * W];
        for (int64_t w = 0; w < W; w++) dst[w] ^= src[w];
      }
    c.enc_par_cols.push_back((int)col);
    piv_row.push_back(pr);
    is_piv[col] = 1;
  }
  if ((int64_t)piv_row.size() != m) {
    c.enc_status = set_error(GF2C_ERR_RANK, "parity-check matrix is rank deficient");
    return c.enc_status;
  }
  c.enc_msg_cols.clear();
  for (int64_t col = 0; col < n; col++)
    if (!is_piv[col]) c.enc_msg_cols.push_back((int)col);
  const int64_t Wm = (m + 63) / 64;
  c.enc_p.assign((size_t)c.k * Wm, 0);
  for (int64_t i = 0; i < c.k; i++) {
    int64_t col = c.enc_msg_cols[i];
    for (int64_t j = 0; j < m; j++)
      if ((rows[(size_t)piv_row[j] * W + (col >> 6)] >> (col & 63)) & 1)
        c.enc_p[(size_t)i * Wm + (j >> 6)] |= 1ull << (j & 63);
  }
  c.enc_status = GF2C_OK;
  return GF2C_OK;
}

// Tables of one upload, in one device allocation with 256-byte aligned parts (an
// allocation per table, two dozen of them, made most of a code's first call).
struct TableUpload {
  struct Part {
    const void* src;
    size_t bytes;
    const void** out;
  };
  std::vector<Part> parts;
  template <class T>
  void add(const std::vector<T>& v, const T** out) {
    parts.push_back(Part{v.data(), sizeof(T) * v.size(), (const void**)out});
  }
  int run(HostCode& c) {
    auto padded = [](size_t x) { return (x + 255) / 256 * 256; };
    size_t total = 0;
    for (const Part& p : parts) total += padded(p.bytes);
    char* base = nullptr;
    if (total) {
      GF2C_CUDA(cudaMalloc((void**)&base, total));
      c.dev_allocs.push_back(base);
    }
    for (const Part& p : parts) {
      if (p.bytes) GF2C_CUDA(cudaMemcpy(base, p.src, p.bytes, cudaMemcpyHostToDevice));
      *p.out = p.bytes ? base : nullptr;
      base += padded(p.bytes);
    }
    return GF2C_OK;
  }
};

int upload_code(HostCode& c) {
  std::lock_guard<std::mutex> lock(c.dev_mu);
  int dev = 0;
  GF2C_CUDA(cudaGetDevice(&dev));
  bool need_enc = c.enc_ready && c.enc_status == GF2C_OK && c.enc_kind == 1 && !c.dev.enc_p;
  if (c.dev_id == dev && !need_enc) return GF2C_OK;
  if (c.dev_id != dev) {
    if (c.dev_id >= 0) return set_error(GF2C_ERR_UNSUPPORTED, "code already bound to another device");
    DevCode d{};
    d.n = (int)c.n;
    d.m = (int)c.m;
    d.k = (int)c.k;
    d.ncg = (int)c.cg.size();
    d.nvg = (int)c.vg.size();
    d.vgs = c.vgs;
    d.e_slots = c.e_slots;
    d.max_dc = c.max_dc;
    d.max_dv = c.max_dv;
    d.words_k = (int)((c.k + 63) / 64);
    d.words_n = (int)((c.n + 63) / 64);
    d.words_m = (int)((c.m + 63) / 64);
    d.layered_ok = c.layered_ok;
    d.lay_bucket = layered_dcmax_bucket(c.max_dc);
    d.max_nchk = c.max_nchk;
    d.lay_dvb = layered_dvb_bucket(c);
    for (uint32_t x : c.cg_sync) d.lay_runs = std::max(d.lay_runs, __builtin_popcount(x | x << 1));
    TableUpload up;
    up.add(c.cg, &d.cg);
    up.add(c.cg_sync, &d.cg_sync);
    up.add(c.slot_var, &d.slot_var);
    up.add(c.chk_cg, &d.chk_cg);
    up.add(c.vg, &d.vg);
    up.add(c.vg_slot, &d.vg_slot);
    up.add(c.vg_chk, &d.vg_chk);
    up.add(c.vg_ci, &d.vg_ci);
    up.add(c.slot_desc, &d.slot_desc);
    if (!c.slot_desc.empty()) up.add(c.cg_ninfo, &d.cg_ninfo);
    d.z = c.slot_desc.empty() ? 0 : c.z;
    up.add(c.sp_cg, &d.sp_cg);
    up.add(c.sp_desc, &d.sp_desc);
    up.add(c.sp_absent, &d.sp_absent);
    up.add(c.sp_cchunk, &d.sp_cchunk);
    up.add(c.sp_vg, &d.sp_vg);
    up.add(c.sp_ci, &d.sp_ci);
    up.add(c.sp_vchunk, &d.sp_vchunk);
    up.add(c.sp_u2v, &d.sp_u2v);
    d.sp_ncchunk = (int)c.sp_cchunk.size();
    d.sp_nvchunk = (int)c.sp_vchunk.size();
    d.sp_mode = c.sp_mode;
    d.sp_nvd = (int)c.sp_vd.size();
    d.sp_ndesc = (int)c.sp_desc.size();
    up.add(c.sp_vh, &d.sp_vh);
    up.add(c.sp_vd, &d.sp_vd);
    up.add(c.sp_rot, &d.sp_rot);
    up.add(c.sp_ve, &d.sp_ve);
    std::vector<int> rp(c.row_ptr.begin(), c.row_ptr.end()), ri(c.row_idx.begin(), c.row_idx.end());
    up.add(rp, &d.csr_ptr);
    up.add(ri, &d.csr_idx);
    d.enc_kind = c.kind == 2 ? 0 : 1;
    if (c.kind == 2) {
      d.enc_q = c.q;
      d.enc_rg_total = (int)c.enc_rg_ent.size();
      up.add(c.enc_rg_ptr, &d.enc_rg_ptr);
      up.add(c.enc_rg_ent, &d.enc_rg_ent);
    }
    int rc = up.run(c);
    if (rc) return rc;
    c.dev = d;
    c.dev_id = dev;
  }
  if (need_enc) {
    TableUpload up;
    up.add(c.enc_p, &c.dev.enc_p);
    up.add(c.enc_msg_cols, &c.dev.enc_msg_cols);
    up.add(c.enc_par_cols, &c.dev.enc_par_cols);
    if (int rc = up.run(c)) return rc;
  }
  return GF2C_OK;
}

HostCode::~HostCode() {
  for (void* p : dev_allocs) cudaFree(p);
}

}  // namespace gf2c
