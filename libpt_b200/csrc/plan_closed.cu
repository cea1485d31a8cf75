// Closed-shell triples of the restricted FP64 solves.
//
// In a restricted solve (src/pt.c:469-473) the same-spin blocks are, by
// pt.h's contract, the antisymmetrised mixed-spin ones:
//   t_aa[ij][ab] = t_ij[ab] - t_ij[ba],      t_ij[ab] = t_ji[ba],
//   O_aa[ij][xl] = O_ij[xl] - O_ji[xl],      I_aa[i][d][bc] = I_i[d][bc] - I_i[d][cb]
// (no suffix: abab).  Every contraction of the triples i < j < k of one
// occupied set -- the same-spin one and the mixed-spin (ij;k), (ik;j),
// (jk;i) -- is then a signed sum of six products over ordered p, q, r of the
// set,
//   Z_pqr[x][y,z] = - t_pr[x,d] I_q[d;y,z] - O_pr[x,l] t_q[l;y,z]
// (x, y, z the virtuals at p, q, r), 12 v^4 flops where the four triples'
// own products (plan_cases.cu) take 27 v^4.  Three jobs per group and
// amplitude, one per row index p, sum the two products of p:
//   A1[a][b][c] = Z_ijk[a][b,c] + Z_ikj[a][c,b]
//   A2[b][a][c] = Z_jik[b][a,c] + Z_jki[b][c,a]
//   A3[c][b][a] = Z_kji[c][b,a] + Z_kij[c][a,b]
// the second one through transposed views of the same blocks
// (gemm_dmma.cu), and one epilogue adds the four energies (epi_closed.cu),
// each into its triple's own slot.
//
// A mixed-spin triple with a repeated index, (ij;i) or (ij;j), needs three
// products, 6 v^4 flops (8 v^4 by the general jobs): with f the repeated index
// and s the other, A1 above for (f, s, f), which serves as A3 too, and
//   Z[b][a][c] = Z_sff[b][a,c],  A2[b][a][c] = Z[b][a][c] + Z[b][c][a].
//
// The relations are measured on the device for every solve, on the operands
// themselves, and have to hold exactly: every same-spin element the FP64
// difference of its two mixed-spin ones, t_ij[ab] the same number as t_ji[ba]
// (for the OVVV block: by occupied index).  Then the groups read what the
// caller passed, up to that difference's own rounding, and the energy's error
// stays the general jobs' (1e-16 of the same-spin energy, o = 3, v = 48,
// against 80-bit sums).  A bound on the deviation does not keep it: blocks
// that differ by 2^-43 of the largest element, which integrals transformed
// block by block in FP64 do (5e-14 of it in the reference's own fixtures),
// move that energy by 8.5e-15 (random deviations) to 2.7e-13 (a common
// factor), because the groups read the mixed-spin blocks in place of the
// same-spin ones.  A caller who accepts that names the bound in
// LIBPT_CLOSED_TOL (closed_tol).
//
// Only the one-call solves run groups: plans and shards run any subset of
// the queue and promise the same bits for every split, so a triple's
// arithmetic there must not depend on which others run beside it.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "plan_impl.h"

namespace ptb {

namespace {

// Views of an operand block [P][K][v][v4] as a group job's B: dims
// (4, K, first index, quads of the second, P) with a box of one stage.
int map_grp(CUtensorMap *m, const double *p, int64_t v, int64_t K, int64_t P,
            bool tr) {
  const int64_t v4 = pad4(v);
  const int64_t dims[5] = {4, K, v, v4 / 4, P};
  const int64_t strides[4] = {v * v4 * 8, v4 * 8, 32, K * v * v4 * 8};
  const int box[5] = {4, GEMM_BK, tr ? GRP_BZ : GRP_BY,
                      (tr ? GRP_BY : GRP_BZ) / 4, 1};
  return map_f64(m, p, 5, dims, strides, box);
}

// Index of a queue entry of the first same-spin / mixed-spin case.
int64_t mixed_entry(const libpt_plan *p, int64_t first, int i, int j, int k) {
  const int64_t o = p->oa;
  return first + ((int64_t)i * o - (int64_t)i * (i + 1) / 2 + (j - i - 1)) * o + k;
}

const SpinCase *case_of(const libpt_plan *p, int type) {
  for (const SpinCase &c : p->cases)
    if (c.type == type && c.flip == 0) return &c;
  return nullptr;
}

bool holds(const libpt_plan *p, const unsigned long long *w) {
  double dev, mag;
  std::memcpy(&dev, &w[0], 8);
  std::memcpy(&mag, &w[1], 8);
  return std::isfinite(dev) && std::isfinite(mag) && dev <= p->closed_tol * mag;
}

}  // namespace

// Largest deviation from the relations, as a share of the block's largest
// element, that a solve may run groups with; negative: none does, and its
// energy is a plan's bit for bit.
double closed_tol() {
  const char *t = std::getenv("LIBPT_CLOSED_TOL");
  return t ? std::atof(t) : 0.0;
}

// Whether a solve may run groups at all (its relations aside).
bool closed_possible(const libpt_plan *p) {
  return p->closed_tol >= 0.0 && !p->unrestricted &&
         p->precision == LIBPT_PREC_FP64 &&
         p->va >= CLOSED_MIN_V && p->oa >= 2;
}

// The group case: views, job templates, epilogue tiles.
int closed_build(libpt_plan *p) {
  SpinCase &c = p->closed;
  const int64_t o = p->oa, v = p->va, v4 = pad4(v), ldr = v * v4;
  const int nset = p->ft ? 2 : 1;
  c.type = 2;
  c.oa = c.ob = (int)o;
  c.va = c.vb = (int)v;
  c.bm = dmma_rows(v);
  EpiArgs &e = c.epi;
  std::memset(&e, 0, sizeof(e));
  int64_t stride = 0;
  for (int x = 0; x < 2; ++x)
    for (int q = 0; q < 3; ++q) {
      int64_t *off = x ? e.offR : e.offL;
      off[q] = x < nset ? stride : -1;
      if (x < nset) stride += pad32(v * ldr);
    }
  c.ws_stride = stride;
  for (int x = 0; x < nset; ++x) {
    const OperandSet &S = x ? p->R : p->L;
    const int m = 6 * x;
    int r;
    if ((r = map_a(&c.maps.m[m + 0], S.tau[1], v, v, o, o, c.bm))) return r;
    if ((r = map_a(&c.maps.m[m + 1], S.oovo[1], o, v, o, o, c.bm))) return r;
    for (int t = 0; t < 2; ++t) {
      if ((r = map_grp(&c.maps.m[m + 2 + t], S.ovvv[1], v, v, o, t))) return r;
      if ((r = map_grp(&c.maps.m[m + 4 + t], S.tau[1], v, o, o, t))) return r;
    }
    // rows p; the columns' occupied indices in order (q, r); see above
    const int rows[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
    for (int n = 0; n < 3; ++n) {
      const int P = rows[n][0], Q = rows[n][1], R = rows[n][2];
      JobT j;
      j.off = (x ? e.offR : e.offL)[n];
      j.M = (int)v;
      j.N = (int)v;
      j.ldc = ldr;
      j.nseg = 4;
      // A operands: map_a coordinates (second index, first index)
      j.seg[0] = seg(m + 0, m + 2, true, R, P, Q, v);
      j.seg[1] = seg(m + 1, m + 4, true, R, P, Q, o);
      j.seg[2] = seg(m + 0, m + 3, true, Q, P, R, v);
      j.seg[3] = seg(m + 1, m + 5, true, Q, P, R, o);
      j.seg[2].neg |= GRP_TR;
      j.seg[3].neg |= GRP_TR;
      c.jobs.push_back(j);
    }
  }
  e.ld[0] = ldr;
  e.rowU1 = v4;
  e.oa = e.ob = (int)o;
  e.va = e.vb = (int)v;
  e.d_a = e.d_b = p->d_ov;
  e.ov1_a = e.ov1_b = p->ov1;
  e.ov2_a = e.ov2_b = p->ov2;
  e.g1_ab = p->oovv[1];
  e.g1_ld_ab = v;
  e.g2_ab = p->L.tau[1];
  e.g2_ld_ab = v4;
  std::vector<int4> tiles;
  for (int a = 0; a < v; a += GEPI_T)
    for (int b = 0; b <= a; b += GEPI_T)
      for (int d = 0; d <= b; d += GEPI_T)
        if (std::min<int64_t>(a + GEPI_T, v) - 1 > d)   // not one lone index
          tiles.push_back(make_int4(a, b, d, 0));
  c.ntiles = (int)tiles.size();
  c.ctiles = 1;
  if (dalloc(p, (void **)&c.d_tiles, tiles.size() * sizeof(int4)))
    return LIBPT_ERR_NOMEM;
  DEV(cudaMemcpyAsync(c.d_tiles, tiles.data(), tiles.size() * sizeof(int4),
                      cudaMemcpyHostToDevice, p->st));
  DEV(cudaStreamSynchronize(p->st));
  e.ntiles = c.ntiles;
  e.tiles = c.d_tiles;
  e.ctiles = 1;
  e.has_f = p->has_f ? 1 : 0;
  const SpinCase *aaa = case_of(p, 0), *aab = case_of(p, 1);
  c.flops_per_triple = aaa->flops_per_triple + 3 * aab->flops_per_triple;
  c.count = 1;
  if (dalloc(p, (void **)&c.d_maps, sizeof(MapSet))) return LIBPT_ERR_NOMEM;
  if (dalloc(p, (void **)&c.d_epi, sizeof(EpiArgs))) return LIBPT_ERR_NOMEM;
  DEV(cudaMemcpyAsync(c.d_maps, &c.maps, sizeof(MapSet),
                      cudaMemcpyHostToDevice, p->st));
  DEV(cudaMemcpyAsync(c.d_epi, &c.epi, sizeof(EpiArgs),
                      cudaMemcpyHostToDevice, p->st));
  return LIBPT_OK;
}

// The OVVV relation of occupied indices [i0, i1), on stream s.
int closed_check_ovvv(libpt_plan *p, int i0, int i1, cudaStream_t s) {
  const int64_t v = p->va, v4 = pad4(v), ldp = pad4(npair(v));
  for (int x = 0; x < (p->ft ? 2 : 1); ++x) {
    const OperandSet &S = x ? p->R : p->L;
    DEV(closed_check_launch(S.ovvv[0] + i0 * v * ldp,
                            S.ovvv[1] + i0 * v * v * v4, (i1 - i0) * v, (int)v,
                            ldp, v4, true, 1, false, v,
                            p->closed_words + 16 + 2 * (x * p->oa + i0), s));
  }
  return LIBPT_OK;
}

// Measures the relations of everything but deferred OVVV blocks (words, in
// pairs of deviation and magnitude: 0 i_oovv, 1 + 2x t2 / l2, 2 + 2x OOVO of
// set x, from 8 on OVVV by set and occupied index).
int closed_check(libpt_plan *p) {
  const int64_t o = p->oa, v = p->va, v4 = pad4(v);
  const size_t bytes = (16 + 4 * (size_t)o) * 8;
  if (dalloc(p, (void **)&p->closed_words, bytes)) return LIBPT_ERR_NOMEM;
  DEV(cudaMemsetAsync(p->closed_words, 0, bytes, p->st));
  unsigned long long *w = p->closed_words;
  DEV(closed_check_launch(p->oovv[0], p->oovv[1], o * o, (int)v, v, v, false,
                          (int)o, true, o * o, w, p->st));
  for (int x = 0; x < (p->ft ? 2 : 1); ++x) {
    const OperandSet &S = x ? p->R : p->L;
    DEV(closed_check_launch(S.tau[0], S.tau[1], o * o, (int)v, v4, v4, false,
                            (int)o, true, o * o, w + 2 + 4 * x, p->st));
    DEV(closed_check_oovo_launch(S.oovo[0], S.oovo[1], (int)o, v * pad4(o),
                                 w + 4 + 4 * x, p->st));
  }
  if (p->deferred.empty()) return closed_check_ovvv(p, 0, (int)o, p->st);
  return LIBPT_OK;
}

int closed_read(libpt_plan *p, cudaStream_t s, int upto) {
  const int nset = p->ft ? 2 : 1;
  std::vector<unsigned long long> words(16 + 4 * (size_t)p->oa);
  CK(cudaMemcpyAsync(words.data(), p->closed_words, words.size() * 8,
                     cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const unsigned long long *w = words.data();
  p->closed_on = holds(p, w);
  for (int x = 0; x < nset; ++x)
    p->closed_on = p->closed_on && holds(p, w + 2 + 4 * x) &&
                   holds(p, w + 4 + 4 * x);
  p->closed_ok.assign((size_t)p->oa, 0);
  for (int i = 0; i < upto; ++i) {
    bool ok = true;
    for (int x = 0; x < nset; ++x)
      ok = ok && holds(p, w + 16 + 2 * (x * p->oa + i));
    p->closed_ok[(size_t)i] = ok;
  }
  return LIBPT_OK;
}

// Splits the entries of the whole queue whose largest occupied index lies in
// [lo, hi) into groups and pairs (queue entry, i, j, k; a pair's i == k or j ==
// k) and the rest.
void closed_split(const libpt_plan *p, int lo, int hi,
                  std::vector<int4> &groups, std::vector<int64_t> &rest) {
  const SpinCase *aaa = case_of(p, 0), *aab = case_of(p, 1);
  const int o = p->oa;
  auto grouped = [&](int i, int j, int k) {
    return p->closed_on && p->closed_ok[(size_t)i] &&
           p->closed_ok[(size_t)j] && p->closed_ok[(size_t)k];
  };
  int64_t q = aaa->first;
  for (int i = 0; i < o; ++i)
    for (int j = i + 1; j < o; ++j)
      for (int k = j + 1; k < o; ++k, ++q) {
        if (k < lo || k >= hi) continue;
        if (grouped(i, j, k))
          groups.push_back(make_int4((int)q, i, j, k));
        else
          rest.push_back(q);
      }
  q = aab->first;
  for (int i = 0; i < o; ++i)
    for (int j = i + 1; j < o; ++j)
      for (int k = 0; k < o; ++k, ++q) {
        const int top = std::max(j, k);
        if (top < lo || top >= hi) continue;
        if (!grouped(i, j, k))
          rest.push_back(q);
        else if (k == i || k == j)
          groups.push_back(make_int4((int)q, i, j, k));
      }
}

// Appends groups and pairs to a round while they fit the plan's round
// resources; *taken = those appended.  A group counts as its four triples.
int closed_append(libpt_plan *p, const int4 *groups, size_t n, PlanCursor &cur,
                  Round &r, size_t *taken) {
  *taken = 0;
  SpinCase &c = p->closed;
  const int64_t first = case_of(p, 1)->first;
  const int ft = p->ft ? 1 : 0;
  GemmGroup grp;
  grp.kind = 3;
  grp.bm = c.bm;
  for (size_t t = 0; t < n; ++t) {
    const int q = groups[t].x, k = groups[t].w;
    const bool pair = k == groups[t].y || k == groups[t].z;
    // a pair's occupied indices (f, s, f)
    const bool swapped = k == groups[t].z;
    const int ijk[3] = {pair && swapped ? groups[t].z : groups[t].y,
                        pair && swapped ? groups[t].y : groups[t].z, k};
    const int ne = pair ? 1 : 4;   // queue entries
    if (cur.triples + ne > p->tri_cap || cur.ws + c.ws_stride > p->ws_cap ||
        cur.part + ne * (int64_t)c.ntiles > p->part_cap)
      break;
    double *ws = p->ws + cur.ws, *partials = p->partials + cur.part;
    cur.ws += c.ws_stride;
    cur.part += ne * (int64_t)c.ntiles;
    cur.triples += ne;
    ++*taken;
    std::vector<GemmJob> &jobs = r.gemm[grp];
    const int map0 = r.maps[grp].add(c.d_maps, c.maps.m, MAX_MAPS);
    for (size_t n = 0; n < c.jobs.size(); ++n) {
      // a pair: rows f as they are, rows s without the transposed half, and
      // the third array is the first
      if (pair && n % 3 == 2) continue;
      const JobT &jt = c.jobs[n];
      GemmJob g;
      std::memset(&g, 0, sizeof(g));
      g.out = ws + jt.off;
      g.ldc = jt.ldc;
      g.M = jt.M;
      g.N = jt.N;
      g.maps = c.d_maps;
      g.map0 = map0;
      g.ntiles_n = ((jt.N + GRP_BY - 1) / GRP_BY) *
                   ((jt.N + GRP_BZ - 1) / GRP_BZ);
      g.mtiles = (jt.M + c.bm - 1) / c.bm;
      g.nseg = pair && n % 3 == 1 ? 2 : jt.nseg;
      for (int s = 0; s < g.nseg; ++s) {
        const SegT &st = jt.seg[s];
        GemmSeg &gs = g.seg[s];
        gs.amap = st.amap;
        gs.bmap = st.bmap;
        gs.neg = st.neg;
        gs.klast = (int16_t)dmma_klast(st.k);
        gs.a_q = ijk[st.aq];
        gs.a_p = ijk[st.ap];
        gs.b_p = ijk[st.bp];
        gs.ksteps = st.ksteps;
      }
      jobs.push_back(g);
    }
    EpiItem e;
    std::memset(&e, 0, sizeof(e));
    e.args = c.d_epi;
    e.ws = ws;
    e.partials = partials;
    e.i = ijk[0];
    e.j = ijk[1];
    e.k = ijk[2];
    e.nblk = c.ntiles;
    e.pad_ = swapped ? 1 : 0;
    r.grp[pair][ft].push_back(e);
    if (p->has_f) r.grp_hasf[pair][ft] = true;
    for (int x = 0; x < ne; ++x) {
      // a group's: its same-spin triple, then (ij;k), (ik;j), (jk;i)
      const int64_t slot =
          x == 0   ? q
          : x == 1 ? mixed_entry(p, first, ijk[0], ijk[1], ijk[2])
          : x == 2 ? mixed_entry(p, first, ijk[0], ijk[2], ijk[1])
                   : mixed_entry(p, first, ijk[1], ijk[2], ijk[0]);
      RedItem red;
      red.partials = partials + (int64_t)x * c.ntiles;
      red.dst = p->e_slot + slot;
      red.n = c.ntiles;
      red.pad_ = 0;
      r.red.push_back(red);
    }
    r.gemm_flops += pair ? case_of(p, 1)->flops_per_triple : c.flops_per_triple;
    r.triples += ne;
  }
  return LIBPT_OK;
}

// Runs groups and remaining entries in shared rounds.
int closed_run(libpt_plan *p, const std::vector<int4> &groups,
               const std::vector<int64_t> &rest) {
  if (groups.empty()) return run_entries(p, rest);
  if (int r = ensure_capacity(p, rest, groups.size())) return r;
  Round round;
  size_t g0 = 0, b0 = 0;
  while (g0 < groups.size() || b0 < rest.size()) {
    round.clear();
    PlanCursor cur;
    size_t tg = 0, te = 0;
    if (int r = closed_append(p, groups.data() + g0, groups.size() - g0, cur,
                              round, &tg))
      return r;
    g0 += tg;
    if (g0 == groups.size())
      if (int r = plan_append(p, rest.data() + b0, rest.size() - b0, cur,
                              round, &te))
        return r;
    b0 += te;
    if (tg + te == 0) {
      set_error("a triple does not fit the round resources");
      return LIBPT_ERR_NOMEM;
    }
    if (int r = p->exec.run(round, p->d_err, p->timing ? &p->tm : nullptr,
                            &p->launches))
      return r;
  }
  return LIBPT_OK;
}

// Whether a plan with fixed round resources can hold a group.
bool closed_fits(const libpt_plan *p) {
  return !p->arena || (p->tri_cap >= 4 && p->closed.ws_stride <= p->ws_cap &&
                       4 * (int64_t)p->closed.ntiles <= p->part_cap);
}

int plan_run_solve(libpt_plan *p) {
  const size_t total = p->queue.size();
  if (!p->closed_on || !closed_fits(p)) return plan_run(p, nullptr, total);
  std::vector<int4> groups;
  std::vector<int64_t> rest;
  closed_split(p, 0, p->oa, groups, rest);
  if (ensure_capacity(p, rest, groups.size()) != LIBPT_OK) {
    // a group's outputs may not fit where a triple's do
    cudaGetLastError();
    p->closed_on = false;
    return plan_run(p, nullptr, total);
  }
  return closed_run(p, groups, rest);
}

}  // namespace ptb
