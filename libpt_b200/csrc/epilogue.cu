// Energy epilogues: assemble W(abc) from a triple's contraction outputs,
// add the disconnected term and the denominator, and reduce the triple's
// energy (src/pt.c:291-295, 433-445 for (T); 697-700, 916-927 for (fT)).
//
// Same-spin triples (i<j<k):  one output T[x][pair] per amplitude, and
//   W[a>b>c] = T[a][bc] - T[b][ac] + T[c][ab]                (pair = p(p-1)/2+q)
// Mixed-spin triples (i<j alpha, k beta): outputs U1[x][y][c], U2[x][c][y],
// P[c][pair] per amplitude, and
//   W[a>b,c] = U1[a][b][c] + U2[a][c][b] - U1[b][a][c] - U2[b][c][a]
//              + P[c][ab].
// Energy per element: (W - X) * R / D with R = W for (T) and R = the right
// amplitude for (fT); X is the disconnected term, D the denominator.
//
// A CTA handles an 8 (a) x 8 (b) x 32 (c) tile of one triple; warp w takes
// a = a0 + w, lane l takes c = c0 + l, and a thread the tile's 8 values of b.
// U1 and T rows are read along c (coalesced).  The operands that are
// contiguous in b or a (T[c][ab], U2, P) are needed as runs of 8 doubles per
// (a, c) or (b, c):
//   (T)   copied to shared memory with cp.async, which holds no registers, so
//         all of a tile's loads are in flight together: mixed-spin runs by 8
//         lanes each into [row][x][c] with rows of EPI_CS doubles (copies and
//         reads free of bank conflicts), same-spin runs 16 bytes a copy, as
//         the five aligned pairs that cover pair(a, b0) .. + 7;
//   (fT)  twice the operands: that staging leaves one mixed-spin CTA an SM.
//         Runs are read 32 bytes a load into the thread that needs them, and
//         only U2[b][c][a], which belongs to the eight warps, is staged.
// Measured (v = 180): mixed-spin (fT) 2.9 -> 2.0 ms with the direct loads;
// (T) with them 1.04 ms against 0.95 ms staged (24 triples of v = 201), and
// 16-byte copies of the mixed-spin runs 1.15 ms (they spread a copy over more
// rows and double the bank cycles of the reads).
// Each CTA tile writes one partial sum; reduce_partials adds them in a fixed
// order.  Launches are persistent: a fixed grid strides over the flat tiles
// of a device-memory item list (EpiList), whose items (triples) may belong
// to different plans; each item points at its spin case's fixed arguments,
// which a CTA copies to shared memory.
#include "common.cuh"
#include "engine.h"

namespace ptb {

namespace {

// CTAs per SM the energy kernels are compiled for.  (T): three, of 80
// registers; the kernels are latency-bound, and three CTAs of 256 threads keep
// more loads in flight than two (31 -> 40 % of DRAM peak measured), four
// spill.  (fT): two, of 128 registers, which hold a thread's operand runs
// (v = 180: 2.02 ms with two, 2.20 ms with three and spills).
constexpr int epi_minb(bool ft) { return ft ? 2 : 3; }

// Shared-memory layout (doubles) of the mixed-spin epilogue's staged
// disconnected-term slices, after its U2 staging: g1[j,k][b][c],
// g1[i,k][b][c] (EPI_B x EPI_C each), g1[j,i][b][a] (EPI_B x EPI_A), t1[i][b],
// t1[j][b], d[j][b] (EPI_B each), then the same for the f_ov half.
constexpr int EPI_SD_G1JK = 0, EPI_SD_G1IK = 256, EPI_SD_G1JI = 512,
              EPI_SD_T1I = 576, EPI_SD_T1J = 584, EPI_SD_DJ = 592,
              EPI_SD_G2JK = 600, EPI_SD_G2IK = 856, EPI_SD_G2JI = 1112,
              EPI_SD_F1I = 1176, EPI_SD_F1J = 1184, EPI_SD_SIZE = 1192;
// The same-spin epilogue's: g1 of (j,k), (i,k), (j,i) as [b][c], then as
// [b][a], t1[i,j,k][b] and d[j][b]; the f_ov half follows.
constexpr int EPI_SA_BC = 0, EPI_SA_BA = 768, EPI_SA_T1 = 960,
              EPI_SA_DJ = 984, EPI_SA_F = 992, EPI_SA_SIZE = 2 * EPI_SA_F;
static_assert(EPI_THREADS == EPI_B * EPI_C && EPI_B * EPI_C == 256 &&
                  EPI_A * EPI_B == 64 && EPI_A == 8 && EPI_B == 8,
              "one staged (b, c) per thread; offsets above");

__device__ __forceinline__ int pair32(int p, int q) {
  return p * (p - 1) / 2 + q;
}

// Fixed-order block reduction of one double per thread.
__device__ double block_sum(double x) {
  __shared__ double red[EPI_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = x;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < EPI_THREADS / 32; ++i) s += red[i];
  return s;
}

// ---------------------------------------------------------------- aaa ----

// v[k] += row[p0 + k], k < 8, by aligned loads of four: p0 % 4 is the same
// for the whole warp.  Loads past the row (ld, a multiple of 4) are moved
// back into it; their elements are not needed.
__device__ __forceinline__ void add8_at(const double *row, int p0, int ld,
                                        double (&v)[8]) {
  double q[12];
  const int b = p0 & ~3, last = ld - 4;
  load4(row + min(b, last), q);
  load4(row + min(b + 4, last), q + 4);
  switch (p0 & 3) {
    case 0:
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += q[k];
      return;
    case 1:
      load4(row + min(b + 8, last), q + 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += q[k + 1];
      return;
    case 2:
      load4(row + min(b + 8, last), q + 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += q[k + 2];
      return;
    default:
      load4(row + min(b + 8, last), q + 8);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += q[k + 3];
      return;
  }
}

// row[x0 .. x0 + 7] of a row of ld doubles (x0, ld multiples of 4).
__device__ __forceinline__ void load8(const double *row, int x0, int ld,
                                      double (&v)[8]) {
  load4(row + x0, v);
  load4(row + (x0 + 4 < ld ? x0 + 4 : x0), v + 4);
}

// The same for 16 bytes (both addresses 16-byte aligned).
__device__ __forceinline__ void cp_async16(double *dst, const double *src,
                                           bool ok) {
  asm volatile(
      "cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)),
      "l"(src), "r"(ok ? 16 : 0)
      : "memory");
}

// Staged runs of a packed pair row: [row][pair of doubles][c].
__device__ __forceinline__ int pairs_at(int row, int x, int c) {
  return ((row * 5 + (x >> 1)) * EPI_C + c) * 2 + (x & 1);
}

// The five pairs of base[c * ld + (p0 & ~1) ..] for the tile's 32 c.
__device__ __forceinline__ void stage_pairs(double *dst, const double *base,
                                            int64_t ld, int p0, int c0, int nc,
                                            bool ok) {
  const int row = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ok = ok && c0 + lane < nc;
  const double *src = base + (ok ? (c0 + lane) * ld : 0);
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int x = (p0 & ~1) + 2 * q;
    const bool in = ok && x < ld;
    cp_async16(dst + pairs_at(row, 2 * q, lane), src + (in ? x : 0), in);
  }
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::
                   : "memory");
}

// A persistent CTA's walk over the items of an EpiList, kept in shared
// memory (no registers live across tiles): its tiles come in increasing
// order and an item spans many of them, so the binary search (a chain of
// dependent global loads) runs only when a tile leaves the current item, and
// the case arguments are copied to shared memory only when they change
// (items of one spin case of one plan share them).  Thread 0 advances it
// before the barrier that ends a tile.
struct ItemWalk {
  int cur, next_begin;          // item index; first tile of the next item
  const EpiArgs *staged;        // whose arguments shared memory holds
  __device__ __forceinline__ void seek(const EpiList *l, int blk) {
    if (blk < next_begin) return;
    cur = find_entry(l->items, l->nitems, blk, &EpiItem::block_begin);
    next_begin = cur + 1 < l->nitems ? l->items[cur + 1].block_begin
                                     : 0x7fffffff;
  }
};

// Copies an item's case arguments into shared memory (all threads).
__device__ __forceinline__ void load_args(EpiArgs &dst, const EpiArgs *src) {
  static_assert(sizeof(EpiArgs) % 8 == 0, "8-byte words");
  constexpr int W = (int)(sizeof(EpiArgs) / 8);
  for (int x = threadIdx.x; x < W; x += blockDim.x)
    reinterpret_cast<long long *>(&dst)[x] =
        reinterpret_cast<const long long *>(src)[x];
  __syncthreads();
}

template <bool FT, bool LOOP, bool HASF>
__global__ void __launch_bounds__(EPI_THREADS, epi_minb(FT))
    epi_aaa_kernel(const EpiList *__restrict__ list,
                   const EpiItem *__restrict__ items) {
  extern __shared__ double sm[];   // EPI_SA_*, then (T): T[c][ab] runs
  __shared__ EpiArgs p;
  double *s3 = sm + EPI_SA_SIZE;
  // LOOP: a fixed grid striding over the flat tiles of all items; else one
  // CTA per (tile, item) of a 2-D grid
  int blk = blockIdx.x;
  if (LOOP && blk >= list->nblocks) return;
  __shared__ ItemWalk walk;
  if (LOOP) {
    if (threadIdx.x == 0) {
      walk.next_begin = 0;
      walk.staged = nullptr;
      walk.seek(list, blk);
    }
    __syncthreads();
  }
  do {
  const EpiItem &item = LOOP ? list->items[walk.cur] : items[blockIdx.y];
  const int local = LOOP ? blk - item.block_begin : blk;
  if (!LOOP && local >= item.nblk) return;
  if (!LOOP || item.args != walk.staged) {   // uniform over the CTA
    load_args(p, item.args);   // ends with a barrier
    if (LOOP && threadIdx.x == 0) walk.staged = item.args;
  }
  const int4 tl = p.tiles[local];
  const int a0 = tl.x, b0 = tl.y, c0 = tl.z;
  const int i = item.i, j = item.j, k = item.k;
  const int v = p.va, o = p.oa;
  const bool has_f = HASF && p.has_f != 0;   // HASF false: f_ov is zero
  const int g1l = (int)p.g1_ld_aa, g2l = (int)p.g2_ld_aa;
  const double *base = item.ws;
  const double *T = base + p.offL[0];
  const double *R = FT ? base + p.offR[0] : nullptr;
  const int ldi = (int)p.ld[0];

  const int a_ = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = a0 + a_, c = c0 + lane;
  const int ac = a < v ? a : v - 1;       // clamped indices for addressing
  const int cc = c < v ? c : v - 1;
  if (!FT)
    stage_pairs(s3, T, ldi, pair32(ac, b0), c0, v, a < v);
  // disconnected term (src/pt.c:162-175)
  const int64_t sl1 = (int64_t)v * p.g1_ld_aa, sl2 = (int64_t)v * p.g2_ld_aa;
  const double *u1 = p.ov1_a, *u2 = p.ov2_a;
  // its parts that vary with b are the same for every warp: staged once
  // (zero outside the space; those elements are masked)
  {
    const int t = threadIdx.x;
    const int bt = b0 + (t >> 5), ct = c0 + (t & 31);
    const bool okbc = bt < v && ct < v;
#pragma unroll
    for (int h = 0; h < (HASF ? 2 : 1); ++h) {
      if (h && !has_f) break;
      const int64_t sl = h ? sl2 : sl1;
      const int ld = h ? g2l : g1l;
      const double *g = h ? p.g2_aa : p.g1_aa;
      const double *gs[3] = {g + ((int64_t)j * o + k) * sl,
                             g + ((int64_t)i * o + k) * sl,
                             g + ((int64_t)j * o + i) * sl};
      double *s = sm + h * EPI_SA_F;
#pragma unroll
      for (int q = 0; q < 3; ++q)
        cp_async8(&s[EPI_SA_BC + 256 * q + t], gs[q] + (okbc ? bt * ld + ct : 0),
                  okbc);
      if (t < EPI_B * EPI_A) {
        const int bb = b0 + (t >> 3), aa = a0 + (t & 7);
        const bool ok = bb < v && aa < v;
#pragma unroll
        for (int q = 0; q < 3; ++q)
          cp_async8(&s[EPI_SA_BA + 64 * q + t], gs[q] + (ok ? bb * ld + aa : 0),
                    ok);
      } else if (t < EPI_B * EPI_A + 3 * EPI_B) {
        const int q = (t - EPI_B * EPI_A) >> 3, bb = b0 + (t & 7);
        const int occ = q == 0 ? i : q == 1 ? j : k;
        cp_async8(&s[EPI_SA_T1 + (t - EPI_B * EPI_A)],
                  (h ? u2 : u1) + (bb < v ? occ * v + bb : 0), bb < v);
      } else if (h == 0 && t < EPI_B * EPI_A + 4 * EPI_B) {
        const int bb = b0 + (t & 7);
        cp_async8(&s[EPI_SA_DJ + (t & 7)], p.d_a + (bb < v ? j * v + bb : 0),
                  bb < v);
      }
    }
  }
  const int64_t ac1 = (int64_t)ac * p.g1_ld_aa + cc,
                ac2 = (int64_t)ac * p.g2_ld_aa + cc;
  const double *g1 = p.g1_aa, *g2 = p.g2_aa;
  const int64_t sjk = (int64_t)j * o + k, sik = (int64_t)i * o + k,
                sji = (int64_t)j * o + i;
  const double A1jk = g1[sjk * sl1 + ac1], A1ik = g1[sik * sl1 + ac1],
               A1ji = g1[sji * sl1 + ac1];
  const double A2jk = g2[sjk * sl2 + ac2], A2ik = g2[sik * sl2 + ac2],
               A2ji = g2[sji * sl2 + ac2];
  const double t1ia = u1[i * v + ac], t1ja = u1[j * v + ac],
               t1ka = u1[k * v + ac];
  const double t1ic = u1[i * v + cc], t1jc = u1[j * v + cc],
               t1kc = u1[k * v + cc];
  const double f_ia = u2[i * v + ac], f_ja = u2[j * v + ac],
               f_ka = u2[k * v + ac];
  const double f_ic = u2[i * v + cc], f_jc = u2[j * v + cc],
               f_kc = u2[k * v + cc];
  const double dia = p.d_a[i * v + ac], dkc = p.d_a[k * v + cc];
  // W (and R) of the thread's 8 b; the pair index needs c < b (else any
  // element of the row: those are masked)
  double w8[EPI_B], r8[EPI_B];
#pragma unroll
  for (int side = 0; side < (FT ? 2 : 1); ++side) {
    const double *X = side ? R : T;
    double(&w)[EPI_B] = side ? r8 : w8;
#pragma unroll
    for (int b_ = 0; b_ < EPI_B; ++b_) {
      const int b = b0 + b_;
      const int bc = b < v ? b : v - 1;
      const int cb = c < b && b < a && a < v ? c : 0;
      // offsets < 2^31 (checked by the plan)
      w[b_] = X[ac * ldi + pair32(bc, cb)] - X[bc * ldi + pair32(ac, cb)];
    }
    if (FT) add8_at(X + (int64_t)cc * ldi, pair32(ac, b0), ldi, w);
  }
  cp_async_wait_all();
  __syncthreads();

  double e = 0.0;
#pragma unroll
  for (int b_ = 0; b_ < EPI_B; ++b_) {
    const int b = b0 + b_;
    const bool ok = a < v && b < a && c < b;
    const double w =
        FT ? w8[b_]
           : w8[b_] + s3[pairs_at(a_, b_ + (pair32(ac, b0) & 1), lane)];
    const double rr = FT ? r8[b_] : w;
    const double *bc = sm + EPI_SA_BC + b_ * EPI_C + lane;
    const double *ba = sm + EPI_SA_BA + b_ * EPI_A + a_;
    const double *tb = sm + EPI_SA_T1 + b_;
    // the 9-term sums of src/pt.c:166-174 for (t1, i_oovv) and (f_ov, t2);
    // the second is skipped when f_ov is zero (its terms would all be 0)
    double x = t1ia * bc[0] - t1ja * bc[256] - t1ka * bc[512] - tb[0] * A1jk +
               tb[8] * A1ik + tb[16] * A1ji - t1ic * ba[0] + t1jc * ba[64] +
               t1kc * ba[128];
    if (has_f) {
      bc += EPI_SA_F;
      ba += EPI_SA_F;
      tb += EPI_SA_F;
      x += f_ia * bc[0] - f_ja * bc[256] - f_ka * bc[512] - tb[0] * A2jk +
           tb[8] * A2ik + tb[16] * A2ji - f_ic * ba[0] + f_jc * ba[64] +
           f_kc * ba[128];
    }
    const double dd = (dia + sm[EPI_SA_DJ + b_]) + dkc;
    if (ok) e += (w - x) * rr * recip_nr(dd);
  }
  const double s = block_sum(e);
  if (threadIdx.x == 0) item.partials[local] = s;
  if (!LOOP) break;
  blk += gridDim.x;
  if (threadIdx.x == 0) walk.seek(list, blk);
  __syncthreads();   // shared memory is refilled by the next tile
  } while (blk < list->nblocks);
}

// ---------------------------------------------------------------- aab ----

template <bool FT, bool LOOP, bool HASF>
__global__ void __launch_bounds__(EPI_THREADS, epi_minb(FT))
    epi_aab_kernel(const EpiList *__restrict__ list,
                   const EpiItem *__restrict__ items) {
  extern __shared__ double sm[];
  __shared__ EpiArgs p;
  constexpr int S = EPI_A * EPI_B * (FT ? EPI_C : EPI_CS);
  // (T): sy[b_][a_][c_] = U2[b][c][a], sx[a_][b_][c_] = U2[a][c][b],
  //      sp[a_][b_][c_] = P[c][pair(a,b)]
  // (fT): sy, then its R copy
  double *sy = sm, *sx = sm + S, *sp = sm + 2 * S;
  // LOOP: a fixed grid striding over the flat tiles of all items; else one
  // CTA per (tile, item) of a 2-D grid
  int blk = blockIdx.x;
  if (LOOP && blk >= list->nblocks) return;
  __shared__ ItemWalk walk;
  if (LOOP) {
    if (threadIdx.x == 0) {
      walk.next_begin = 0;
      walk.staged = nullptr;
      walk.seek(list, blk);
    }
    __syncthreads();
  }
  do {
  const EpiItem &item = LOOP ? list->items[walk.cur] : items[blockIdx.y];
  const int local = LOOP ? blk - item.block_begin : blk;
  if (!LOOP && local >= item.nblk) return;
  if (!LOOP || item.args != walk.staged) {   // uniform over the CTA
    load_args(p, item.args);   // ends with a barrier
    if (LOOP && threadIdx.x == 0) walk.staged = item.args;
  }
  const int npairs = p.ntiles / p.ctiles;   // tiles: c block major
  // the (a, b) tiles are the triangle a0 = 8t, b0 = 8u, u <= t, in row
  // order (the last row may stop at u = t - 1); tile L sits in row
  // t = floor((sqrt(8L + 1) - 1) / 2), computed here instead of loaded from
  // the case's tile table, so the data loads need one dependent load less
  const int L = local % npairs;
  int t = (int)((sqrtf(8.0f * (float)L + 1.0f) - 1.0f) * 0.5f);
  while ((t + 1) * (t + 2) / 2 <= L) ++t;
  while (t * (t + 1) / 2 > L) --t;
  const int a0 = EPI_A * t, b0 = EPI_B * (L - t * (t + 1) / 2);
  const int c0 = (local / npairs) * EPI_C;
  const int i = item.i, j = item.j, k = item.k;
  const int oa = p.oa, va = p.va, ob = p.ob, vb = p.vb;
  const double *base = item.ws;
  const int64_t ld2 = p.ld[1];
  const int ldp = (int)p.ld[2], r2 = (int)p.rowU2;
  // 32-bit strides for the per-element loop (the plan keeps a triple's
  // arrays and the i_oovv / amplitude slices under 2^31 elements)
  const int ld1 = (int)p.ld[0], r1 = (int)p.rowU1;
  const int g1lab = (int)p.g1_ld_ab, g2lab = (int)p.g2_ld_ab;
  const int g1laa = (int)p.g1_ld_aa, g2laa = (int)p.g2_ld_aa;
  const bool has_f = HASF && p.has_f != 0;   // HASF false: f_ov is zero

  const int a_ = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = a0 + a_, c = c0 + lane;
  const int ac = a < va ? a : va - 1, cc = c < vb ? c : vb - 1;
  if (!FT) {
    // thread: one (c, w) of every row u, w the index within the run
    const int w = threadIdx.x & 7, cs = threadIdx.x >> 3, cg = c0 + cs;
    const bool cok = cg < vb;
    const int ax0 = a0, bx = b0 + w, ay = a0 + w;
    const double *px = base + p.offL[1] + (int64_t)a0 * ld2 + cg * r2 + bx;
    const double *py = base + p.offL[1] + (int64_t)b0 * ld2 + cg * r2 + ay;
    const double *pp = base + p.offL[2] + (int64_t)cg * ldp + pair32(a0, bx);
    const bool xok = cok && bx < va, yok = cok && ay < va;
#pragma unroll
    for (int u = 0; u < EPI_A; ++u) {
      const int ax = ax0 + u;
      const int idx = (u * EPI_B + w) * EPI_CS + cs;
      const bool okx = xok && ax < va, oky = yok && b0 + u < va;
      const bool okp = okx && bx < ax;
      cp_async8(&sx[idx], okx ? px : base, okx);
      cp_async8(&sy[idx], oky ? py : base, oky);
      cp_async8(&sp[idx], okp ? pp : base, okp);
      px += ld2;
      py += ld2;
      pp += ax;   // pair(a + 1, b) = pair(a, b) + a
    }
  }
  // disconnected-term slices (src/pt.c:433-442)
  const double *g1jk = p.g1_ab + ((int64_t)j * ob + k) * va * p.g1_ld_ab;
  const double *g1ik = p.g1_ab + ((int64_t)i * ob + k) * va * p.g1_ld_ab;
  const double *g1ji = p.g1_aa + ((int64_t)j * oa + i) * va * p.g1_ld_aa;
  const double *g2jk = p.g2_ab + ((int64_t)j * ob + k) * va * p.g2_ld_ab;
  const double *g2ik = p.g2_ab + ((int64_t)i * ob + k) * va * p.g2_ld_ab;
  const double *g2ji = p.g2_aa + ((int64_t)j * oa + i) * va * p.g2_ld_aa;
  const double *u1 = p.ov1_a, *u2 = p.ov2_a;
  // The parts of the disconnected term that vary with b -- g[b][c] rows,
  // g[b][a], and the per-b amplitudes and denominators -- are the same for
  // every warp (a) of the tile: staged once into shared memory (zero where
  // b or c is outside the space; those elements are masked) instead of
  // loaded by each warp in the b loop.
  double *sd = sm + (FT ? 2 : 3) * S;
  {
    const int t = threadIdx.x;   // one (b, c) per thread
    const int bt = b0 + (t >> 5), ct = c0 + (t & 31);
    const bool okbc = bt < va && ct < vb;
    cp_async8(&sd[EPI_SD_G1JK + t], g1jk + (okbc ? bt * g1lab + ct : 0), okbc);
    cp_async8(&sd[EPI_SD_G1IK + t], g1ik + (okbc ? bt * g1lab + ct : 0), okbc);
    if (has_f) {
      cp_async8(&sd[EPI_SD_G2JK + t], g2jk + (okbc ? bt * g2lab + ct : 0),
                okbc);
      cp_async8(&sd[EPI_SD_G2IK + t], g2ik + (okbc ? bt * g2lab + ct : 0),
                okbc);
    }
    if (t < EPI_B * EPI_A) {   // (b, a) of g[j][i]
      const int bb = b0 + (t >> 3), aa = a0 + (t & 7);
      const bool okba = bb < va && aa < va;
      cp_async8(&sd[EPI_SD_G1JI + t], g1ji + (okba ? bb * g1laa + aa : 0),
                okba);
      if (has_f)
        cp_async8(&sd[EPI_SD_G2JI + t], g2ji + (okba ? bb * g2laa + aa : 0),
                  okba);
    } else if (t < EPI_B * EPI_A + EPI_B) {   // per b
      const int b_ = t - EPI_B * EPI_A, bb = b0 + b_;
      const bool okb = bb < va;
      cp_async8(&sd[EPI_SD_T1I + b_], u1 + (okb ? i * va + bb : 0), okb);
      cp_async8(&sd[EPI_SD_T1J + b_], u1 + (okb ? j * va + bb : 0), okb);
      cp_async8(&sd[EPI_SD_DJ + b_], p.d_a + (okb ? j * va + bb : 0), okb);
      if (has_f) {
        cp_async8(&sd[EPI_SD_F1I + b_], u2 + (okb ? i * va + bb : 0), okb);
        cp_async8(&sd[EPI_SD_F1J + b_], u2 + (okb ? j * va + bb : 0), okb);
      }
    }
  }
  const int64_t ac1 = (int64_t)ac * p.g1_ld_ab + cc,
                ac2 = (int64_t)ac * p.g2_ld_ab + cc;
  const double A1jk = g1jk[ac1], A1ik = g1ik[ac1];
  const double A2jk = g2jk[ac2], A2ik = g2ik[ac2];
  const double t1ia = u1[i * va + ac], t1ja = u1[j * va + ac];
  const double f_ia = u2[i * va + ac], f_ja = u2[j * va + ac];
  const double o1k = p.ov1_b[k * vb + cc], o2k = p.ov2_b[k * vb + cc];
  const double dia = p.d_a[i * va + ac], dkc = p.d_b[k * vb + cc];
  // U1 in both orientations, and for (fT) all of W and R but U2[b][c][a],
  // which this warp reads for b = b0 + a_ and stages for the others
  double w8[EPI_B], r8[EPI_B];
#pragma unroll
  for (int side = 0; side < (FT ? 2 : 1); ++side) {
    const int64_t *off = side ? p.offR : p.offL;
    const double *U1 = base + off[0], *U2 = base + off[1], *P = base + off[2];
    double(&w)[EPI_B] = side ? r8 : w8;
    if (FT) {
      const int by = b0 + a_ < va ? b0 + a_ : va - 1;
      double y[EPI_A];
      load8(U2 + (int64_t)by * ld2 + cc * r2, a0, r2, y);
      load8(U2 + (int64_t)ac * ld2 + cc * r2, b0, r2, w);
#pragma unroll
      for (int x = 0; x < EPI_A; ++x)
        sy[side * S + (a_ * EPI_A + x) * EPI_C + lane] = y[x];
    }
#pragma unroll
    for (int b_ = 0; b_ < EPI_B; ++b_) {   // offsets < 2^31 (plan check)
      const int bc = b0 + b_ < va ? b0 + b_ : va - 1;
      const double u =
          U1[ac * ld1 + bc * r1 + cc] - U1[bc * ld1 + ac * r1 + cc];
      w[b_] = FT ? w[b_] + u : u;
    }
    if (FT) add8_at(P + (int64_t)cc * ldp, pair32(ac, b0), ldp, w);
  }
  cp_async_wait_all();
  __syncthreads();

  double e = 0.0;
#pragma unroll
  for (int b_ = 0; b_ < EPI_B; ++b_) {
    const int b = b0 + b_;
    const bool ok = a < va && b < a && c < vb;
    constexpr int CS = FT ? EPI_C : EPI_CS;
    const int ix = (a_ * EPI_B + b_) * CS + lane;
    const int iy = (b_ * EPI_A + a_) * CS + lane;
    const double w =
        FT ? w8[b_] - sy[iy]
           : w8[b_] + sx[ix] - sy[iy] + sp[ix];
    const double rr = FT ? r8[b_] - sy[S + iy] : w;
    const int bcl = b_ * EPI_C + lane, ba = b_ * EPI_A + a_;
    double x = t1ia * sd[EPI_SD_G1JK + bcl] - sd[EPI_SD_T1I + b_] * A1jk -
               t1ja * sd[EPI_SD_G1IK + bcl] + sd[EPI_SD_T1J + b_] * A1ik +
               o1k * sd[EPI_SD_G1JI + ba];
    if (has_f)   // the (f_ov, t2) half, zero when f_ov is
      x += f_ia * sd[EPI_SD_G2JK + bcl] - sd[EPI_SD_F1I + b_] * A2jk -
           f_ja * sd[EPI_SD_G2IK + bcl] + sd[EPI_SD_F1J + b_] * A2ik +
           o2k * sd[EPI_SD_G2JI + ba];
    const double dd = (dia + sd[EPI_SD_DJ + b_]) + dkc;
    if (ok) e += (w - x) * rr * recip_nr(dd);
  }
  const double s = block_sum(e);
  if (threadIdx.x == 0) item.partials[local] = s;
  if (!LOOP) break;
  blk += gridDim.x;
  if (threadIdx.x == 0) walk.seek(list, blk);
  __syncthreads();   // shared memory is refilled by the next tile
  } while (blk < list->nblocks);
}

__global__ void __launch_bounds__(256)
    reduce_partials_kernel(const RedList *__restrict__ list) {
  __shared__ double red[256];
  const int nitems = list->nitems;
  for (int t = blockIdx.x; t < nitems; t += gridDim.x) {
    const RedItem it = list->items[t];
    double s = 0.0;
    for (int x = threadIdx.x; x < it.n; x += 256) s += it.partials[x];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
      __syncthreads();
    }
    if (threadIdx.x == 0) *it.dst = red[0];
    __syncthreads();
  }
}

template <typename K>
cudaError_t launch_epi(K kern, const EpiList *d_list, const EpiItem *d_items,
                       size_t smem, dim3 grid, cudaStream_t st) {
  cudaError_t e = set_smem(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<grid, EPI_THREADS, smem, st>>>(d_list, d_items);
  return cudaGetLastError();
}

}  // namespace

size_t epi_smem_bytes(bool aab, bool ft) {
  const size_t ab = (size_t)EPI_A * EPI_B;
  const size_t pairs = (size_t)EPI_A * 10 * EPI_C;   // runs of a packed row
  return (aab ? (ft ? 2 * ab * EPI_C : 3 * ab * EPI_CS) + EPI_SD_SIZE
              : EPI_SA_SIZE + (ft ? 0 : pairs)) *
         sizeof(double);
}

int epi_blocks_per_sm(bool aab, bool ft) {
  const size_t smem = epi_smem_bytes(aab, ft);
  int n = 0;
  cudaError_t e;
  if (aab) {
    if (ft) {
      set_smem(epi_aab_kernel<true, true, true>, smem);
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, epi_aab_kernel<true, true, true>, EPI_THREADS, smem);
    } else {
      set_smem(epi_aab_kernel<false, true, true>, smem);
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, epi_aab_kernel<false, true, true>, EPI_THREADS, smem);
    }
  } else {
    if (ft) {
      set_smem(epi_aaa_kernel<true, true, true>, smem);
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, epi_aaa_kernel<true, true, true>, EPI_THREADS, smem);
    } else {
      set_smem(epi_aaa_kernel<false, true, true>, smem);
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, epi_aaa_kernel<false, true, true>, EPI_THREADS, smem);
    }
  }
  return (e == cudaSuccess && n > 0) ? n : 1;
}

// Persistent launches (fixed grids, graph replays) use the general kernels;
// direct launches whose items all have a zero f_ov (hasf false) use the
// kernels compiled without the f_ov terms.
cudaError_t epi_aaa_launch(const EpiList *d_list, const EpiItem *d_items,
                           bool ft, bool hasf, int grid, int nitems,
                           bool persistent, cudaStream_t st) {
  if (grid <= 0 || nitems <= 0) return cudaSuccess;
  if (!persistent && !d_items) return cudaErrorInvalidValue;
  const size_t smem = epi_smem_bytes(false, ft);
  const dim3 g(grid, persistent ? 1 : nitems);
  if (persistent)
    return ft ? launch_epi(epi_aaa_kernel<true, true, true>, d_list, d_items, smem, g, st)
              : launch_epi(epi_aaa_kernel<false, true, true>, d_list, d_items, smem, g, st);
  if (hasf)
    return ft ? launch_epi(epi_aaa_kernel<true, false, true>, d_list, d_items, smem, g, st)
              : launch_epi(epi_aaa_kernel<false, false, true>, d_list, d_items, smem, g, st);
  return ft ? launch_epi(epi_aaa_kernel<true, false, false>, d_list, d_items, smem, g, st)
            : launch_epi(epi_aaa_kernel<false, false, false>, d_list, d_items, smem, g, st);
}

cudaError_t epi_aab_launch(const EpiList *d_list, const EpiItem *d_items,
                           bool ft, bool hasf, int grid, int nitems,
                           bool persistent, cudaStream_t st) {
  if (grid <= 0 || nitems <= 0) return cudaSuccess;
  if (!persistent && !d_items) return cudaErrorInvalidValue;
  const size_t smem = epi_smem_bytes(true, ft);
  const dim3 g(grid, persistent ? 1 : nitems);
  if (persistent)
    return ft ? launch_epi(epi_aab_kernel<true, true, true>, d_list, d_items, smem, g, st)
              : launch_epi(epi_aab_kernel<false, true, true>, d_list, d_items, smem, g, st);
  if (hasf)
    return ft ? launch_epi(epi_aab_kernel<true, false, true>, d_list, d_items, smem, g, st)
              : launch_epi(epi_aab_kernel<false, false, true>, d_list, d_items, smem, g, st);
  return ft ? launch_epi(epi_aab_kernel<true, false, false>, d_list, d_items, smem, g, st)
            : launch_epi(epi_aab_kernel<false, false, false>, d_list, d_items, smem, g, st);
}

cudaError_t reduce_partials_launch(const RedList *d_list, int grid,
                                   cudaStream_t st) {
  if (grid <= 0) return cudaSuccess;
  reduce_partials_kernel<<<grid, 256, 0, st>>>(d_list);
  return cudaGetLastError();
}

}  // namespace ptb
