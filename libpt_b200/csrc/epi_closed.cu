// Closed-shell triples: the check that a restricted solve's same-spin blocks
// are the antisymmetrised mixed-spin ones, and the energy epilogue of a group
// of triples {i, j, k} (plan_closed.cu).
//
// A group i < j < k holds the same-spin triple (src/pt.c:187-302) and the
// mixed-spin triples (ij;k), (ik;j), (jk;i) (src/pt.c:304-452).  All their
// amplitudes are signed sums of one spin-free tensor
//   V[a,b,c] = A1[a][b][c] + A2[b][a][c] + A3[c][b][a]
// (a at i, b at j, c at k; the three arrays are the group's contraction
// outputs), and their disconnected terms of the same sums of
//   X[a,b,c] = u_ia g_jk[b,c] + u_jb g_ik[a,c] + u_kc g_ij[a,b]
// over (u, g) = (t1, i_oovv) and (f_ov, t2), abab blocks:
//   W(ij;k)[a,b;c] = V[a,b,c] - V[b,a,c]   (a at i, b at j, c at k), and so on
//   W(ijk)[a,b,c]  = the six signed permutations.
// A mixed-spin triple with a repeated index, (ij;i) or (ij;j), is a pair: V of
// (f, s, f), f the repeated index, is symmetric in its outer virtuals,
//   V[a,b,c] = A1[a][b][c] + A1[c][b][a] + Z[b][a][c] + Z[b][c][a]
// from two contraction outputs, A1 of rows f and Z of rows s.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace ptb {

namespace {

constexpr int T = GEPI_T;
static_assert(T == 8, "one lane per c, 8 a values per thread");
// shared-memory strides of one permutation's block (doubles): odd-ish, so
// that reads along any of its indices meet few bank conflicts
constexpr int S2 = T + 1, S1 = T * S2 + T + 1;
constexpr int PB = T * S1;
// one block pair of a staged g slice: rows of T + 1
constexpr int GB = T * (T + 1);

// Block order of (a, b, c) in each of the six permutations of the tile's
// index blocks (0, 1, 2) = (X, Y, Z).
__device__ __forceinline__ void perm_blocks(int p, int &a, int &b, int &c) {
  a = p >> 1;
  const int lo = a == 0 ? 1 : 0, hi = a == 2 ? 1 : 2;
  b = (p & 1) ? hi : lo;
  c = (p & 1) ? lo : hi;
}

// out[8] = A1[a][b][c] + A2[b][a][c] + A3[c][b][a] for a = a0 .. a0+7; a pair
// also adds A2[b][c][a] (its A3 is A1).  b and c are inside the space, rows
// past it are read at its last row and never used.  ldr = v pad4(v), v4 =
// pad4(v).
template <bool PAIR>
__device__ __forceinline__ void gather(const double *A1, const double *A2,
                                       const double *A3, int64_t ldr, int v,
                                       int v4, int a0, int b, int c,
                                       double (&out)[T]) {
  double x[T], y[T], z[T];
  const double *p1 = A1 + b * v4 + c, *p2 = A2 + b * ldr + c,
               *p3 = (PAIR ? A1 : A3) + c * ldr + b * v4 + a0,
               *p4 = A2 + b * ldr + c * v4 + a0;
  const int hi = a0 + 4 < v4 ? 4 : 0;   // a0 < v: the row holds a0 .. a0+3
#pragma unroll
  for (int a = 0; a < T; ++a) {
    const int ac = min(a0 + a, v - 1);
    x[a] = __ldg(p1 + ac * ldr);
    y[a] = __ldg(p2 + ac * v4);
  }
  load4(p3, z);
  load4(p3 + hi, z + 4);
#pragma unroll
  for (int a = 0; a < T; ++a) out[a] = x[a] + y[a] + z[a];
  if (PAIR) {
    load4(p4, z);
    load4(p4 + hi, z + 4);
#pragma unroll
    for (int a = 0; a < T; ++a) out[a] += z[a];
  }
}

// Energies of one tile of one group or pair: the unordered index sets
// {x >= y >= z} with x, y, z in the tile's blocks X >= Y >= Z.  Phase 1: V (and
// R) of every permutation of the blocks into shared memory, 64 threads a
// permutation, a thread holding 8 a of one (b, c), so every contraction output
// is read once; a pair's V is symmetric in its outer virtuals and needs three
// of the six.  Phase 2: an index set at a time, a thread keeping its (y, z):
// X of its permutations from the staged g slices, then the energies.
//
// Bound: HBM, 24 v^3 bytes of contraction outputs a group (48 for (fT), 16 and
// 32 a pair).  One pass for the four triples reads them once; the general
// epilogues would read 8 (3 v^3 / 6 + 3 * 5 v^3 / 2) bytes for the same
// triples, 2.6 times as many, and evaluate nine disconnected terms a set
// instead of six shorter ones.  CTAs of 192 threads, four an SM, so that one's
// loads run beside another's arithmetic (two of 384 that kept V - X and V in
// shared memory: 2.7 TB/s, a quarter of the cycles at barriers).
template <bool FT, bool HASF, bool PAIR>
__global__ void __launch_bounds__(GEPI_THREADS, 4)
    epi_closed_kernel(const EpiItem *__restrict__ items) {
  constexpr int NP = PAIR ? 3 : 6;
  extern __shared__ double sm[];
  __shared__ EpiArgs p;
  __shared__ double sd[3][3][T], su[3][3][T], sf[3][3][T];   // [occ][block][]
  __shared__ double red[4][GEPI_THREADS / 32];
  const EpiItem &item = items[blockIdx.y];
  const int tile = blockIdx.x;
  if (tile >= item.nblk) return;
  {
    constexpr int W = (int)(sizeof(EpiArgs) / 8);
    for (int x = threadIdx.x; x < W; x += GEPI_THREADS)
      reinterpret_cast<long long *>(&p)[x] =
          reinterpret_cast<const long long *>(item.args)[x];
  }
  __syncthreads();
  const int4 tl = p.tiles[tile];
  const int v = p.va, o = p.oa, v4 = (int)p.rowU1;
  const int64_t ldr = p.ld[0];
  const int oi = item.i, oj = item.j, ok_ = item.k;
  const bool has_f = HASF && p.has_f != 0;
  auto block = [&](int n) { return n == 0 ? tl.x : n == 1 ? tl.y : tl.z; };
  double *sW = sm, *sR = sm + NP * PB, *sg = sm + (FT ? 2 : 1) * NP * PB;
  // g_jk, g_ik, g_ij on the six ordered block pairs (of both halves with f)
#pragma unroll
  for (int it = 0; it < (HASF ? 12 : 6); ++it) {
    if (it >= 6 && !has_f) break;
    const int e = threadIdx.x + (it % 6) * GEPI_THREADS;
    const int sl = (e >> 6) / 6, pq = (e >> 6) % 6;
    int P, Q, rest;
    perm_blocks(pq, P, Q, rest);
    const int r = block(P) + ((e >> 3) & 7), c = block(Q) + (e & 7);
    const bool in = r < v && c < v;
    const int ld = (int)(it < 6 ? p.g1_ld_ab : p.g2_ld_ab);
    const double *g = (it < 6 ? p.g1_ab : p.g2_ab) +
                      ((int64_t)(sl == 0 ? oj : oi) * o + (sl == 2 ? oj : ok_)) *
                          v * ld;
    cp_async8(&sg[((it / 6) * 18 + sl * 6 + pq) * GB + ((e >> 3) & 7) * (T + 1) +
                  (e & 7)],
              g + (in ? r * ld + c : 0), in);
  }
  if (threadIdx.x < 9 * T) {
    const int q = threadIdx.x / (3 * T), bl = (threadIdx.x / T) % 3,
              x = threadIdx.x % T;
    const int occ = q == 0 ? oi : q == 1 ? oj : ok_;
    const int n = block(bl) + x;
    const bool in = n < v;
    sd[q][bl][x] = in ? p.d_a[occ * v + n] : 0.0;
    su[q][bl][x] = in ? p.ov1_a[occ * v + n] : 0.0;
    sf[q][bl][x] = in && has_f ? p.ov2_a[occ * v + n] : 0.0;
  }
  const int yl = (threadIdx.x / T) % T, zl = threadIdx.x % T;
  // (perm_blocks' order of (P, Q) is that of (a, b): pairs 0..5 = (X,Y) (X,Z)
  // (Y,X) (Y,Z) (Z,X) (Z,Y))
#pragma unroll 1
  for (int pm = threadIdx.x / (T * T); pm < NP; pm += GEPI_THREADS / (T * T)) {
    int ab, bb, cb;
    perm_blocks(pm, ab, bb, cb);
    const int a0 = block(ab), b = min(block(bb) + yl, v - 1),
              c = min(block(cb) + zl, v - 1);
    const double *base = item.ws;
    double w[T];
    gather<PAIR>(base + p.offL[0], base + p.offL[1], base + p.offL[2], ldr, v,
                 v4, a0, b, c, w);
#pragma unroll
    for (int a = 0; a < T; ++a) sW[pm * PB + a * S1 + yl * S2 + zl] = w[a];
    if (FT) {
      gather<PAIR>(base + p.offR[0], base + p.offR[1], base + p.offR[2], ldr,
                   v, v4, a0, b, c, w);
#pragma unroll
      for (int a = 0; a < T; ++a) sR[pm * PB + a * S1 + yl * S2 + zl] = w[a];
    }
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  double e[4] = {0.0, 0.0, 0.0, 0.0};
  const int y = tl.y + yl, z = tl.z + zl;
  const double diy = sd[0][1][yl], djy = sd[1][1][yl], dky = sd[2][1][yl];
  const double diz = sd[0][2][zl], djz = sd[1][2][zl], dkz = sd[2][2][zl];
#pragma unroll 1
  for (int xl = threadIdx.x / (T * T); xl < T; xl += GEPI_THREADS / (T * T)) {
    const int x = tl.x + xl;
    const bool xy = x > y, yz = y > z;
    // a set with a repeated index has one mixed-spin assignment, not three
    if (x >= v || y >= v || z >= v || x < y || y < z || !(xy || yz)) continue;
    // permutations 0..5 = (x,y,z) (x,z,y) (y,x,z) (y,z,x) (z,x,y) (z,y,x) of
    // (a at i, b at j, c at k), each in the block of its own permutation
    const int at[6] = {xl * S1 + yl * S2 + zl, xl * S1 + zl * S2 + yl,
                       yl * S1 + xl * S2 + zl, yl * S1 + zl * S2 + xl,
                       zl * S1 + xl * S2 + yl, zl * S1 + yl * S2 + xl};
    double u[6], w[6];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      u[q] = sW[q * PB + at[q]];
      w[q] = FT ? sR[q * PB + at[q]] : u[q];
    }
    // X, subtracted from u: pairs 0..5 of a slice at the set's elements
    const int gp[6] = {0 * GB + xl * (T + 1) + yl, 1 * GB + xl * (T + 1) + zl,
                       2 * GB + yl * (T + 1) + xl, 3 * GB + yl * (T + 1) + zl,
                       4 * GB + zl * (T + 1) + xl, 5 * GB + zl * (T + 1) + yl};
#pragma unroll
    for (int h = 0; h < (HASF ? 2 : 1); ++h) {
      if (h && !has_f) break;
      const double(*t)[3][T] = h ? sf : su;
      const double *jk = sg + h * 18 * GB, *ik = jk + 6 * GB, *ij = ik + 6 * GB;
      const double ix = t[0][0][xl], iy = t[0][1][yl], iz = t[0][2][zl];
      const double jx = t[1][0][xl], jy = t[1][1][yl], jz = t[1][2][zl];
      const double kx = t[2][0][xl], ky = t[2][1][yl], kz = t[2][2][zl];
      u[0] -= ix * jk[gp[3]] + jy * ik[gp[1]] + kz * ij[gp[0]];
      u[1] -= ix * jk[gp[5]] + jz * ik[gp[0]] + ky * ij[gp[1]];
      u[2] -= iy * jk[gp[1]] + jx * ik[gp[3]] + kz * ij[gp[2]];
      if (!PAIR) {
        u[3] -= iy * jk[gp[4]] + jz * ik[gp[2]] + kx * ij[gp[3]];
        u[4] -= iz * jk[gp[0]] + jx * ik[gp[5]] + ky * ij[gp[4]];
        u[5] -= iz * jk[gp[2]] + jy * ik[gp[4]] + kx * ij[gp[5]];
      }
    }
    // 1 / (d_i + d_j + d_k) of each permutation that an energy uses
    const double dix = sd[0][0][xl], djx = sd[1][0][xl], dkx = sd[2][0][xl];
    if (PAIR) {
      // one triple: (f,s;f) of (ij;i), or (s,f;f) of (ij;j), whose W has the
      // other sign and whose a lies at s; (y,z,x) = (x,z,y), (z,x,y) =
      // (y,x,z), (z,y,x) = (x,y,z)
      const bool sw = item.pad_ != 0;
      const double d0 = sw ? (diy + djx) + dkz : (dix + djy) + dkz;
      const double d1 = sw ? (diz + djx) + dky : (dix + djz) + dky;
      const double d3 = sw ? (diz + djy) + dkx : (diy + djz) + dkx;
      if (xy) e[0] += (u[0] - u[2]) * (w[0] - w[2]) * recip_nr(d0);
      if (xy && yz) e[0] += (u[1] - u[2]) * (w[1] - w[2]) * recip_nr(d1);
      if (yz) e[0] += (u[1] - u[0]) * (w[1] - w[0]) * recip_nr(d3);
      continue;
    }
    const double r0 = recip_nr((dix + djy) + dkz);
    const double r1 = recip_nr((dix + djz) + dky);
    const double r2 = recip_nr((diy + djx) + dkz);
    const double r3 = recip_nr((diy + djz) + dkx);
    const double r4 = recip_nr((diz + djx) + dky);
    // (p - q) of U times (p - q) of W
    auto term = [&](int q, int n) { return (u[q] - u[n]) * (w[q] - w[n]); };
    if (xy && yz) {
      e[0] += (((u[0] - u[1]) - (u[2] - u[3])) + (u[4] - u[5])) *
              (((w[0] - w[1]) - (w[2] - w[3])) + (w[4] - w[5])) * r0;
      // (a, b; c) = (x, z; y)
      e[1] += term(1, 4) * r1;
      e[2] += term(0, 5) * r0;
      e[3] += term(2, 3) * r2;
    }
    if (xy) {   // (x, y; z)
      e[1] += term(0, 2) * r0;
      e[2] += term(1, 3) * r1;
      e[3] += term(4, 5) * r4;
    }
    if (yz) {   // (y, z; x)
      e[1] += term(3, 5) * r3;
      e[2] += term(2, 4) * r2;
      e[3] += term(0, 1) * r0;
    }
  }
  // fixed-order sums over the CTA
#pragma unroll
  for (int q = 0; q < (PAIR ? 1 : 4); ++q) {
#pragma unroll
    for (int n = 16; n > 0; n >>= 1)
      e[q] += __shfl_down_sync(0xffffffffu, e[q], n);
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = e[q];
  }
  __syncthreads();
  if (threadIdx.x < (PAIR ? 1 : 4)) {
    double s = 0.0;
    for (int n = 0; n < GEPI_THREADS / 32; ++n) s += red[threadIdx.x][n];
    item.partials[(int64_t)threadIdx.x * item.nblk + tile] = s;
  }
}

template <bool FT, bool HASF, bool PAIR>
cudaError_t launch(const EpiItem *d_items, int grid, int nitems,
                   cudaStream_t st) {
  constexpr size_t smem =
      ((FT ? 2 : 1) * (PAIR ? 3 : 6) * PB + (HASF ? 36 : 18) * GB) *
      sizeof(double);
  const cudaError_t e = set_smem(epi_closed_kernel<FT, HASF, PAIR>, smem);
  if (e != cudaSuccess) return e;
  epi_closed_kernel<FT, HASF, PAIR>
      <<<dim3(grid, nitems), GEPI_THREADS, smem, st>>>(d_items);
  return cudaGetLastError();
}

// ---- the closed-shell relations -------------------------------------------

__device__ __forceinline__ double warp_max(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(~0u, x, o));
  return x;
}

// Adds a thread's largest deviation and magnitude to dst[0], dst[1] (bit
// patterns of non-negative doubles order like the values).  A NaN deviation
// is recorded as the largest value.
__device__ __forceinline__ void record(double dev, double mag,
                                       unsigned long long *dst) {
  dev = warp_max(dev);
  mag = warp_max(mag);
  if ((threadIdx.x & 31) == 0) {
    if (dev > 0.0)
      atomicMax(&dst[0], (unsigned long long)__double_as_longlong(dev));
    if (mag > 0.0)
      atomicMax(&dst[1], (unsigned long long)__double_as_longlong(mag));
  }
}

__device__ __forceinline__ double deviation(double x, double y) {
  const double d = fabs(x - y);
  return d >= 0.0 ? d : __longlong_as_double(0x7ff0000000000000ll);
}

// Matrices m (v x v): same[m][a][b] against mixed[m][a][b] - mixed[m][b][a],
// and, with `partner`, mixed[m][a][b] against mixed[partner(m)][b][a],
// m = i * o + j, partner = j * o + i.  `same` is packed over a > b
// (row stride lds per m) or has rows of lds.  One 32 x 32 tile at a time
// through shared memory; results per m / per_dst in dst.
__global__ void closed_check_kernel(const double *__restrict__ same,
                                    const double *__restrict__ mixed, int v,
                                    int64_t lds, int64_t ldm, bool packed,
                                    int o, bool partner, int64_t per_dst,
                                    unsigned long long *dst) {
  __shared__ double t[32][33], q[32][33];
  const int64_t m = blockIdx.x;
  const int nb = (v + 31) / 32;
  const double *M = mixed + m * v * ldm;
  const double *P = partner ? mixed + ((m % o) * o + m / o) * v * ldm : M;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double dev = 0.0, mag = 0.0;
  for (int tile = blockIdx.y; tile < nb * nb; tile += gridDim.y) {
    const int a0 = (tile / nb) * 32, b0 = (tile % nb) * 32;
    if (packed && b0 > a0) continue;   // uniform
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
      const bool ok = b0 + r < v && a0 + tx < v;
      t[r][tx] = ok ? M[(b0 + r) * ldm + a0 + tx] : 0.0;
      if (partner) q[r][tx] = ok ? P[(b0 + r) * ldm + a0 + tx] : 0.0;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
      const int a = a0 + r, b = b0 + tx;
      if (a >= v || b >= v || (packed && b >= a)) continue;
      const double x = M[a * ldm + b];
      const double s =
          packed ? same[m * lds + (int64_t)a * (a - 1) / 2 + b]
                 : same[(m * v + a) * lds + b];
      dev = fmax(dev, deviation(s, x - t[tx][r]));
      if (partner) dev = fmax(dev, deviation(x, q[tx][r]));
      mag = fmax(mag, fmax(fabs(x), fabs(t[tx][r])));
    }
  }
  record(dev, mag, dst + 2 * (m / per_dst));
}

// OOVO: same[p][q][n] against mixed[p][q][n] - mixed[q][p][n], n < len.
__global__ void closed_check_oovo_kernel(const double *__restrict__ same,
                                         const double *__restrict__ mixed,
                                         int o, int64_t len,
                                         unsigned long long *dst) {
  const int p = blockIdx.x / o, q = blockIdx.x % o;
  const int64_t pq = (int64_t)blockIdx.x * len, qp = ((int64_t)q * o + p) * len;
  double dev = 0.0, mag = 0.0;
  for (int64_t n = threadIdx.x; n < len; n += blockDim.x) {
    const double x = mixed[pq + n];
    dev = fmax(dev, deviation(same[pq + n], x - mixed[qp + n]));
    mag = fmax(mag, fabs(x));
  }
  record(dev, mag, dst);
}

}  // namespace

cudaError_t epi_closed_launch(const EpiItem *d_items, bool pair, bool ft,
                              bool hasf, int grid, int nitems,
                              cudaStream_t st) {
  if (grid <= 0 || nitems <= 0) return cudaSuccess;
  using F = cudaError_t (*)(const EpiItem *, int, int, cudaStream_t);
  constexpr F f[2][2][2] = {
      {{launch<false, false, false>, launch<false, true, false>},
       {launch<true, false, false>, launch<true, true, false>}},
      {{launch<false, false, true>, launch<false, true, true>},
       {launch<true, false, true>, launch<true, true, true>}}};
  return f[pair][ft][hasf](d_items, grid, nitems, st);
}

cudaError_t closed_check_launch(const double *same, const double *mixed,
                                int64_t nmat, int v, int64_t lds, int64_t ldm,
                                bool packed, int o, bool partner,
                                int64_t per_dst, unsigned long long *dst,
                                cudaStream_t st) {
  if (nmat <= 0 || v <= 0) return cudaSuccess;
  const int nb = (v + 31) / 32;
  // enough CTAs for the device whatever the number of matrices
  const int64_t want = 148 * 8;
  int gy = (int)std::min<int64_t>(nb * nb, (want + nmat - 1) / nmat);
  closed_check_kernel<<<dim3((unsigned)nmat, (unsigned)std::max(gy, 1)), 256, 0,
                        st>>>(same, mixed, v, lds, ldm, packed, o, partner,
                              per_dst, dst);
  return cudaGetLastError();
}

cudaError_t closed_check_oovo_launch(const double *same, const double *mixed,
                                     int o, int64_t len,
                                     unsigned long long *dst,
                                     cudaStream_t st) {
  if (o <= 0 || len <= 0) return cudaSuccess;
  closed_check_oovo_kernel<<<o * o, 256, 0, st>>>(same, mixed, o, len, dst);
  return cudaGetLastError();
}

}  // namespace ptb
