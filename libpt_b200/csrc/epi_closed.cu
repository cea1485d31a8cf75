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

// Block order of (a, b, c) in each of the six permutations of the tile's
// index blocks (0, 1, 2) = (X, Y, Z).
__device__ __forceinline__ void perm_blocks(int p, int &a, int &b, int &c) {
  a = p >> 1;
  const int lo = a == 0 ? 1 : 0, hi = a == 2 ? 1 : 2;
  b = (p & 1) ? hi : lo;
  c = (p & 1) ? lo : hi;
}

__device__ __forceinline__ void ld4(const double *p, double *v) {
  asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}

// v[8] = A1[a][b][c] + A2[b][a][c] + A3[c][b][a] for a = a0 .. a0+7 (b and c
// inside the space; zero beyond it).  ldr = v pad4(v), v4 = pad4(v).
__device__ __forceinline__ void gather(const double *A1, const double *A2,
                                       const double *A3, int64_t ldr, int v,
                                       int v4, int a0, int b, int c,
                                       double (&out)[T]) {
  double x[T], y[T], z[T];
  const double *p1 = A1 + b * v4 + c, *p2 = A2 + b * ldr + c,
               *p3 = A3 + c * ldr + b * v4 + a0;
#pragma unroll
  for (int a = 0; a < T; ++a) {
    const bool ok = a0 + a < v;
    x[a] = ok ? __ldg(p1 + (a0 + a) * ldr) : 0.0;
    y[a] = ok ? __ldg(p2 + (a0 + a) * v4) : 0.0;
    z[a] = 0.0;
  }
  ld4(p3, z);                          // a0 < v: the row holds these four
  if (a0 + 4 < v4) ld4(p3 + 4, z + 4);
#pragma unroll
  for (int a = 0; a < T; ++a) out[a] = x[a] + y[a] + z[a];
}

// Energies of one tile of one group: the unordered index sets {x >= y >= z}
// with x, y, z in the tile's blocks X >= Y >= Z.  384 threads: phase 1, one
// permutation of the blocks per 64 threads (a thread holds 8 a of one (b, c))
// gathers V and V - X into shared memory, so every contraction output is read
// once; phase 2, one index set per thread, adds the four triples' energies.
//
// Bound: HBM, 24 v^3 bytes of contraction outputs a group (48 for (fT)).
// One pass for the four triples reads them once; the general epilogues would
// read 8 (3 v^3 / 6 + 3 * 5 v^3 / 2) bytes for the same triples, 2.6 times
// as many, and evaluate nine disconnected terms a set instead of six shorter
// ones.
template <bool FT, bool HASF>
__global__ void __launch_bounds__(GEPI_THREADS, 2)
    epi_closed_kernel(const EpiItem *__restrict__ items) {
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
  const int blk[3] = {tl.x, tl.y, tl.z};
  const int v = p.va, o = p.oa, v4 = (int)p.rowU1;
  const int64_t ldr = p.ld[0];
  const int occ[3] = {item.i, item.j, item.k};
  const bool has_f = HASF && p.has_f != 0;
  if (threadIdx.x < 9 * T) {
    const int q = threadIdx.x / (3 * T), bl = (threadIdx.x / T) % 3,
              x = threadIdx.x % T;
    const int q_ = q == 0 ? occ[0] : q == 1 ? occ[1] : occ[2];
    const int n = (bl == 0 ? blk[0] : bl == 1 ? blk[1] : blk[2]) + x;
    const bool ok = n < v;
    sd[q][bl][x] = ok ? p.d_a[q_ * v + n] : 0.0;
    su[q][bl][x] = ok ? p.ov1_a[q_ * v + n] : 0.0;
    sf[q][bl][x] = ok && has_f ? p.ov2_a[q_ * v + n] : 0.0;
  }
  __syncthreads();

  double *sU = sm, *sW = sm + 6 * PB;   // V - X, and V (or R)
  {
    const int pm = threadIdx.x / (T * T), bl = (threadIdx.x / T) % T,
              cl = threadIdx.x % T;
    int ab, bb, cb;
    perm_blocks(pm, ab, bb, cb);
    const int a0 = ab == 0 ? blk[0] : ab == 1 ? blk[1] : blk[2];
    const int b = (bb == 0 ? blk[0] : bb == 1 ? blk[1] : blk[2]) + bl;
    const int c = (cb == 0 ? blk[0] : cb == 1 ? blk[1] : blk[2]) + cl;
    const bool ok = b < v && c < v;
    double w[T], u[T];
    if (ok) {
      const double *base = item.ws;
      gather(base + p.offL[0], base + p.offL[1], base + p.offL[2], ldr, v, v4,
             a0, b, c, w);
      // X over (t1, i_oovv), then (f_ov, t2)
      double x[T];
      {
        const int ld = (int)p.g1_ld_ab;
        const int64_t sl = (int64_t)v * ld;
        const double *gjk = p.g1_ab + ((int64_t)occ[1] * o + occ[2]) * sl;
        const double *gik = p.g1_ab + ((int64_t)occ[0] * o + occ[2]) * sl;
        const double *gij = p.g1_ab + ((int64_t)occ[0] * o + occ[1]) * sl;
        const double g0 = gjk[b * ld + c], ub = su[1][bb][bl],
                     uc = su[2][cb][cl];
#pragma unroll
        for (int a = 0; a < T; ++a) {
          const int ac = a0 + a < v ? a0 + a : v - 1;
          x[a] = su[0][ab][a] * g0 + ub * gik[ac * ld + c] +
                 uc * gij[ac * ld + b];
        }
      }
      if (has_f) {
        const int ld = (int)p.g2_ld_ab;
        const int64_t sl = (int64_t)v * ld;
        const double *gjk = p.g2_ab + ((int64_t)occ[1] * o + occ[2]) * sl;
        const double *gik = p.g2_ab + ((int64_t)occ[0] * o + occ[2]) * sl;
        const double *gij = p.g2_ab + ((int64_t)occ[0] * o + occ[1]) * sl;
        const double g0 = gjk[b * ld + c], ub = sf[1][bb][bl],
                     uc = sf[2][cb][cl];
#pragma unroll
        for (int a = 0; a < T; ++a) {
          const int ac = a0 + a < v ? a0 + a : v - 1;
          x[a] += sf[0][ab][a] * g0 + ub * gik[ac * ld + c] +
                  uc * gij[ac * ld + b];
        }
      }
#pragma unroll
      for (int a = 0; a < T; ++a) u[a] = w[a] - x[a];
      if (FT)
        gather(base + p.offR[0], base + p.offR[1], base + p.offR[2], ldr, v,
               v4, a0, b, c, w);
    } else {
#pragma unroll
      for (int a = 0; a < T; ++a) u[a] = w[a] = 0.0;
    }
#pragma unroll
    for (int a = 0; a < T; ++a) {
      sU[pm * PB + a * S1 + bl * S2 + cl] = u[a];
      sW[pm * PB + a * S1 + bl * S2 + cl] = w[a];
    }
  }
  __syncthreads();

  double e[4] = {0.0, 0.0, 0.0, 0.0};
  for (int s = threadIdx.x; s < T * T * T; s += GEPI_THREADS) {
    const int xl = s / (T * T), yl = (s / T) % T, zl = s % T;
    const int x = blk[0] + xl, y = blk[1] + yl, z = blk[2] + zl;
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
    for (int q = 0; q < 6; ++q) {
      u[q] = sU[q * PB + at[q]];
      w[q] = sW[q * PB + at[q]];
    }
    // 1 / (d_i + d_j + d_k), of each permutation that an energy uses
    const double r0 =
        recip_nr((sd[0][0][xl] + sd[1][1][yl]) + sd[2][2][zl]);
    const double r1 =
        recip_nr((sd[0][0][xl] + sd[1][2][zl]) + sd[2][1][yl]);
    const double r2 =
        recip_nr((sd[0][1][yl] + sd[1][0][xl]) + sd[2][2][zl]);
    const double r3 =
        recip_nr((sd[0][1][yl] + sd[1][2][zl]) + sd[2][0][xl]);
    const double r4 =
        recip_nr((sd[0][2][zl] + sd[1][0][xl]) + sd[2][1][yl]);
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
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int n = 16; n > 0; n >>= 1)
      e[q] += __shfl_down_sync(0xffffffffu, e[q], n);
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = e[q];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int n = 0; n < GEPI_THREADS / 32; ++n) s += red[threadIdx.x][n];
    item.partials[(int64_t)threadIdx.x * item.nblk + tile] = s;
  }
}

constexpr size_t GEPI_SMEM = (size_t)12 * PB * sizeof(double);

template <bool FT, bool HASF>
cudaError_t launch(const EpiItem *d_items, int grid, int nitems,
                   cudaStream_t st) {
  const cudaError_t e = cudaFuncSetAttribute(
      epi_closed_kernel<FT, HASF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      (int)GEPI_SMEM);
  if (e != cudaSuccess) return e;
  epi_closed_kernel<FT, HASF><<<dim3(grid, nitems), GEPI_THREADS, GEPI_SMEM,
                                st>>>(d_items);
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

cudaError_t epi_closed_launch(const EpiItem *d_items, bool ft, bool hasf,
                              int grid, int nitems, cudaStream_t st) {
  if (grid <= 0 || nitems <= 0) return cudaSuccess;
  if (ft)
    return hasf ? launch<true, true>(d_items, grid, nitems, st)
                : launch<true, false>(d_items, grid, nitems, st);
  return hasf ? launch<false, true>(d_items, grid, nitems, st)
              : launch<false, false>(d_items, grid, nitems, st);
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
