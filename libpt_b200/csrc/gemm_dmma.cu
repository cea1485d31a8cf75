// FP64 contraction kernel: signed multi-segment GEMM on DMMA tensor cores.
//
// Replaces the reference's per-triple dgemm_ calls (src/pt.c:40-160): one
// CTA computes a BM x 128 tile of one triple's contraction output, summing
// all of that output's amplitude x integral products (up to six, each with
// its own sign) in one K loop, so the permuted contributions the reference
// adds one GEMM at a time (e.g. src/pt.c:236-290) meet in the accumulator.
//
// Pipeline: one elected lane of the last warp stages A and B tiles with TMA
// into a GEMM_STAGES-deep ring of shared-memory buffers guarded by mbarriers;
// the consumer warps run mma.sync.m16n8k4.f64 on 48 x 32 warp tiles.
// BM is 96 rows (two warp rows, one CTA an SM) or 48 (one warp row, two CTAs
// an SM, whose tile transitions hide behind each other); dmma_rows picks.  A
// job's last M tile multiplies only the 16-row fragments that hold rows of the
// job, shared out to the warp rows of the tile: each has one warp on every SM
// sub-partition, so a tile's DMMA time follows its fragment count (v = 143: 144
// rows of work, not 192).
//
// Shared-memory layouts (no swizzle; TMA box rows are 32 bytes):
//   A stage [k/4][m][k%4]   -- one box of (4 k) x BM rows x 4
//   B stage [n/4][k][n%4]   -- one box of (4 n) x 16 k x 32
// so the fragment loads of a half-warp read 16 consecutive doubles (no bank
// conflicts) for both operands.  The views split K (A) and N (B) in fours to
// make that layout one copy per operand and stage: with a copy per box of 4
// columns (36 per stage) the TMA unit's rate of copies, about one in 90
// cycles, held a stage at 3.4 k cycles whatever its rows; 96 rows of DMMA
// work take 3.1 k.
//
// Persistent: dmma_grid(BM) CTAs take the launch's tiles one at a time from the
// tile queue of a device-memory work list (GemmList; common.cuh tq_*), so
// one launch can hold the triples of many plans, tiles of uneven length
// spread over the SMs, and a captured CUDA graph can be replayed with new
// lists.  The producer takes a tile, hands its index to the consumer warps
// through a shared-memory ring, and runs ahead into the next tile's operands
// while the consumers store the current one.  Each job carries its plan's
// tensor maps (device memory; fenced before first use).
//
// Tiles are numbered M-tile fastest inside a job and taken in order, so the
// CTAs that share one B (OVVV) tile run at the same time and the tile is
// fetched from DRAM once.
// Group jobs (GRP; closed-shell triples, see plan_closed.cu) have columns
// (y, z) over two virtual indices, and their B operands come in both orders:
// [k][y][z], or [k][z][y] for a transposed segment.  A tile covers 8 y x 16 z
// columns and its fragments run along the diagonals of 4 x 4 blocks of
// (y, z): lane g of a fragment reads (y, z) = (g % 4, (g % 4 + s) % 4), s the
// diagonal, so that of either layout
//   [z/4][y][k][z%4]  (natural: one box of (4 z) x 16 k x 8 y x 4)
//   [y/4][z][k][y%4]  (transposed: one box of (4 y) x 16 k x 16 z x 2)
// a half-warp reads 16 different banks.  The sum of both orders therefore
// needs no transposed copy of the integrals.  At the store two lanes exchange
// half of their values so that each holds the four z of one y (32 bytes).
#include "common.cuh"
#include "engine.h"

namespace ptb {

namespace {

constexpr int BN = GEMM_BN, BK = GEMM_BK, ST = GEMM_STAGES;

// Consumer warps of a CTA: warp rows of 16 MF rows, four columns of 32.
template <int BM>
struct Dmma {
  static constexpr int CTAS = BM == 48 ? 2 : 1;   // an SM
  static constexpr int WR = BM > 64 ? 2 : 1;   // warp rows
  static constexpr int MF = BM / (16 * WR);    // m16 fragments of a warp
  static constexpr int NCW = 4 * WR;
  static constexpr int THREADS = (NCW + 1) * 32;
};

template <int BM>
constexpr uint32_t stage_bytes() {
  return (BM * BK + BK * BN) * sizeof(double);
}

// Four K columns of a warp: NF 16-row fragments of A times its 32 columns
// of B.
template <int NF, int MF>
__device__ __forceinline__ void mma_k4(double (&acc)[MF][4][4],
                                       const double *A, const double *B,
                                       const int (&boff)[4],
                                       unsigned long long mask) {
  double a0[NF], a1[NF], b[4];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    a0[f] = flip_sign(A[64 * f], mask);
    a1[f] = flip_sign(A[64 * f + 32], mask);
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) b[h] = B[boff[h]];
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int h = 0; h < 4; ++h) dmma_16x8x4(acc[f][h], a0[f], a1[f], b[h]);
}

// One pipeline stage of a warp: its first nkq fours of K (all of them but in
// a segment's last stage, whose remaining columns are zero).
template <int NF, int MF, int BM>
__device__ __forceinline__ void mma_stage(double (&acc)[MF][4][4],
                                          const double *A, const double *B,
                                          const int (&boff)[4],
                                          unsigned long long mask, int nkq) {
  if (nkq == BK / 4) {
#pragma unroll
    for (int kq = 0; kq < BK / 4; ++kq)
      mma_k4<NF, MF>(acc, A + kq * BM * 4, B + kq * 16, boff, mask);
  } else {
#pragma unroll 1
    for (int kq = 0; kq < nkq; ++kq)
      mma_k4<NF, MF>(acc, A + kq * BM * 4, B + kq * 16, boff, mask);
  }
}

// 9 or 10 warps an SM: one SM sub-partition hosts 3 of them, which bounds the
// kernel at 168 registers per thread (16K registers per sub-partition).  The
// kernels' launch bounds ask for the CTAs an SM that dmma_grid counts on, so
// the compiler keeps to it (158 registers, group kernels 166, no spills).
template <int BM, bool PM, bool GRP>
__device__ __forceinline__ void dmma_body(const LaunchMaps *pm,
                                          const GemmJob *__restrict__ jobs,
                                          const int njobs, const int ntiles,
                                          GemmList *list, unsigned *err) {
  constexpr int MF = Dmma<BM>::MF, NCW = Dmma<BM>::NCW, WR = Dmma<BM>::WR;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double *sA = reinterpret_cast<double *>(smem_raw);
  double *sB = sA + ST * BM * BK;
  uint64_t *full = reinterpret_cast<uint64_t *>(sB + ST * BK * BN);
  uint64_t *empty = full + ST;
  TileRing *tq = reinterpret_cast<TileRing *>(empty + ST);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NCW);
    }
    tq_init(tq, NCW);
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == NCW) {
    // ---------------- producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      int qslot = 0;
      uint32_t qph = 0;
      MapSource<PM> ms(pm);
      // tiles from the launch's queue; the next one is taken while the
      // current one is staged
      int tile = tq_take(list);
      int ji = find_entry(jobs, njobs, tile, &GemmJob::tile_begin);
      while (ok) {
        if (!tq_put(tq, qslot, qph, tile < ntiles ? tile : -1, ji, err) ||
            tile >= ntiles)
          break;
        const int next_tile = tq_take(list);
        const int next_ji = find_entry(jobs, njobs, next_tile,
                                       &GemmJob::tile_begin);
        const GemmJob &job = jobs[ji];
        const int local = tile - job.tile_begin;
        const int m0 = (local % job.mtiles) * BM;
        const int nb = local / job.mtiles;
        const int n0 = nb * BN;
        const int ntz = (job.N + GRP_BZ - 1) / GRP_BZ;   // GRP: N = v
        const int y0 = (nb / ntz) * GRP_BY, z0 = (nb % ntz) * GRP_BZ;
        const int nseg = job.nseg;
        for (int s = 0; s < nseg && ok; ++s) {
          const GemmSeg sg = job.seg[s];
          const CUtensorMap *am = ms.get(job, sg.amap);
          const CUtensorMap *bm = ms.get(job, sg.bmap);
          for (int ks = 0; ks < sg.ksteps; ++ks) {
            if (!mbar_wait(&empty[stage], phase ^ 1u, err)) {
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&full[stage], stage_bytes<BM>());
            double *dA = sA + stage * BM * BK;
            double *dB = sB + stage * BK * BN;
            const int k0 = ks * BK;
            tma_load_5d(dA, am, &full[stage], 0, m0, k0 / 4, sg.a_q, sg.a_p);
            if (!GRP)
              tma_load_4d(dB, bm, &full[stage], 0, k0, n0 / 4, sg.b_p);
            else if (sg.neg & GRP_TR)
              tma_load_5d(dB, bm, &full[stage], 0, k0, z0, y0 / 4, sg.b_p);
            else
              tma_load_5d(dB, bm, &full[stage], 0, k0, y0, z0 / 4, sg.b_p);
            ++issued;
            if (++stage == ST) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
        tile = next_tile;
        ji = next_ji;
      }
      tq_finish(list);
      // Drain: do not leave the CTA while copies issued by it are in flight.
      const int tail = issued < ST ? issued : ST;
      for (int d = 0; d < tail; ++d) {
        int idx = issued - 1 - d;
        mbar_wait(&full[idx % ST], (uint32_t)((idx / ST) & 1), err);
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  const int wn = (warp & 3) * 32;          // warp tile columns
  const int g = lane >> 2, t = lane & 3;

  // Per-lane fragment offsets inside one stage.
  int boff[4], bofft[4];   // bofft: transposed segments of group jobs
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    if (GRP) {
      const int y = 4 * (h >> 1) + (g & 3);
      const int z = 4 * (warp & 3) + ((g + 2 * (h & 1) + (g >> 2)) & 3);
      boff[h] = (((z >> 2) * GRP_BY + y) * BK + t) * 4 + (z & 3);
      bofft[h] = (((y >> 2) * GRP_BZ + z) * BK + t) * 4 + (y & 3);
    } else {
      const int n = wn + 8 * h + g;
      boff[h] = ((n >> 2) * BK + t) * 4 + (n & 3);
      bofft[h] = 0;
    }
  }

  int stage = 0;
  uint32_t phase = 0;
  bool ok = true;
  int qslot = 0;
  uint32_t qph = 0;
  for (;;) {
    int ji;
    const int tile = tq_get(tq, qslot, qph, ji, err, true);
    if (tile < 0) break;
    const GemmJob &job = jobs[ji];
    const int local = tile - job.tile_begin;
    const int m0 = (local % job.mtiles) * BM;
    const int nb = local / job.mtiles;
    const int nseg = job.nseg;

    double acc[MF][4][4];
#pragma unroll
    for (int f = 0; f < MF; ++f)
#pragma unroll
      for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[f][h][e] = 0.0;
    // the tile's 16-row fragments that hold rows of the job, shared out to
    // the two warp rows (a full tile: MF each)
    const int frags = min(WR * MF, (job.M - m0 + 15) >> 4);
    const int f0 = WR == 1 ? frags : (frags + 1) >> 1;
    const int nf = (warp >> 2) ? frags - f0 : f0;
    const int wm = (warp >> 2) ? 16 * f0 : 0;
    const int aoff = (wm + g) * 4 + t;

    for (int s = 0; s < nseg && ok; ++s) {
      const int neg = job.seg[s].neg;
      const unsigned long long mask =
          (GRP ? neg & 1 : neg) ? 0x8000000000000000ull : 0ull;
      int bo[4];
#pragma unroll
      for (int h = 0; h < 4; ++h)
        bo[h] = GRP && (neg & GRP_TR) ? bofft[h] : boff[h];
      const int nk = job.seg[s].ksteps, klast = job.seg[s].klast;
      for (int ks = 0; ks < nk; ++ks) {
        const int nkq = ks + 1 < nk ? BK / 4 : klast;
        if (!mbar_wait(&full[stage], phase, err)) {
          ok = false;
          break;
        }
        const double *A = sA + stage * BM * BK + aoff;
        const double *B = sB + stage * BK * BN;
        if (nf == MF)
          mma_stage<MF, MF, BM>(acc, A, B, bo, mask, nkq);
        else if (nf == 1)
          mma_stage<1, MF, BM>(acc, A, B, bo, mask, nkq);
        else if (nf == 2)
          mma_stage<2, MF, BM>(acc, A, B, bo, mask, nkq);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        if (++stage == ST) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok) break;

    // ---------------- store ----------------
    double *const out = job.out;
    const int64_t ldc = job.ldc;
    const int M = job.M, N = job.N;
    if (GRP) {
      // lanes t and t ^ 2 hold diagonals 0, 2 and 1, 3 of the same two y:
      // each keeps one y and takes its other two values from the partner
      const int v4 = (N + 3) & ~3;
      const int ntz = (N + GRP_BZ - 1) / GRP_BZ;
      const int u = t >> 1, yy = 2 * (t & 1) + u;
      const int z = (nb % ntz) * GRP_BZ + 4 * (warp & 3);
      const bool odd = yy & 1, two = yy & 2;
#pragma unroll
      for (int f = 0; f < MF; ++f) {
        if (f >= nf) break;   // uniform over the warp
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int r = m0 + wm + 16 * f + g + 8 * x;
#pragma unroll
          for (int yq = 0; yq < 2; ++yq) {
            const double e0 = acc[f][2 * yq][2 * x],
                         e1 = acc[f][2 * yq][2 * x + 1],
                         o0 = acc[f][2 * yq + 1][2 * x],
                         o1 = acc[f][2 * yq + 1][2 * x + 1];
            const double re = __shfl_xor_sync(~0u, u ? e0 : e1, 2);
            const double ro = __shfl_xor_sync(~0u, u ? o0 : o1, 2);
            // diagonals 0..3 of this lane's y, then rotated to z order:
            // diagonal s holds z % 4 = (yy + s) % 4
            double d0 = u ? re : e0, d1 = u ? e1 : re, d2 = u ? ro : o0,
                   d3 = u ? o1 : ro;
            if (odd) {
              const double w = d3;
              d3 = d2;
              d2 = d1;
              d1 = d0;
              d0 = w;
            }
            const double s0 = two ? d2 : d0, s1 = two ? d3 : d1,
                         s2 = two ? d0 : d2, s3 = two ? d1 : d3;
            const int y = (nb / ntz) * GRP_BY + 4 * yq + yy;
            if (r < M && y < N && z < v4)
              asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(
                               out + (int64_t)r * ldc + y * v4 + z),
                           "d"(s0), "d"(s1), "d"(s2), "d"(s3)
                           : "memory");
          }
        }
      }
      continue;
    }
    const int n0 = nb * BN;
#pragma unroll
    for (int f = 0; f < MF; ++f) {
      if (f >= nf) break;
      const int r = m0 + wm + 16 * f + g;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int c = n0 + wn + 8 * h + 2 * t;
        if (c < N) {
          if (r < M)
            *reinterpret_cast<double2 *>(out + (int64_t)r * ldc + c) =
                make_double2(acc[f][h][0], acc[f][h][1]);
          if (r + 8 < M)
            *reinterpret_cast<double2 *>(out + (int64_t)(r + 8) * ldc + c) =
                make_double2(acc[f][h][2], acc[f][h][3]);
        }
      }
    }
  }
}

template <int BM>
__global__ void __launch_bounds__(Dmma<BM>::THREADS, Dmma<BM>::CTAS)
    gemm_dmma_kernel(const __grid_constant__ LaunchMaps pm,
                     const GemmJob *__restrict__ jobs, int njobs, int ntiles,
                     GemmList *list, unsigned *err) {
  dmma_body<BM, true, false>(&pm, jobs, njobs, ntiles, list, err);
}

template <int BM>
__global__ void __launch_bounds__(Dmma<BM>::THREADS, Dmma<BM>::CTAS)
    gemm_dmma_kernel_dm(const GemmJob *__restrict__ jobs, GemmList *list,
                        unsigned *err) {
  dmma_body<BM, false, false>(nullptr, jobs, list->njobs, list->ntiles, list, err);
}

// Group jobs (direct launches only).
template <int BM>
__global__ void __launch_bounds__(Dmma<BM>::THREADS, Dmma<BM>::CTAS)
    gemm_dmma_grp_kernel(const __grid_constant__ LaunchMaps pm,
                         const GemmJob *__restrict__ jobs, int njobs,
                         int ntiles, GemmList *list, unsigned *err) {
  dmma_body<BM, true, true>(&pm, jobs, njobs, ntiles, list, err);
}

template <int BM>
cudaError_t launch_grp(const GemmJob *d_jobs, GemmList *d_list, int njobs,
                       int ntiles, const LaunchMaps *pm, int grid,
                       unsigned *d_err, cudaStream_t st) {
  const size_t smem = gemm_smem_bytes(BM);
  const cudaError_t e = set_smem(gemm_dmma_grp_kernel<BM>, smem);
  if (e != cudaSuccess) return e;
  gemm_dmma_grp_kernel<BM><<<grid, Dmma<BM>::THREADS, smem, st>>>(
      *pm, d_jobs, njobs, ntiles, d_list, d_err);
  return cudaGetLastError();
}

template <int BM>
cudaError_t launch(const GemmJob *d_jobs, GemmList *d_list, int njobs,
                   int ntiles, const LaunchMaps *pm, int grid, unsigned *d_err,
                   cudaStream_t st) {
  const size_t smem = gemm_smem_bytes(BM);
  const cudaError_t e = pm ? set_smem(gemm_dmma_kernel<BM>, smem)
                           : set_smem(gemm_dmma_kernel_dm<BM>, smem);
  if (e != cudaSuccess) return e;
  if (pm)
    gemm_dmma_kernel<BM><<<grid, Dmma<BM>::THREADS, smem, st>>>(*pm, d_jobs, njobs,
                                                           ntiles, d_list,
                                                           d_err);
  else
    gemm_dmma_kernel_dm<BM><<<grid, Dmma<BM>::THREADS, smem, st>>>(d_jobs, d_list,
                                                              d_err);
  return cudaGetLastError();
}

}  // namespace

size_t gemm_smem_bytes(int bm) {
  return (size_t)ST * (bm * BK + BK * BN) * sizeof(double) +
         2 * ST * sizeof(uint64_t) + sizeof(TileRing);
}

cudaError_t gemm_dmma_launch(const GemmJob *d_jobs, GemmList *d_list,
                             int njobs, int ntiles, const LaunchMaps *pm,
                             int bm, int grid, unsigned *d_err,
                             cudaStream_t st) {
  if (grid <= 0) return cudaSuccess;
  if (bm == 48)
    return launch<48>(d_jobs, d_list, njobs, ntiles, pm, grid, d_err, st);
  return launch<96>(d_jobs, d_list, njobs, ntiles, pm, grid, d_err, st);
}

cudaError_t gemm_dmma_grp_launch(const GemmJob *d_jobs, GemmList *d_list,
                                 int njobs, int ntiles, const LaunchMaps *pm,
                                 int bm, int grid, unsigned *d_err,
                                 cudaStream_t st) {
  if (grid <= 0) return cudaSuccess;
  if (!pm) return cudaErrorInvalidValue;
  if (bm == 48)
    return launch_grp<48>(d_jobs, d_list, njobs, ntiles, pm, grid, d_err, st);
  return launch_grp<96>(d_jobs, d_list, njobs, ntiles, pm, grid, d_err, st);
}

}  // namespace ptb
