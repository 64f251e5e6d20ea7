// coarsest.cu - direct FP64 solve of the coarsest multigrid level.
//
// The coarsest operator (free DoFs only, compact numbering in reference DoF
// order) is banded: a DoF couples only to DoFs of its own and the two
// neighbouring x-planes, so |i-j| <= band with band about one x-plane of
// DoFs. The setup
//   1. assembles the lower band into band storage,
//   2. factorises it with one persistent kernel: a right-looking band
//      Cholesky over 32-column panels ordered by two progress counters; the
//      CTA that updates the next panel's diagonal block factors it in one
//      warp's registers right away and publishes it (look-ahead), the others
//      fetch the panel rows of their trailing tiles meanwhile, solve them in
//      two warps and update the tile; the factor goes to a separate band array so no
//      CTA reads a panel row another CTA has overwritten,
//   3. splits the rows into P diagonal blocks (boundaries on 32-row panels,
//      each block at least `band` rows, so L is block bidiagonal and block
//      q+1 reaches block q only through a band x band corner), inverts the
//      32x32 diagonal blocks of L and forms W_q = L_qq^-1 for every block by
//      forward substitution in independent 16-column strips (a strip is at
//      most m/32 steps long instead of n/32),
//   4. folds the corners through W_q into G_q = W_q Lc_q and
//      H_q = (Lc_{q+1} W_q[last band rows])^T (FP64 products),
//   5. stores per block W_q (lower triangle), W_q^T (strict upper triangle),
//      G_q and H_q in one row-major matrix in the apply precision.
// The apply z = K^-1 r runs the two triangular solves block by block: a
// lower pass y_q = W_q r_q - G_q y_{q-1}[tail] for q = 0 .. P-1 and an upper
// pass z_q = W_q^T y_q - H_q z_{q+1}[head] for q = P-1 .. 0, each a
// bandwidth-bound product, one warp per row. It reads the P diagonal blocks
// and their couplings (about n^2/P + 2 n band entries) instead of the n^2 of
// the dense W^T W.
//
// Reference: the coarsest solve of GalerkinMatFreeGMG (src/gpu_fem/
// multigrid_v4.py:774-811, 969-984): dense Cholesky with an eps*I retry when a
// pivot is not positive, and two triangular solves per application. The
// factor here is the same (a band Cholesky creates no fill outside the band);
// the triangular solves become products with the explicit inverses of the
// diagonal blocks.
#include "internal.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <stdexcept>
#include <vector>

namespace topo {
namespace cst {

constexpr int CNB = 32;  // panel width

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }

// Band storage: row i holds columns i-band .. i at B[i*ldb + (j - i + band)];
// every access checks i - j <= band first (the band can be narrower than a
// 32-wide panel on small coarsest grids).
__device__ __forceinline__ long long bidx(long long i, long long j, int band, long long ldb) {
  return i * ldb + (j - i + band);
}

// --------------------------------------------------------------- assembly
// one thread per (node, neighbour block)
__global__ void k_band_assemble(Grid g, const double* __restrict__ S, const int* __restrict__ dof_index, int band,
                                long long ldb, double* __restrict__ A) {
  const long long I = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (I >= g.nnodes) return;
  const int iz = (int)(I % g.NZ), iy = (int)((I / g.NZ) % g.NY), ix = (int)(I / ((long long)g.NZ * g.NY));
  const int k = blockIdx.y;
  const int jx = ix + k / 9 - 1, jy = iy + (k / 3) % 3 - 1, jz = iz + k % 3 - 1;
  if (jx < 0 || jx >= g.NX || jy < 0 || jy >= g.NY || jz < 0 || jz >= g.NZ) return;
  const long long J = ((long long)jx * g.NY + jy) * g.NZ + jz;
  int row[3], col[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    row[c] = dof_index[3 * I + c];
    col[c] = dof_index[3 * J + c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (row[c] >= 0 && col[d] >= 0 && col[d] <= row[c] && row[c] - col[d] <= band)
        A[bidx(row[c], col[d], band, ldb)] = S[(long long)(k * 9 + c * 3 + d) * g.nnodes + I];
}

__global__ void k_band_add_diag(int n, int band, long long ldb, double* A, double eps) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) A[bidx(i, i, band, ldb)] += eps;
}

__global__ void k_band_diag_sum(int n, int band, long long ldb, const double* A, double* out) {
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += A[bidx(i, i, band, ldb)];
  double a[1] = {v};
  block_sum<1>(a);
  if (threadIdx.x == 0) *out = a[0];
}

// ------------------------------------------------------------ grid barrier
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Progress of a cooperative launch on monotonic counters: arrive adds one to
// `count` after the CTA's writes, await polls (with a bound: a timeout raises
// err and is reported to every thread of the CTA) until `count` reaches target.
__device__ __forceinline__ void grid_arrive(unsigned* count, unsigned add) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, add);
  }
}

__device__ bool grid_await(const unsigned* count, unsigned target, int* err, int poll) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1, it = 0;
    while (ld_acquire(count) < target) {
      if (++it > poll) {
        ok = 0;
        atomicExch(err, 1);
        break;
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  const bool r = s_ok != 0;
  __syncthreads();  // s_ok is written again by the next call
  return r;
}

// ------------------------------------------------------ persistent Cholesky
// Shared memory of one CTA: the panel's diagonal block W; of its factor the unit
// multipliers MT[j][i] (column j over its pivot, by column) and the reciprocal
// square roots of the pivots, and Ld, the columns themselves before that
// scaling; the panel rows of the two row tiles of the trailing tile it updates
// (by panel column, so that a lane per row and two rows per load are both free
// of bank conflicts); CTA 0's copy of its next tile.
struct __align__(16) CholSmem {
  double Pi[CNB][CNB + 2];
  double Pj[CNB][CNB + 2];
  double A0[CNB][CNB + 2];
  double MT[CNB][CNB + 2];   // MT and invd: published together
  double invd[CNB];
  double col[3][CNB];
  double piv[CNB];
  double Ld[CNB][CNB + 1];
  double W[CNB][CNB + 1];
  int bad, ok;
};
constexpr int LN = CNB * (CNB + 2) + CNB;  // doubles of one published factor

__device__ __forceinline__ void tile_of(int t, int& ti, int& tj) {
  ti = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  while (ti * (ti + 1) / 2 > t) --ti;
  tj = t - ti * (ti + 1) / 2;
}

// 1/d for d in (1e-290, 1e290), where nothing on the way leaves the normal
// numbers: the start r of the PTX instruction rcp.approx.ftz.f64 (its result has
// 20 fraction bits, formed from d's first 20: |e| <= 2^-19 for e = 1 - d r) and
// one step of the hyperpower iteration of order three, r (1 + e + e^2) (Altman,
// Pacific J. Math. 10, 1960), whose error is e^3 <= 2^-57. With the roundings
// of the last two operations that is within one unit in the last place of 1/d,
// which the tests check against the division over the range.
__device__ __forceinline__ double hyper_recip(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

__global__ void k_recip(long long n, const double* __restrict__ d, double* __restrict__ r) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    r[i] = hyper_recip(d[i]);
}

// Two pivots of the warp-register factor of a 32x32 diagonal block (lane =
// row). The pivot index is a template parameter so that every register index
// is a compile-time constant (the array stays in registers). Columns J and J+1
// are broadcast through shared memory together. A warp issues in order and a
// dependent FP64 operation takes about 40 cycles, so the chain is kept short
// and free of branches: the second pivot q1 = d1 - l^2 / d0 is inverted as
// d0 / (d0 d1 - l^2), with the determinant as a difference of products that
// keeps its relative accuracy (Kahan: the rounding of l^2 is taken out again),
// so both reciprocals run side by side. The square roots of all pivots follow
// once at the end. Entries right of a lane's diagonal are updated too but never
// read.
template <int J>
__device__ __forceinline__ void chol_step(double (&wr)[CNB], int lane, CholSmem& S, bool& bad) {
  const double c0 = wr[J], c1 = wr[J + 1];
  S.col[0][lane] = c0;
  S.col[1][lane] = c1;
  __syncwarp();
  const double d0 = S.col[0][J], l = S.col[0][J + 1], d1 = S.col[1][J + 1];
  const double ll = l * l, det = fma(d0, d1, -ll) - fma(l, l, -ll);
  double e0 = d0, e1, r0, r1, t;
  if (d0 > 1e-290 && d0 < 1e290 && det > 1e-290 && det < 1e290) {
    r0 = hyper_recip(d0);
    r1 = d0 * hyper_recip(det);
    t = l * r0;
    e1 = det * r0;
  } else {  // a pivot that is not positive, or out of range (it is then taken as 1)
    const bool ok0 = d0 > 0.0 && isfinite(d0);
    e0 = ok0 ? d0 : 1.0;
    r0 = 1.0 / e0;
    t = l * r0;
    e1 = fma(-l, t, d1);
    const bool ok1 = e1 > 0.0 && isfinite(e1);
    if (!ok1) e1 = 1.0;
    r1 = 1.0 / e1;
    bad |= !ok0 || !ok1;
  }
  const double p1 = fma(-c0, t, c1);  // this lane's entry of column J+1 after pivot J
  S.col[2][lane] = p1;
  const double w0 = c0 * r0, w1 = p1 * r1;
  __syncwarp();
#pragma unroll
  for (int q = J + 2; q < CNB; q += 2) {
    const double2 a = *reinterpret_cast<const double2*>(&S.col[0][q]), b = *reinterpret_cast<const double2*>(&S.col[2][q]);
    wr[q] = fma(-b.x, w1, fma(-a.x, w0, wr[q]));
    wr[q + 1] = fma(-b.y, w1, fma(-a.y, w0, wr[q + 1]));
  }
  S.MT[J][lane] = w0;
  S.MT[J + 1][lane] = w1;
  S.Ld[lane][J] = lane == J ? e0 : c0;
  S.Ld[lane][J + 1] = lane == J + 1 ? e1 : p1;
  if (lane == 0) {
    S.piv[J] = e0;
    S.piv[J + 1] = e1;
  }
  __syncwarp();  // every lane has read the columns that the next round overwrites
  if constexpr (J + 2 < CNB) chol_step<J + 2>(wr, lane, S, bad);
}

// Rows i .. i+31 of panel k (columns k .. k+nb) to P[column][row], zero past
// `lim` or outside the band: warp w of nw takes every nw-th row, lanes along
// the columns (a row is 256 contiguous bytes).
__device__ __forceinline__ void panel_load(const double* A, int band, long long ldb, int k, int nb, int i, int lim,
                                           double (*P)[CNB + 2], int w, int nw, int lane) {
#pragma unroll 8
  for (int r = w; r < CNB; r += nw)
    P[lane][r] = (i + r < lim && lane < nb && i + r - (k + lane) <= band) ? ldcg(A + bidx(i + r, k + lane, band, ldb)) : 0.0;
}

// x Ld^T = a for one row: forward substitution with the unit multipliers (one
// dependent operation per column), scaled by the reciprocal pivots at the end.
template <int J>
__device__ __forceinline__ void solve_step(double (&x)[CNB], const CholSmem& S) {
#pragma unroll
  for (int q = (J + 1) & ~1; q < CNB; q += 2) {
    const double2 m = *reinterpret_cast<const double2*>(&S.MT[J][q]);
    if (q > J) x[q] = fma(-x[J], m.x, x[q]);
    x[q + 1] = fma(-x[J], m.y, x[q + 1]);
  }
  if constexpr (J + 1 < CNB) solve_step<J + 1>(x, S);
}
__device__ __forceinline__ void solve_rows(double (*P)[CNB + 2], const CholSmem& S, int lane) {
  double x[CNB];
#pragma unroll
  for (int j = 0; j < CNB; ++j) x[j] = P[j][lane];
  solve_step<0>(x, S);
#pragma unroll
  for (int j = 0; j < CNB; ++j) P[j][lane] = x[j] * S.invd[j];
}

// Warp 0 factors S.W into S.MT, S.Ld and S.invd; S.bad is set when a pivot was
// not positive (it is then taken as 1).
__device__ __forceinline__ void factor_block(CholSmem& S, int warp, int lane) {
  if (warp == 0) {
    double wr[CNB];
#pragma unroll
    for (int t = 0; t < CNB; ++t) wr[t] = S.W[lane][t];
    bool bad = false;
    chol_step<0>(wr, lane, S, bad);
    __syncwarp();
    S.invd[lane] = rsqrt(S.piv[lane]);
    if (lane == 0) S.bad = bad ? 1 : 0;
  }
}

// Warps: 0 factors diagonal blocks, 2 and 3 solve the panel rows of the two
// row tiles of each trailing tile (3 only for off-diagonal tiles), all 256
// threads update the tile (2x2 outputs each, two partial sums). Look-ahead
// (band >= 32): tile 0 of panel k's trailing update, which CTA 0 owns, is panel
// k+1's diagonal block; CTA 0 keeps its updated values, factors them and
// publishes the factor in Lnext (double-buffered by panel parity), so at panel
// k+1 the other CTAs load it instead of factoring. Panel 0, and every panel when
// the band is narrower than a panel, is factored by every CTA from A.
//
// Order between the panels: count[0] counts the CTAs that have written their
// tiles of a panel, count[32] the published factors. The chain of a panel is
// CTA 0's solve, update, factor and publication; while warp 0 factors, warps
// 4-7 write the factor rows of L, wait for the other CTAs' tiles and fetch the
// next panel's rows. The others fetch their rows while they wait for the
// factor.
//
// Bound by that chain (about 14,000 cycles per panel at band 401: solve 2,700,
// update 1,600, factor 7,200, publication 1,000). With one barrier per panel
// behind a factor of one pivot per round, its square root on the chain, and
// everything above in sequence: 25,000 cycles, 2.97 ms at n = 7,260; now 1.93 ms.
__global__ void __launch_bounds__(256, 1) k_band_chol(int n, int band, long long ldb, double* A, double* L,
                                                      double* Lnext, int* flag, unsigned* count, int* err, int poll) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CholSmem& S = *reinterpret_cast<CholSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool ahead = band >= CNB;
  const int tr = (tid >> 4) * 2, tc = (tid & 15) * 2;  // this thread's 2x2 outputs of a tile
  bool pre = false;  // CTA 0: Pi and A0 hold this panel's first tile already
  auto tile_load = [&](int i0, int j0, int lim, double (&v)[2][2]) {
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int i = i0 + tr + a, j = j0 + tc + b;
        v[a][b] = (i < lim && j < lim && j <= i && i - j <= band) ? ldcg(A + bidx(i, j, band, ldb)) : 0.0;
      }
  };
  for (int k = 0; k < n; k += CNB) {
    const int nb = min(CNB, n - k);
    const int base = k + nb;
    const int lim = min(n, base + band);
    const int nt = (lim - base + CNB - 1) / CNB;
    const int ntiles = lim > base ? nt * (nt + 1) / 2 : 0;
    const int par = (k / CNB) & 1;
    const bool own = ahead && k > 0;  // this panel's factor came from the look-ahead
    const unsigned pi = (unsigned)(k / CNB);
    // 1. the first tile's panel rows and values, and the factored diagonal block
    double a0[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    if (!pre) {
      if (k > 0 && !grid_await(count, pi * gridDim.x, err, poll)) return;
      if ((int)blockIdx.x < ntiles) {
        int ti, tj;
        tile_of(blockIdx.x, ti, tj);
        panel_load(A, band, ldb, k, nb, base + CNB * ti, lim, S.Pi, warp, 8, lane);
        if (tj != ti) panel_load(A, band, ldb, k, nb, base + CNB * tj, lim, S.Pj, warp, 8, lane);
        tile_load(base + CNB * ti, base + CNB * tj, lim, a0);
      }
      if (!own) {
        for (int q = tid; q < CNB * CNB; q += blockDim.x) {
          const int i = q / CNB, j = q % CNB;
          S.W[i][j] = (i < nb && j < nb && j <= i) ? (i - j <= band ? ldcg(A + bidx(k + i, k + j, band, ldb)) : 0.0)
                                                   : (i == j ? 1.0 : 0.0);
        }
      } else if (blockIdx.x != 0) {
        if (!grid_await(count + 32, pi, err, poll)) return;
        const double* src = Lnext + par * LN;
        for (int q = tid; q < LN; q += blockDim.x) (&S.MT[0][0])[q] = ldcg(src + q);
      }
      __syncthreads();
      if (!own) {
        // every CTA does the same arithmetic, so all agree
        factor_block(S, warp, lane);
        __syncthreads();
        if (blockIdx.x == 0) {
          for (int q = tid; q < CNB * CNB; q += blockDim.x) {
            const int i = q / CNB, j = q % CNB;
            if (i < nb && j <= i && i - j <= band) L[bidx(k + i, k + j, band, ldb)] = S.Ld[i][j] * S.invd[j];
          }
          if (tid == 0 && S.bad) *flag = 1;
        }
      }
    }
    // 2. trailing tiles of the band window
    const bool la = ahead && blockIdx.x == 0 && base < n;  // CTA 0 builds panel k+1's block in S.W
    // factor rows of a diagonal tile (its owner writes them; L is not read here)
    auto write_rows = [&](int i0, int t, int nthr) {
      for (int q = t; q < CNB * CNB; q += nthr) {
        const int r = q / CNB, j = q % CNB, i = i0 + r;
        if (i < lim && j < nb && i - (k + j) <= band) L[bidx(i, k + j, band, ldb)] = S.Pi[j][r];
      }
    };
    int late = -1;  // first row of the diagonal tile whose factor rows are still to be written
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      int ti, tj;
      tile_of(t, ti, tj);
      const int i0 = base + CNB * ti, j0 = base + CNB * tj;
      if (i0 - (j0 + CNB - 1) > band) continue;  // whole tile outside the band (uniform)
      if (t != (int)blockIdx.x) {
        if (late >= 0) write_rows(late, tid, 256);
        late = -1;
        __syncthreads();
        panel_load(A, band, ldb, k, nb, i0, lim, S.Pi, warp, 8, lane);
        if (tj != ti) panel_load(A, band, ldb, k, nb, j0, lim, S.Pj, warp, 8, lane);
        tile_load(i0, j0, lim, a0);
        __syncthreads();
      }
      if (warp == 2) solve_rows(S.Pi, S, lane);
      if (warp == 3 && tj != ti) solve_rows(S.Pj, S, lane);
      __syncthreads();
      double(*Pj)[CNB + 2] = (tj == ti) ? S.Pi : S.Pj;
      if (tj == ti) late = i0;
      double acc[2][2][2] = {};
#pragma unroll 8
      for (int q = 0; q < CNB; ++q) {
        const double2 li = *reinterpret_cast<const double2*>(&S.Pi[q][tr]), lj = *reinterpret_cast<const double2*>(&Pj[q][tc]);
        acc[q & 1][0][0] = fma(li.x, lj.x, acc[q & 1][0][0]);
        acc[q & 1][0][1] = fma(li.x, lj.y, acc[q & 1][0][1]);
        acc[q & 1][1][0] = fma(li.y, lj.x, acc[q & 1][1][0]);
        acc[q & 1][1][1] = fma(li.y, lj.y, acc[q & 1][1][1]);
      }
      const bool blk = la && t == 0;  // tile 0 = panel k+1's diagonal block
      const bool held = pre && t == (int)blockIdx.x;
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int i = i0 + tr + a, j = j0 + tc + b;
          const bool in = i < lim && j < lim && j <= i && i - j <= band;
          const double v = in ? (held ? S.A0[tc + b][tr + a] : a0[a][b]) - (acc[0][a][b] + acc[1][a][b]) : 0.0;
          if (in && !blk) A[bidx(i, j, band, ldb)] = v;  // (the block is factored from W and not read again)
          // band >= 32: every entry of the block on or below the diagonal and
          // below row n is in the window; rows past n are identity-padded
          if (blk) S.W[tr + a][tc + b] = in ? v : ((i >= n && tr + a == tc + b) ? 1.0 : 0.0);
        }
      __syncthreads();
    }
    pre = false;
    if (!la) {
      grid_arrive(count, 1u);  // this CTA's tiles of panel k are written
      if (late >= 0) write_rows(late, tid, 256);
      continue;
    }
    // 3. CTA 0: factor panel k+1's block; beside it arrive, write L, fetch panel k+1's first tile
    const int nb1 = min(CNB, n - base), base1 = base + nb1, lim1 = min(n, base1 + band);
    auto bar47 = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    if (warp >= 4) {
      const int t4 = tid - 128;
      if (t4 == 0) {
        __threadfence();
        atomicAdd(count, 1u);
      }
      if (late >= 0) write_rows(late, t4, 128);
      bar47();  // the rows in Pi are written
      if (t4 == 0) {
        int ok = 1, it = 0;
        while (ld_acquire(count) < (pi + 1) * gridDim.x)
          if (++it > poll) {
            ok = 0;
            atomicExch(err, 1);
            break;
          }
        __threadfence();
        S.ok = ok;
      }
      bar47();
      if (S.ok && base1 < lim1) {
        panel_load(A, band, ldb, base, nb1, base1, lim1, S.Pi, warp - 4, 4, lane);
        for (int q = t4; q < CNB * CNB; q += 128) {
          const int r = q / CNB, c = q % CNB, i = base1 + r, j = base1 + c;
          S.A0[c][r] = (i < lim1 && j <= i && i - j <= band) ? ldcg(A + bidx(i, j, band, ldb)) : 0.0;
        }
      }
    } else {
      factor_block(S, warp, lane);
      asm volatile("bar.sync 2, 128;" ::: "memory");  // warps 0-3: the factor is there
      double* dst = Lnext + (par ^ 1) * LN;
      for (int q = tid; q < LN; q += 128) dst[q] = (&S.MT[0][0])[q];
      if (tid == 0 && S.bad) *flag = 1;
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (tid == 0) {
        __threadfence();
        atomicAdd(count + 32, 1u);
      }
    }
    __syncthreads();
    if (!S.ok) return;
    pre = true;
    if (warp >= 4) {
      for (int q = tid - 128; q < CNB * CNB; q += 128) {
        const int i = q / CNB, j = q % CNB;
        if (i < nb1 && j <= i && i - j <= band) L[bidx(base + i, base + j, band, ldb)] = S.Ld[i][j] * S.invd[j];
      }
    }
  }
}

// ------------------------------------------------------ inverse of L
// Dinv_I = L_II^-1 for every 32x32 diagonal block (identity past n): thread c
// forms column c by forward substitution.
__global__ void __launch_bounds__(CNB) k_diag_inverse(int n, int band, long long ldb, const double* __restrict__ L,
                                                      double* __restrict__ Dinv) {
  __shared__ double Ls[CNB][CNB + 1];
  __shared__ double X[CNB][CNB + 1];
  const int I = blockIdx.x, c = threadIdx.x;
  const long long r0 = (long long)I * CNB;
  for (int r = 0; r < CNB; ++r) {
    const long long i = r0 + r;
    Ls[r][c] = (i < n && c <= r && r - c <= band) ? L[bidx(i, r0 + c, band, ldb)] : (r == c ? 1.0 : 0.0);
  }
  __syncwarp();
  for (int r = 0; r < CNB; ++r) {
    double v = (r == c) ? 1.0 : 0.0;
    for (int q = c; q < r; ++q) v -= Ls[r][q] * X[q][c];
    X[r][c] = r >= c ? v / Ls[r][r] : 0.0;
  }
  __syncwarp();
  for (int r = 0; r < CNB; ++r) Dinv[(long long)I * CNB * CNB + r * CNB + c] = X[r][c];
}

// W_q = L_qq^-1 for every diagonal block q by forward substitution, one strip
// of TWC columns per CTA. Every column is an independent forward substitution
// inside its block, so the strips need no communication: a strip with first
// column j0 walks the 32-row blocks I from the one holding j0 to the end of
// its diagonal block:
//   R    = E - sum_{k in [max(j0, 32I-band), 32I)} L[32I.., k] W[k, strip]
//   W_I  = Dinv_I R                    (E: the identity on these rows/columns)
// Every W read is of rows this CTA wrote in an earlier step (visible after
// __syncthreads). A strip takes (block end - j0)/32 steps; CTA r takes strip
// r/P of block r%P, so the longest strips of all blocks start first. A step
// reads its L rows from L2 (all strips at block row I read the same rows) in
// 64-wide chunks, the next chunk prefetched into registers. Warp w takes the
// chunk columns k = w, w+8, ...; lane l keeps rows l%16 and l%16+16 of half
// the strip's columns (6 shared loads per 16 FMA, no bank conflicts); the 8
// warp partials are summed through shared memory. The step's diagonal inverse
// is fetched at its start. W_q goes to W64 (lower part, FP64) and to the
// apply matrix (C64 or C32) as W_q in the lower triangle and W_q^T in the
// strict upper triangle of the block's columns 0 .. m-1.
constexpr int TIT = 256, TKC = 64, TWC = 16;
struct TriSmem {
  double Ls[CNB][TKC + 1];
  double Wc[TKC][TWC];
  double red[TIT / 32][CNB][TWC + 1];
  double Rs[CNB][TWC + 1];
  double Ds[CNB][CNB + 1];
};

__global__ void __launch_bounds__(TIT) k_tri_inverse(int n, int band, long long ldb, const double* __restrict__ L,
                                                     const double* __restrict__ Dinv, CoarseBlocks bk, double* W64,
                                                     double* C64, float* C32) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TriSmem& S = *reinterpret_cast<TriSmem*>(smem_raw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int blk = (int)blockIdx.x % bk.P;
  const int b0 = bk.b[blk], iend = bk.b[blk + 1];
  const int j0 = b0 + ((int)blockIdx.x / bk.P) * TWC;
  if (j0 >= iend) return;  // uniform over the CTA
  const int nT = (iend + CNB - 1) / CNB;
  const long long ld = bk.ld[blk];
  double* Wq = W64 + bk.off[blk];
  double* C64q = C64 != nullptr ? C64 + bk.off[blk] : nullptr;
  float* C32q = C32 != nullptr ? C32 + bk.off[blk] : nullptr;
  constexpr int PL = CNB * TKC / TIT;  // L values fetched per thread per chunk
  constexpr int PW = TKC * TWC / TIT;  // W values fetched per thread per chunk
  constexpr int PO = CNB * TWC / TIT;  // outputs per thread per step
  static_assert(PL * TIT == CNB * TKC && PW * TIT == TKC * TWC && PO * TIT == CNB * TWC, "tile split");
  // lane mapping of the partial product: rows rl and rl+16, columns ch .. ch+TWC/2
  const int rl = lane & 15, ch = (lane >> 4) * (TWC / 2);
  double pl[PL], pw[PW];
  double dpre[CNB * CNB / TIT];
  for (int I = j0 / CNB; I < nT; ++I) {
    const int i0 = I * CNB;
    const int klo = max(j0, i0 - band);
#pragma unroll
    for (int m = 0; m < CNB * CNB / TIT; ++m) dpre[m] = Dinv[(long long)I * CNB * CNB + t + TIT * m];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int m = 0; m < PL; ++m) {
        const int q = t + TIT * m;
        const int i = i0 + q / TKC, k = k0 + q % TKC;
        pl[m] = (i < n && k < i0 && i - k <= band) ? L[bidx(i, k, band, ldb)] : 0.0;
      }
#pragma unroll
      for (int m = 0; m < PW; ++m) {
        const int q = t + TIT * m;
        const int kw = k0 + q / TWC, cw = j0 + q % TWC;
        pw[m] = (kw < i0 && cw < iend && cw <= kw) ? Wq[(long long)(kw - b0) * ld + (cw - b0)] : 0.0;
      }
    };
    double acc[TWC];
#pragma unroll
    for (int c = 0; c < TWC; ++c) acc[c] = 0.0;
    if (klo < i0) fetch(klo);
    for (int k0 = klo; k0 < i0; k0 += TKC) {
      __syncthreads();
#pragma unroll
      for (int m = 0; m < PL; ++m) {
        const int q = t + TIT * m;
        S.Ls[q / TKC][q % TKC] = pl[m];
      }
#pragma unroll
      for (int m = 0; m < PW; ++m) {
        const int q = t + TIT * m;
        S.Wc[q / TWC][q % TWC] = pw[m];
      }
      __syncthreads();
      if (k0 + TKC < i0) fetch(k0 + TKC);
#pragma unroll 4
      for (int m = 0; m < TKC / 8; ++m) {
        const int kk = warp + 8 * m;
        const double a0 = S.Ls[rl][kk], a1 = S.Ls[rl + 16][kk];
        const double2* wr = reinterpret_cast<const double2*>(&S.Wc[kk][ch]);
#pragma unroll
        for (int c2 = 0; c2 < TWC / 4; ++c2) {
          const double2 w = wr[c2];
          acc[2 * c2] = fma(a0, w.x, acc[2 * c2]);
          acc[2 * c2 + 1] = fma(a0, w.y, acc[2 * c2 + 1]);
          acc[TWC / 2 + 2 * c2] = fma(a1, w.x, acc[TWC / 2 + 2 * c2]);
          acc[TWC / 2 + 2 * c2 + 1] = fma(a1, w.y, acc[TWC / 2 + 2 * c2 + 1]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < TWC / 2; ++c) {
      S.red[warp][rl][ch + c] = acc[c];
      S.red[warp][rl + 16][ch + c] = acc[TWC / 2 + c];
    }
#pragma unroll
    for (int m = 0; m < CNB * CNB / TIT; ++m) {
      const int q = t + TIT * m;
      S.Ds[q >> 5][q & 31] = dpre[m];
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PO; ++p) {
      const int q = t + TIT * p;
      const int r = q / TWC, c = q % TWC;
      double v = (i0 + r == j0 + c) ? 1.0 : 0.0;
#pragma unroll
      for (int w = 0; w < TIT / 32; ++w) v -= S.red[w][r][c];
      S.Rs[r][c] = v;
    }
    __syncthreads();
    double wv[PO];
#pragma unroll
    for (int p = 0; p < PO; ++p) {
      const int q = t + TIT * p;
      const int r = q / TWC, c = q % TWC;
      double v = 0.0;
      for (int m = 0; m <= r; ++m) v = fma(S.Ds[r][m], S.Rs[m][c], v);
      wv[p] = v;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PO; ++p) {
      const int q = t + TIT * p;
      const int r = q / TWC, c = q % TWC;
      const int i = i0 + r, col = j0 + c;
      S.Rs[r][c] = wv[p];
      if (i < iend && col < iend && col <= i) {
        const long long a = (long long)(i - b0) * ld + (col - b0);
        Wq[a] = wv[p];
        if (C64q != nullptr && C64q != Wq) C64q[a] = wv[p];
        if (C32q != nullptr) C32q[a] = (float)wv[p];
      }
    }
    __syncthreads();
    // transposed copy: rows j0 .. j0+TWC-1 of the upper triangle, columns i0 .. i0+31
    for (int e = t; e < TWC * CNB; e += TIT) {
      const int cr = j0 + e / CNB, ic = i0 + e % CNB;
      if (cr < iend && ic < iend && ic > cr) {
        const double v = S.Rs[e % CNB][e / CNB];
        const long long a = (long long)(cr - b0) * ld + (ic - b0);
        if (C64q != nullptr) C64q[a] = v;
        if (C32q != nullptr) C32q[a] = (float)v;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------- couplings between the blocks
// With the block-bidiagonal L (diagonal blocks L_qq, corners Lc_q = the rows
// b[q] .. b[q]+band-1 of L over the columns b[q]-band .. b[q]-1), the two
// triangular solves of K^-1 r become, block by block,
//   y_q = W_q r_q - G_q y_{q-1}[m_{q-1}-band ..],   G_q = W_q[:, 0:band] Lc_q
//   z_q = W_q^T y_q - H_q z_{q+1}[0 .. band),       H_q = (Lc_{q+1} W_q[m-band.., :])^T
// k_couplings forms G_q (q >= 1) and H_q (q < P-1) in FP64 from W64 and L:
// one CTA per 64 x 32 output tile, 16-wide l chunks staged in shared memory,
// each thread 2 rows x 4 columns. Lc_q[l][k] is non-zero for l <= k only and
// W_q is lower triangular, so a tile's l range is clipped to where both are.
constexpr int GTI = 64, GTK = 32, GTL = 16;
__global__ void __launch_bounds__(256) k_couplings(int band, long long ldb, const double* __restrict__ L,
                                                   CoarseBlocks bk, const double* W64, double* C64, float* C32) {
  __shared__ __align__(16) double As[GTL][GTI + 2];
  __shared__ __align__(16) double Bs[GTL][GTK + 2];
  const int q = (int)blockIdx.y >> 1, type = (int)blockIdx.y & 1;  // type 0: G_q, 1: H_q
  if (q >= bk.P || (type == 0 && q == 0) || (type == 1 && q == bk.P - 1)) return;
  const int m = bk.b[q + 1] - bk.b[q];
  const int nkt = (band + GTK - 1) / GTK;
  const int i0 = ((int)blockIdx.x / nkt) * GTI, k0 = ((int)blockIdx.x % nkt) * GTK;
  if (i0 >= m) return;
  const long long ld = bk.ld[q];
  const double* Wq = W64 + bk.off[q];
  // rows of L holding the corner: G_q uses block q's, H_q block q+1's
  const long long cb = type == 0 ? bk.b[q] : bk.b[q + 1];
  int lo, hi;
  if (type == 0) {  // l <= k and l <= i
    lo = 0;
    hi = min(band, min(k0 + GTK, i0 + GTI));
  } else {          // l >= k and m-band+l >= i
    lo = max(k0, i0 - (m - band));
    lo = max(lo, 0);
    hi = band;
  }
  const int t = threadIdx.x, tx = t & 7, ty = t >> 3;  // columns 4tx.., rows 2ty, 2ty+1
  double acc[2][4] = {};
  for (int l0 = lo; l0 < hi; l0 += GTL) {
    __syncthreads();
    // A(i, l): G: W_q[i][l]; H: W_q[m-band+l][i]
#pragma unroll
    for (int u = 0; u < GTI * GTL / 256; ++u) {
      const int e = t + 256 * u;
      int il, ll;
      if (type == 0) { ll = e % GTL; il = e / GTL; }   // l fastest: a row of W_q
      else { il = e % GTI; ll = e / GTI; }             // i fastest: a row of W_q
      const int i = i0 + il, l = l0 + ll;
      double v = 0.0;
      if (i < m && l < hi) {
        if (type == 0) { if (l <= i) v = Wq[(long long)i * ld + l]; }
        else { const int r = m - band + l; if (r >= i) v = Wq[(long long)r * ld + i]; }
      }
      As[ll][il] = v;
    }
    // B(l, k): G: Lc_q[l][k] = L[cb+l][cb-band+k]; H: Lc_{q+1}[k][l] = L[cb+k][cb-band+l]
#pragma unroll
    for (int u = 0; u < GTK * GTL / 256; ++u) {
      const int e = t + 256 * u;
      int kl, ll;
      if (type == 0) { kl = e % GTK; ll = e / GTK; }
      else { ll = e % GTL; kl = e / GTL; }
      const int k = k0 + kl, l = l0 + ll;
      double v = 0.0;
      if (k < band && l < hi) {
        if (type == 0) { if (l <= k) v = L[bidx(cb + l, cb - band + k, band, ldb)]; }
        else { if (k <= l) v = L[bidx(cb + k, cb - band + l, band, ldb)]; }
      }
      Bs[ll][kl] = v;
    }
    __syncthreads();
    const int lend = min(GTL, hi - l0);
    for (int ll = 0; ll < lend; ++ll) {
      const double2 a = *reinterpret_cast<const double2*>(&As[ll][2 * ty]);
      const double2 b01 = *reinterpret_cast<const double2*>(&Bs[ll][4 * tx]);
      const double2 b23 = *reinterpret_cast<const double2*>(&Bs[ll][4 * tx + 2]);
      const double b[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc[0][c] = fma(a.x, b[c], acc[0][c]);
        acc[1][c] = fma(a.y, b[c], acc[1][c]);
      }
    }
  }
  const int col0 = (type == 0 ? bk.gofs[q] : bk.hofs[q]) + k0 + 4 * tx;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int i = i0 + 2 * ty + r;
    if (i >= m) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (k0 + 4 * tx + c >= band) continue;
      const long long a = bk.off[q] + (long long)i * ld + col0 + c;
      if (C64 != nullptr) C64[a] = acc[r][c];
      if (C32 != nullptr) C32[a] = (float)acc[r][c];
    }
  }
}

// --------------------------------------------------------------- apply
// z = K^-1 r block by block: the lower pass for q = 0 .. P-1 forms
// y_q = W_q r_q - G_q y_{q-1}[tail] (row i reads C_q[i][0..i] and G_q[i]), the
// upper pass for q = P-1 .. 0 forms z_q = W_q^T y_q - H_q z_{q+1}[head] (row i
// reads C_q[i][i..m-1] and H_q[i]) and scatters it to the free DoFs. Each row
// is split over RW warps (interleaved 32-lane chunks of 16-byte loads; row
// strides and segment starts are multiples of 32 elements, so every segment
// starts 16-byte aligned), FP64 accumulation, the RW partial sums added
// through shared memory. With four warps per row one block
// (about 4 band rows) is a single short wave, so the 2P dependent launches of
// an apply cost about 5 us each. The restriction to the coarsest level writes
// the compact right-hand side; both passes read the compact vectors through L1 (plain loads: the kernels of
// a chain overlap, so nothing that one of them writes is read with __ldg).
constexpr int RW = 4;  // warps per row

// One warp's share of sum_{j in [lo, hi)} Ci[j] v[j] over a row segment:
// chunks c = sub, sub+RW, ... of 32 lanes x one 16-byte load, four chunks in
// flight. Every load begins below hi at a multiple of V and every segment
// (W_q: m columns, G_q and H_q: band columns) is padded to a multiple of 32,
// so none leaves its segment; entries outside [lo, hi) are not used.
template <typename TX>
__device__ __forceinline__ double seg_dot(const TX* __restrict__ Ci, const double* v, int lo, int hi,
                                          int lane, int sub) {
  constexpr int V = 16 / sizeof(TX);
  constexpr int STEP = RW * 32 * V;
  constexpr int U = 4;
  double acc = 0.0;
  int j = (lo / V) * V + (sub * 32 + lane) * V;
  for (; j + (U - 1) * STEP < hi; j += U * STEP) {
    TX w[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u) *reinterpret_cast<uint4*>(w[u]) = __ldg(reinterpret_cast<const uint4*>(Ci + j + u * STEP));
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const int jj = j + u * STEP + q;
        if (jj >= lo && jj < hi) acc += (double)w[u][q] * v[jj];
      }
  }
  for (; j < hi; j += STEP) {
    TX w[V];
    *reinterpret_cast<uint4*>(w) = __ldg(reinterpret_cast<const uint4*>(Ci + j));
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const int jj = j + q;
      if (jj >= lo && jj < hi) acc += (double)w[q] * v[jj];
    }
  }
  return acc;
}

// Sum of the RW warp partials of each row of the CTA (every thread calls it).
__device__ __forceinline__ double row_sum(double acc, int warp, int lane) {
  __shared__ double part[8];
  acc = warp_sum(acc);
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  double t = 0.0;
  if (warp % RW == 0)
#pragma unroll
    for (int k = 0; k < RW; ++k) t += part[warp + k];
  return t;
}

// pass one, block q (rows b0 .. b0+m-1): y_q = W_q r_q - G_q y_{q-1}[m_{q-1}-band ..]
template <typename TX>
__global__ void __launch_bounds__(256) k_coarse_lower(int m, int b0, long long ld, int gofs, int band, int prev,
                                                      const TX* __restrict__ Cq, const double* rc,
                                                      double* y, const KrylovState* st, long long vswork) {
  chain_enter();
  if (st != nullptr && st->done) return;  // uniform over the grid
  rc += blockIdx.y * vswork;              // column
  y += blockIdx.y * vswork;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = (int)blockIdx.x * (8 / RW) + warp / RW, sub = warp % RW;
  const bool live = row < m;
  double acc = 0.0;
  if (live) {
    const TX* Ci = Cq + (long long)row * ld;
    acc = seg_dot(Ci, rc + b0, 0, row + 1, lane, sub);
    if (prev) acc -= seg_dot(Ci + gofs, y + (b0 - band), 0, band, lane, sub);
  }
  acc = row_sum(acc, warp, lane);
  if (live && sub == 0 && lane == 0) y[b0 + row] = acc;
}

// pass two, block q: z_q = W_q^T y_q - H_q z_{q+1}[0 .. band), kept compact in
// z and scattered to the free DoFs of x
template <typename T, typename TX>
__global__ void __launch_bounds__(256) k_coarse_upper(int m, int b0, long long ld, int hofs, int band, int next,
                                                      long long nfull, const TX* __restrict__ Cq,
                                                      const int* __restrict__ free_list, const double* y, double* z,
                                                      T* x, const KrylovState* st, long long vswork,
                                                      long long vsx) {
  chain_enter();
  if (st != nullptr && st->done) return;  // uniform over the grid
  y += blockIdx.y * vswork;               // column
  z += blockIdx.y * vswork;
  x += blockIdx.y * vsx;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = (int)blockIdx.x * (8 / RW) + warp / RW, sub = warp % RW;
  const bool live = row < m;
  double acc = 0.0;
  if (live) {
    const TX* Ci = Cq + (long long)row * ld;
    acc = seg_dot(Ci, y + b0, row, m, lane, sub);
    if (next) acc -= seg_dot(Ci + hofs, z + (b0 + m), 0, band, lane, sub);
  }
  acc = row_sum(acc, warp, lane);
  if (live && sub == 0 && lane == 0) {
    z[b0 + row] = acc;
    const int f = free_list[b0 + row];
    if (topo_in_range(f, nfull)) x[f] = (T)acc;
  }
}

}  // namespace cst

// ================================================================ host side
CoarsestPlan coarsest_plan(const Grid& g, const std::vector<int>& free_list) {
  CoarsestPlan p;
  p.n = (int)free_list.size();
  p.nfull = g.ndof;
  p.nt = (p.n + cst::CNB - 1) / cst::CNB;
  return p;
}

void coarsest_alloc(CoarsestFactor& f, const CoarsestPlan& p, int band, bool f64, void* (*alloc_bytes)(void*, size_t),
                    void* ctx) {
  auto A = [&](size_t bytes) { return alloc_bytes(ctx, bytes); };
  f.band = band;
  f.ldb = band + 1;
  f.f64 = f64;
  const int n = std::max(p.n, 1);
  const size_t nbs = (size_t)n * f.ldb;
  f.A = (double*)A(nbs * sizeof(double));
  f.L = (double*)A(nbs * sizeof(double));
  f.Dinv = (double*)A((size_t)std::max(p.nt, 1) * cst::CNB * cst::CNB * sizeof(double));
  f.Lnext = (double*)A(2 * (size_t)cst::LN * sizeof(double));
  // diagonal blocks of W: at least max(4 band, 512) rows each (every block at
  // least `band` rows), boundaries on 32-row panels
  CoarseBlocks& bk = f.blk;
  int P = std::max(1, std::min(COARSE_MAXB, n / std::max(4 * band, 512)));
  for (;;) {
    bk.P = P;
    bk.b[0] = 0;
    for (int q = 1; q < P; ++q) bk.b[q] = (int)((long long)q * n / P / cst::CNB * cst::CNB);
    bk.b[P] = n;
    bool ok = true;
    for (int q = 0; q < P; ++q) ok = ok && bk.b[q + 1] - bk.b[q] >= std::max(band, 1);
    if (ok || P == 1) break;
    --P;
  }
  const long long bandp = ((long long)band + 31) / 32 * 32;
  long long off = 0;
  int maxm = 0;
  for (int q = 0; q < bk.P; ++q) {
    const int m = bk.b[q + 1] - bk.b[q];
    maxm = std::max(maxm, m);
    bk.gofs[q] = (m + 31) / 32 * 32;
    bk.hofs[q] = (int)(bk.gofs[q] + bandp);
    bk.ld[q] = bk.gofs[q] + (bk.P > 1 ? 2 * bandp : 0);
    bk.off[q] = off;
    off += (long long)m * bk.ld[q];
  }
  f.strips_per_block = (maxm + cst::TWC - 1) / cst::TWC;
  f.W64 = (double*)A((size_t)off * sizeof(double));
  f.C = f64 ? (void*)f.W64 : A((size_t)off * sizeof(float));
  f.flag = (int*)A(sizeof(int) * 4);
  f.bar = (unsigned*)A(sizeof(unsigned) * 64);  // the two counters in lines of their own
  f.err = f.flag + 1;
  // persistent factorisation: cooperative grid sized by co-residency
  int dev = 0, nsm = 0, per_sm = 0;
  TOPO_CUDA_CHECK(cudaGetDevice(&dev));
  TOPO_CUDA_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  TOPO_CUDA_CHECK(cudaFuncSetAttribute(cst::k_band_chol, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(cst::CholSmem)));
  TOPO_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cst::k_band_chol, 256, sizeof(cst::CholSmem)));
  const int tiles_max = ((band + cst::CNB - 1) / cst::CNB) * ((band + cst::CNB - 1) / cst::CNB + 1) / 2;
  f.chol_grid = std::max(1, std::min(std::min(nsm * std::max(per_sm, 1), nsm), std::max(tiles_max, 1)));
  TOPO_CUDA_CHECK(cudaFuncSetAttribute(cst::k_tri_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(cst::TriSmem)));
  f.plan = p;
}

void pivot_recip(long long n, const double* d, double* r, cudaStream_t s) {
  cst::k_recip<<<(unsigned)std::min<long long>((n + 255) / 256, 1184), 256, 0, s>>>(n, d, r);
  TOPO_LAUNCH_CHECK();
}

void coarsest_assemble(CoarsestFactor& f, const Grid& g, const double* S, const int* dof_index, cudaStream_t s) {
  TOPO_CUDA_CHECK(cudaMemsetAsync(f.A, 0, sizeof(double) * (size_t)std::max(f.plan.n, 1) * f.ldb, s));
  const int bs = 128;
  cst::k_band_assemble<<<dim3((unsigned)((g.nnodes + bs - 1) / bs), 27), bs, 0, s>>>(g, S, dof_index, f.band, f.ldb, f.A);
  TOPO_LAUNCH_CHECK();
}

void coarsest_regularise(CoarsestFactor& f, double* dtmp, cudaStream_t s) {
  const int n = f.plan.n;
  cst::k_band_diag_sum<<<1, 256, 0, s>>>(n, f.band, f.ldb, f.A, dtmp);
  TOPO_LAUNCH_CHECK();
  double dsum = 0.0;
  TOPO_CUDA_CHECK(cudaMemcpyAsync(&dsum, dtmp, sizeof(double), cudaMemcpyDeviceToHost, s));
  TOPO_CUDA_CHECK(cudaStreamSynchronize(s));
  const double eps = std::max(dsum / n * 1e-8, 1e-14);
  cst::k_band_add_diag<<<(n + 255) / 256, 256, 0, s>>>(n, f.band, f.ldb, f.A, eps);
  TOPO_LAUNCH_CHECK();
}

void coarsest_factor(CoarsestFactor& f, cudaStream_t s) {
  const CoarsestPlan& p = f.plan;
  const int n = p.n;
  if (n == 0) return;
  TOPO_CUDA_CHECK(cudaMemsetAsync(f.flag, 0, sizeof(int) * 4, s));
  TOPO_CUDA_CHECK(cudaMemsetAsync(f.bar, 0, sizeof(unsigned) * 64, s));
  TOPO_CUDA_CHECK(cudaMemsetAsync(f.L, 0, sizeof(double) * (size_t)n * f.ldb, s));
  {
    int nn = n, band = f.band;
    long long ldb = f.ldb;
    double* A = f.A;
    double* L = f.L;
    double* Ln = f.Lnext;
    int* flag = f.flag;
    unsigned* cnt = f.bar;
    int* err = f.err;
    int poll = 1 << 24;
    void* args[] = {&nn, &band, &ldb, &A, &L, &Ln, &flag, &cnt, &err, &poll};
    TOPO_CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)cst::k_band_chol, dim3(f.chol_grid), dim3(256), args,
                                                sizeof(cst::CholSmem), s));
    count_launches(1);
  }
  cst::k_diag_inverse<<<p.nt, cst::CNB, 0, s>>>(n, f.band, f.ldb, f.L, f.Dinv);
  TOPO_LAUNCH_CHECK();
  const CoarseBlocks& bk = f.blk;
  double* C64 = f.f64 ? f.W64 : nullptr;
  float* C32 = f.f64 ? nullptr : (float*)f.C;
  cst::k_tri_inverse<<<(unsigned)(bk.P * f.strips_per_block), cst::TIT, sizeof(cst::TriSmem), s>>>(
      n, f.band, f.ldb, f.L, f.Dinv, bk, f.W64, C64, C32);
  TOPO_LAUNCH_CHECK();
  if (bk.P > 1) {
    int maxm = 0;
    for (int q = 0; q < bk.P; ++q) maxm = std::max(maxm, bk.b[q + 1] - bk.b[q]);
    const int nkt = (f.band + cst::GTK - 1) / cst::GTK;
    const dim3 grid((unsigned)(((maxm + cst::GTI - 1) / cst::GTI) * nkt), (unsigned)(2 * bk.P));
    cst::k_couplings<<<grid, 256, 0, s>>>(f.band, f.ldb, f.L, bk, f.W64, C64, C32);
    TOPO_LAUNCH_CHECK();
  }
}

// Returns the non-positive-pivot flag (1) or a barrier timeout (< 0).
int coarsest_status(CoarsestFactor& f, cudaStream_t s) {
  int h[2] = {0, 0};
  TOPO_CUDA_CHECK(cudaMemcpyAsync(h, f.flag, sizeof(h), cudaMemcpyDeviceToHost, s));
  TOPO_CUDA_CHECK(cudaStreamSynchronize(s));
  if (h[1]) return -1;
  return h[0] ? 1 : 0;
}

// work: 2n doubles (y, then the compact right-hand side, overwritten by the
// compact solution in the second pass). Only the free DoFs of x are written.
template <typename T, typename TX>
static void apply_blocks(const CoarsestFactor& f, double* work, T* x, const KrylovState* st, cudaStream_t s, int nv,
                         long long vswork, long long vsx) {
  const CoarsestPlan& p = f.plan;
  const CoarseBlocks& bk = f.blk;
  const int n = p.n;
  constexpr int rpb = 8 / cst::RW;  // rows per 256-thread CTA
  double* y = work;
  double* rc = work + n;
  const TX* C = (const TX*)f.C;
  for (int q = 0; q < bk.P; ++q) {
    const int m = bk.b[q + 1] - bk.b[q];
    launch_chained(cst::k_coarse_lower<TX>, dim3((unsigned)((m + rpb - 1) / rpb), (unsigned)nv), 256, 0, s, m, bk.b[q], bk.ld[q], bk.gofs[q], f.band, (int)(q > 0), C + bk.off[q], rc, y, st, vswork);
  }
  for (int q = bk.P - 1; q >= 0; --q) {
    const int m = bk.b[q + 1] - bk.b[q];
    launch_chained(cst::k_coarse_upper<T, TX>, dim3((unsigned)((m + rpb - 1) / rpb), (unsigned)nv), 256, 0, s, m, bk.b[q], bk.ld[q], bk.hofs[q], f.band, (int)(q < bk.P - 1), p.nfull, C + bk.off[q], f.d_free, y, rc, x, st, vswork, vsx);
  }
}

void coarsest_apply(const CoarsestFactor& f, bool vec64, double* work, void* x, const KrylovState* st, cudaStream_t s, int nv,
                    long long vswork, long long vsx) {
  if (f.plan.n == 0) return;
  if (vec64) {
    if (!f.f64) throw std::runtime_error("coarsest apply: FP64 vectors need the FP64 inverse");
    apply_blocks<double, double>(f, work, (double*)x, st, s, nv, vswork, vsx);
  } else if (f.f64) {
    apply_blocks<float, double>(f, work, (float*)x, st, s, nv, vswork, vsx);
  } else {
    apply_blocks<float, float>(f, work, (float*)x, st, s, nv, vswork, vsx);
  }
}

TOPO_BOUNDS_READER(bounds_flag_coarsest)

}  // namespace topo
