// coarse.cu - coarse multigrid levels on 27-point block stencils.
//
// Every coarse operator of the hierarchy is stored as a structured stencil:
// for node n and neighbour offset k = (dx+1)*9+(dy+1)*3+(dz+1), the 3x3 block
// coupling n to n+(dx,dy,dz) sits at S[(k*9 + c*3 + d) * nnodes + n]
// (coefficient-major, so consecutive threads read consecutive addresses).
// Rows and columns of fixed DoFs are zero. This replaces the reference's CSR
// matrices on compact free-DoF vectors (src/gpu_fem/multigrid_v4.py:132-270,
// 747-772) with no index arrays at all.
#include "internal.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <stdexcept>
#include <vector>

namespace topo {

__constant__ double cQ[8 * 576];  // Q_stu = P24_stu^T KE P24_stu, stu = 4s+2t+u

void set_galerkin_q(const double* Q) { TOPO_CUDA_CHECK(cudaMemcpyToSymbol(cQ, Q, sizeof(double) * 8 * 576)); }

__host__ __device__ constexpr int corner_of(int bx, int by, int bz) {
  return bz * 4 + (by ? (bx ? 2 : 3) : (bx ? 1 : 0));
}

__device__ __forceinline__ void node_xyz(const Grid& g, long long n, int& ix, int& iy, int& iz) {
  if (g.nnodes < (1LL << 31)) {  // 32-bit division
    const unsigned u = (unsigned)n, r = u / (unsigned)g.NZ;
    iz = (int)(u - r * (unsigned)g.NZ);
    ix = (int)(r / (unsigned)g.NY);
    iy = (int)(r - (unsigned)ix * (unsigned)g.NY);
    return;
  }
  iz = (int)(n % g.NZ);
  iy = (int)((n / g.NZ) % g.NY);
  ix = (int)(n / ((long long)g.NZ * g.NY));
}

// ------------------------------------------------------------ level-1 Galerkin
// Coarse element e contributes Kc_e = sum_stu E_f(2e+stu, clamped) Q_stu
// (multigrid_v4.py:182-203, 256). One thread per (coarse node I, neighbour
// J = I + delta) gathers the 3x3 block sum over the coarse elements that
// contain both. The offset k is uniform over a CTA (blockIdx.y): the at most
// 64 blocks Q_stu[a][m] it needs sit in shared memory, and a thread forms its
// block for L1N nodes, so that a (broadcast) load feeds L1N multiply-adds.
// Bound by the 627 M FP64 multiply-adds at 160x80x80 (35 us). There: a node's
// 27 blocks as one thread's loop over constant memory 324 us, one thread per
// block 280 us, now 222 us.
constexpr int L1T = 128, L1N = 2;
__global__ void __launch_bounds__(L1T) k_level1_assemble(Grid f, Grid c, const double* __restrict__ Ef,
                                                         const uint8_t* __restrict__ mc, double* __restrict__ S) {
  __shared__ __align__(16) double qs[64][10];  // [o * 8 + stu][3 cc + dd]
  const int k = blockIdx.y;
  const int dx = k / 9 - 1, dy = (k / 3) % 3 - 1, dz = k % 3 - 1;
  for (int i = threadIdx.x; i < 64 * 9; i += L1T) {
    const int os = i / 9, q = i % 9, o = os >> 3;
    const int ox = (o >> 2) - 1, oy = ((o >> 1) & 1) - 1, oz = (o & 1) - 1;
    const int mx = dx - ox, my = dy - oy, mz = dz - oz;
    if (mx < 0 || mx > 1 || my < 0 || my > 1 || mz < 0 || mz > 1) continue;
    qs[os][q] = cQ[(os & 7) * 576 + (3 * corner_of(-ox, -oy, -oz) + q / 3) * 24 + 3 * corner_of(mx, my, mz) + q % 3];
  }
  __syncthreads();
  long long I[L1N];
  int ix[L1N], iy[L1N], iz[L1N];
  bool in[L1N], jin[L1N];
  double B[L1N][9];
#pragma unroll
  for (int n = 0; n < L1N; ++n) {
    I[n] = (blockIdx.x * (long long)L1N + n) * L1T + threadIdx.x;
    in[n] = I[n] < c.nnodes;
    node_xyz(c, in[n] ? I[n] : 0, ix[n], iy[n], iz[n]);
    const int jx = ix[n] + dx, jy = iy[n] + dy, jz = iz[n] + dz;
    jin[n] = in[n] && jx >= 0 && jx < c.NX && jy >= 0 && jy < c.NY && jz >= 0 && jz < c.NZ;
#pragma unroll
    for (int q = 0; q < 9; ++q) B[n][q] = 0.0;
  }
  for (int o = 0; o < 8; ++o) {
    const int ox = (o >> 2) - 1, oy = ((o >> 1) & 1) - 1, oz = (o & 1) - 1;
    const int mx = dx - ox, my = dy - oy, mz = dz - oz;
    if (mx < 0 || mx > 1 || my < 0 || my > 1 || mz < 0 || mz > 1) continue;  // uniform
    double Ee[L1N][8];
#pragma unroll
    for (int n = 0; n < L1N; ++n) {
      const int ex = ix[n] + ox, ey = iy[n] + oy, ez = iz[n] + oz;
      const bool e = jin[n] && ex >= 0 && ex < c.nx && ey >= 0 && ey < c.ny && ez >= 0 && ez < c.nz;
#pragma unroll
      for (int stu = 0; stu < 8; ++stu) {
        const int fx = min(2 * ex + (stu >> 2), f.nx - 1), fy = min(2 * ey + ((stu >> 1) & 1), f.ny - 1),
                  fz = min(2 * ez + (stu & 1), f.nz - 1);
        Ee[n][stu] = e ? Ef[((long long)fx * f.ny + fy) * f.nz + fz] : 0.0;
      }
    }
#pragma unroll
    for (int stu = 0; stu < 8; ++stu) {
      const double* Q = qs[o * 8 + stu];
      double qv[9];
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        const double2 v = *reinterpret_cast<const double2*>(Q + q);
        qv[q] = v.x;
        qv[q + 1] = v.y;
      }
      qv[8] = Q[8];
#pragma unroll
      for (int n = 0; n < L1N; ++n)
#pragma unroll
        for (int q = 0; q < 9; ++q) B[n][q] += Ee[n][stu] * qv[q];
    }
  }
#pragma unroll
  for (int n = 0; n < L1N; ++n) {
    if (!in[n]) continue;
    const long long J = jin[n] ? (((long long)(ix[n] + dx) * c.NY + iy[n] + dy) * c.NZ + iz[n] + dz) : 0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const bool keep = jin[n] && mc[3 * I[n] + q / 3] && mc[3 * J + q % 3];
      S[(long long)(k * 9 + q) * c.nnodes + I[n]] = keep ? B[n][q] : 0.0;
    }
  }
}

void level1_assemble(const Grid& fine, const Grid& coarse, const double* E_f, const uint8_t* mask_c, double* S,
                     cudaStream_t s) {
  const int bs = L1T * L1N;
  k_level1_assemble<<<dim3((unsigned)((coarse.nnodes + bs - 1) / bs), 27), L1T, 0, s>>>(fine, coarse, E_f, mask_c, S);
  TOPO_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------- R.A.P
// K_c = P^T K_f P with the row-normalised trilinear P restricted to free DoFs
// (multigrid_v4.py:747-751). P is a product of one-dimensional prolongations,
// and a 27-point stencil stays one under each of them, so the product is formed
// in three passes, coarsening z, then y, then x. Along the coarsened dimension
// block (I, J = I + d) sums over the fine pairs i = 2I + s, j = i + e
// (s, e in {-1,0,1}): node 2I is I's own; 2I+1 belongs to I with weight a and
// to I+1 with 1/2 (a = 1/2, or 1 where I+1 lies beyond the coarse grid); 2I-1
// to I-1 and I with 1/2 each. Nine reads give the three blocks d = -1, 0, 1.
// One thread per (output node, coefficient of the other two dimensions and of
// the 3x3 block), lanes along z. Couplings to neighbours outside a grid are
// zero in the input and written as zero. Bound by HBM: level 1 of 160x80x80
// is read once (265 MB) and the passes write 136, 69 and 35 MB. The direct form
// (one thread per block over up to 343 pairs) took 1500 us for both levels of
// that hierarchy, the passes 152 us.
struct RapDim {
  int nf, nc;            // fine / coarse elements along the dimension
  long long inner;       // nodes below it (stride of the dimension)
  long long outer;       // nodes above it
  int kstride;           // step of the dimension's offset in k: 9, 3 or 1
  long long sin, sout;   // nodes between two coefficients of the input / output
  int i0, ni;            // the output's first node along the dimension and its number of them
  int f0, nfs;           // the input's
  long long at;          // node of the first output in the coarse grid (last pass)
};

template <bool MASK>
__global__ void __launch_bounds__(256) k_rap_dim(RapDim D, const double* __restrict__ Sin, double* __restrict__ Sout, Grid c,
                                                 const uint8_t* __restrict__ mc) {
  const long long nin = D.sin, nout = D.outer * D.ni * D.inner;
  const long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (o >= nout) return;
  const int cq = blockIdx.y;  // (other two offsets) * 9 + coefficient
  const int q = cq % 9, kk = cq / 9;
  // k of the middle block (offset 0 along the dimension)
  const int k0 = D.kstride == 1 ? kk * 3 + 1 : D.kstride == 3 ? (kk / 3) * 9 + 3 + kk % 3 : 9 + kk;
  const long long in_ = o % D.inner, t = o / D.inner;
  const int I = D.i0 + (int)(t % D.ni);
  const long long out_ = t / D.ni;
  const double* base = Sin + (long long)(k0 * 9 + q) * nin + (out_ * D.nfs + 2 * I - D.f0) * D.inner + in_;
  const long long ks = (long long)D.kstride * 9 * nin;
  const bool h = I + 1 <= D.nc, up = 2 * I + 1 <= D.nf, dn = I >= 1;
  const double a = h ? 0.5 : 1.0;
  double m0 = 0.0, mp = 0.0, mm = 0.0, p0 = 0.0, pp = 0.0, pm = 0.0, d0 = 0.0, dp = 0.0, dm = 0.0;
  if (2 * I <= D.nf) {  // (one fine element: nodes 0 and 1 only)
    m0 = __ldg(base);
    mp = __ldg(base + ks);
    mm = __ldg(base - ks);
  }
  if (up) {
    p0 = __ldg(base + D.inner);
    pp = __ldg(base + D.inner + ks);
    pm = __ldg(base + D.inner - ks);
  }
  if (dn) {
    d0 = __ldg(base - D.inner);
    dp = __ldg(base - D.inner + ks);
    dm = __ldg(base - D.inner - ks);
  }
  double r[3];
  r[1] = m0 + a * mp + 0.5 * mm + a * (pm + a * p0) + 0.5 * (dp + 0.5 * d0);
  r[2] = h ? 0.5 * mp + a * (0.5 * p0 + pp) : 0.0;
  r[0] = dn ? 0.5 * mm + 0.5 * (0.5 * d0 + dm) : 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int k = k0 + (d - 1) * D.kstride;
    double v = r[d];
    if (MASK) {  // last pass: rows and columns of fixed DoFs
      int ix, iy, iz;
      node_xyz(c, D.at + o, ix, iy, iz);
      const int jx = ix + k / 9 - 1, jy = iy + (k / 3) % 3 - 1, jz = iz + k % 3 - 1;
      const bool jin = jx >= 0 && jx < c.NX && jy >= 0 && jy < c.NY && jz >= 0 && jz < c.NZ;
      const long long J = jin ? ((long long)jx * c.NY + jy) * c.NZ + jz : 0;
      if (!(jin && mc[3 * (D.at + o) + q / 3] && mc[3 * J + q % 3])) v = 0.0;
    }
    Sout[(long long)(k * 9 + q) * D.sout + o] = v;
  }
}

// Scratch of the passes: two intermediate operators on some x planes of the
// fine grid. 2P + 1 planes give P planes of the coarse grid, so the passes run
// slab by slab where the whole is above kRapScratch, 512 MB (160x80x80 needs 205;
// about 2.7 million elements reach it): the intermediates are three quarters of
// level 1's operator, memory that the largest meshes do not have. A slab repeats
// one fine plane of the one before.
constexpr long long kRapScratch = 1LL << 26;  // doubles
static long long rap_plane(const Grid& f, const Grid& c) { return 243LL * (f.NY + c.NY) * c.NZ; }

long long rap_scratch(const Grid& f, const Grid& c) {
  const long long w = rap_plane(f, c);
  return std::min((long long)f.NX, std::max(3LL, kRapScratch / w)) * w;
}

// room: doubles of scratch (three planes or the whole, at least)
void rap(const Grid& fine, const Grid& coarse, const double* S_f, const uint8_t* mask_c, double* S_c, double* scratch,
         long long room, cudaStream_t s) {
  const Grid &f = fine, &c = coarse;
  const long long fits = room / rap_plane(f, c), inner = (long long)c.NY * c.NZ;
  const int P = fits >= f.NX ? c.NX : (int)((fits - 1) / 2);
  if (P < 1) throw std::runtime_error("R.A.P: too little scratch");
  auto nb = [](const RapDim& D) { return dim3((unsigned)((D.outer * D.ni * D.inner + 255) / 256), 81); };
  for (int I0 = 0; I0 < c.NX; I0 += P) {
    const int I1 = std::min(c.NX, I0 + P), f0 = std::max(0, 2 * I0 - 1), np = std::min(f.nx, 2 * I1 - 1) - f0 + 1;
    const long long n1 = (long long)np * f.NY * c.NZ, n2 = np * inner;
    double* T1 = scratch;
    double* T2 = scratch + 243LL * n1;
    const RapDim dz{f.nz, c.nz, 1, (long long)np * f.NY, 1, f.nnodes, n1, 0, c.NZ, 0, f.NZ, 0},
        dy{f.ny, c.ny, c.NZ, np, 3, n1, n2, 0, c.NY, 0, f.NY, 0},
        dx{f.nx, c.nx, inner, 1, 9, n2, c.nnodes, I0, I1 - I0, f0, np, I0 * inner};
    k_rap_dim<false><<<nb(dz), 256, 0, s>>>(dz, S_f + (long long)f0 * f.NY * f.NZ, T1, c, mask_c);
    TOPO_LAUNCH_CHECK();
    k_rap_dim<false><<<nb(dy), 256, 0, s>>>(dy, T1, T2, c, mask_c);
    TOPO_LAUNCH_CHECK();
    k_rap_dim<true><<<nb(dx), 256, 0, s>>>(dx, T2, S_c + I0 * inner, c, mask_c);
    TOPO_LAUNCH_CHECK();
  }
}

// ------------------------------------------------------------- stencil apply
// Coefficient q = c*3 + d of block k of node n at S[(k*9 + q) * ns + n], in
// every precision; ns is the node count (BF16: rounded up to even, because a
// thread reads the coefficients of two nodes at once).
//
// A CTA owns 32 NPT consecutive nodes and has one warp per component c: a
// thread accumulates row c of its NPT nodes, 81 coefficients each, coalesced
// over the lanes and fetched a third (9 blocks) ahead of their use. The u
// values of the nine (dx, dy) runs of nodes around the CTA's are staged once
// in shared memory (rounded to BF16 there when BF). Couplings to nodes outside
// the grid are zero, so the run's neighbours in memory stand in for them. The
// rows meet in shared memory and the epilogue runs in order of the DoFs.
// The sums of a row are those of a thread per node, in the same order.
//
// Bound by HBM / L2 on large levels (243 coefficients per node), by one chain
// of three fetches on small ones. Against one thread per node (FP32 / BF16
// blocks padded to 12 coefficients), Chebyshev step, B200: FP64 4,225 nodes
// 21.9 -> 6.1 us, 30,625 nodes (59 MB of coefficients) 43 -> 18 us; BF16
// 136,161 nodes (66 MB) 30 -> 26 us.
template <typename TC, int NPT>
struct CoefV;
template <>
struct CoefV<double, 1> {
  using V = double;
};
template <>
struct CoefV<float, 1> {
  using V = float;
};
template <>
struct CoefV<__nv_bfloat16, 2> {
  using V = uint32_t;
};

// TC: stencil coefficient type; T: vector type; BF: round u to BF16.
// NV columns (vs entries apart) share the coefficients a thread has fetched;
// blockIdx.y is the group of NV columns (of nv).
template <typename TC, typename T, bool BF, Epi EPI, int NPT, int NV>
__global__ void __launch_bounds__(96)
k_stencil(Grid g, long long ns, const TC* __restrict__ S, const T* u, const uint8_t* __restrict__ mask,
          EpiDev<T> ep, const KrylovState* st, int nv, long long vs) {
  using V = typename CoefV<TC, NPT>::V;
  constexpr int NN = 32 * NPT, RUN = 3 * (NN + 2);
  __shared__ T us[NV][9][RUN];
  __shared__ T os[NV][3 * NN];
  const int v0 = NV > 1 ? blockIdx.y * NV : 0, nc = NV > 1 ? min(NV, nv - v0) : 1;
  u += v0 * vs;
  const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
  const long long n0 = blockIdx.x * (long long)NN, n = n0 + lane * NPT;
  const bool live = n < g.nnodes;
  const V* Sp = reinterpret_cast<const V*>(S + (long long)(3 * c) * ns + (live ? n : 0));
  const long long step = ns / NPT;  // in V
  V cf[2][27];
  auto fetch = [&](int dx, V (&w)[27]) {
#pragma unroll
    for (int k = 0; k < 9; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d) w[3 * k + d] = live ? __ldg(Sp + (long long)((9 * dx + k) * 9 + d) * step) : (V)0;
  };
  fetch(0, cf[0]);
  chain_wait();
  chain_release();
  if (st != nullptr && st->done) return;
  // nodes n0 - 1 .. n0 + NN of each run, shifted by (dx, dy)
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const long long base = 3 * (n0 - 1 + ((long long)(r / 3 - 1) * g.NY + (r % 3 - 1)) * g.NZ);
    for (int i = threadIdx.x; i < RUN; i += 96) {
      const long long j = base + i;
      const bool in = j >= 0 && j < g.ndof && topo_in_range(j, g.ndof);
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        T v = (in && q < nc) ? u[q * vs + j] : (T)0;
        if constexpr (BF) v = __bfloat162float(__float2bfloat16_rn((float)v));
        us[q][r][i] = v;
      }
    }
  }
  __syncthreads();
  T a[NV][NPT];
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int p = 0; p < NPT; ++p) a[q][p] = 0;
#pragma unroll
  for (int dx = 0; dx < 3; ++dx) {
    if (dx < 2) fetch(dx + 1, cf[(dx + 1) & 1]);
    const V(&w)[27] = cf[dx & 1];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
#pragma unroll
      for (int p = 0; p < NPT; ++p) {
        T s[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if constexpr (NPT == 2) s[d] = (T)__uint_as_float(p ? (w[3 * k + d] & 0xFFFF0000u) : (w[3 * k + d] << 16));
          else s[d] = (T)w[3 * k + d];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          const T* uj = &us[q][3 * dx + k / 3][3 * (lane * NPT + p + k % 3)];
          a[q][p] += fma(s[2], uj[2], fma(s[0], uj[0], s[1] * uj[1]));
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int p = 0; p < NPT; ++p) os[q][3 * (lane * NPT + p) + c] = a[q][p];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    if (q >= nc) break;
    const long long co = (v0 + q) * vs;
    EpiDev<T> e = ep;
    if constexpr (EPI == Epi::Store || EPI == Epi::Residual) e.y += co;
    if constexpr (EPI == Epi::Residual) e.b += co;
    if constexpr (EPI == Epi::RUpd || EPI == Epi::ChebR) e.r += co;
    if constexpr (EPI == Epi::ChebR) {
      e.x += co;
      e.d_out += co;
    }
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const int t = threadIdx.x + 96 * h;
      const long long i = 3 * n0 + t;
      if (i < g.ndof && topo_in_range(i, g.ndof)) epilogue_store<T, EPI>(e, i, mask[i] != 0, os[q][t], u[q * vs + i]);
    }
  }
}

template <typename TC, typename T, bool BF, int NV>
static void launch_stencil(const Grid& g, const void* S, const void* u, const uint8_t* mask, void* y, Epi epi,
                           const EpiArgs& ea, cudaStream_t s, int nv, long long vs) {
  constexpr int NPT = sizeof(TC) == 2 ? 2 : 1;
  const dim3 nb((unsigned)((g.nnodes + 32 * NPT - 1) / (32 * NPT)), (unsigned)((nv + NV - 1) / NV));
  const long long ns = NPT == 2 ? stencil16_stride(g.nnodes) : g.nnodes;
  const TC* SS = (const TC*)S;
  const T* uu = (const T*)u;
  const EpiDev<T> ep = make_epi<T>(y, ea);
  switch (epi) {
    case Epi::Store:
      launch_chained(k_stencil<TC, T, BF, Epi::Store, NPT, NV>, nb, 96, 0, s, g, ns, SS, uu, mask, ep, ea.st, nv, vs);
      break;
    case Epi::Residual:
      launch_chained(k_stencil<TC, T, BF, Epi::Residual, NPT, NV>, nb, 96, 0, s, g, ns, SS, uu, mask, ep, ea.st, nv, vs);
      break;
    case Epi::ChebR:
      launch_chained(k_stencil<TC, T, BF, Epi::ChebR, NPT, NV>, nb, 96, 0, s, g, ns, SS, uu, mask, ep, ea.st, nv, vs);
      break;
    case Epi::RUpd:
      launch_chained(k_stencil<TC, T, BF, Epi::RUpd, NPT, NV>, nb, 96, 0, s, g, ns, SS, uu, mask, ep, ea.st, nv, vs);
      break;
    default:
      throw std::runtime_error("stencil_apply: unsupported epilogue");
  }
}

// Columns that share one fetch of the coefficients (static shared memory: FP64 4 x 8.1 KB).
constexpr int kStencilCols = 4;

void stencil_apply(Prec p, bool vec64, const Grid& g, const void* S, const void* u, const uint8_t* mask, void* y,
                   Epi epi, const EpiArgs& ea, cudaStream_t s, int nv, long long vs) {
#define TOPO_STENCIL(TC, T, BF)                                                            \
  do {                                                                                     \
    if (nv > 1) launch_stencil<TC, T, BF, kStencilCols>(g, S, u, mask, y, epi, ea, s, nv, vs); \
    else launch_stencil<TC, T, BF, 1>(g, S, u, mask, y, epi, ea, s, 1, 0);                 \
  } while (0)
  if (vec64) {
    if (p != Prec::F64) throw std::runtime_error("stencil_apply: FP64 vectors need an FP64 stencil");
    TOPO_STENCIL(double, double, false);
  } else if (p == Prec::F32) {
    TOPO_STENCIL(float, float, false);
  } else if (p == Prec::BF16) {
    TOPO_STENCIL(__nv_bfloat16, float, true);
  } else {
    throw std::runtime_error("stencil_apply: FP32 vectors need an FP32 or BF16 stencil");
  }
#undef TOPO_STENCIL
}

// Jacobi inverse diagonal from the centre block (k = 13), with the
// reference's guard |d| <= 1e-12 -> 1 (multigrid_v4.py:269, 752).
__global__ void k_stencil_dinv(Grid g, const double* __restrict__ S, const uint8_t* __restrict__ mask,
                               double* __restrict__ d64, float* __restrict__ d32) {
  const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (n >= g.nnodes) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double d = S[(long long)(13 * 9 + c * 3 + c) * g.nnodes + n];
    d = fabs(d) > 1e-12 ? d : 1.0;
    const double v = mask[3 * n + c] ? 1.0 / d : 0.0;
    if (d64) d64[3 * n + c] = v;
    if (d32) d32[3 * n + c] = (float)v;
  }
}

void stencil_dinv(const Grid& g, const double* S, const uint8_t* mask, double* dinv64, float* dinv32,
                  cudaStream_t s) {
  const int bs = 256;
  k_stencil_dinv<<<(unsigned)((g.nnodes + bs - 1) / bs), bs, 0, s>>>(g, S, mask, dinv64, dinv32);
  TOPO_LAUNCH_CHECK();
}

// FP64 setup stencil -> FP32 / BF16 apply copies in the same order.
__global__ void __launch_bounds__(256) k_convert(long long nnodes, long long ns16, const double* __restrict__ S, float* __restrict__ S32,
                                                 __nv_bfloat16* __restrict__ S16) {
  const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (n >= nnodes) return;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const long long k = blockIdx.y * 9LL + q;
    const float v = (float)S[k * nnodes + n];
    if (S32) S32[k * nnodes + n] = v;
    if (S16) S16[k * ns16 + n] = __float2bfloat16_rn(v);
  }
}

long long stencil16_stride(long long nnodes) { return (nnodes + 1) & ~1LL; }

// nnodes: nodes of the level; the copies hold 243 nnodes (S16: 243
// stencil16_stride(nnodes)) values.
void stencil_convert(long long nnodes, const double* S, float* S32, __nv_bfloat16* S16, cudaStream_t s) {
  k_convert<<<dim3((unsigned)((nnodes + 255) / 256), 27), 256, 0, s>>>(nnodes, stencil16_stride(nnodes), S, S32, S16);
  TOPO_LAUNCH_CHECK();
}

// ----------------------------------------------------------------- transfers
// Coarse free set by injection, reproducing the reference's linear-index test
// (solver_v2.py:717-764): coarse node (I,J,K) reads fine node index
// 2I*(ny_f+1)*(nz_f+1) + 2J*(nz_f+1) + 2K; a DoF past the end is fixed.
__global__ void k_inject_mask(Grid f, Grid c, const uint8_t* __restrict__ mf, uint8_t* __restrict__ mc) {
  const long long I = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (I >= c.nnodes) return;
  int ix, iy, iz;
  node_xyz(c, I, ix, iy, iz);
  const long long fn = 2LL * ix * f.NY * f.NZ + 2LL * iy * f.NZ + 2LL * iz;
  for (int d = 0; d < 3; ++d) {
    const long long fd = 3 * fn + d;
    mc[3 * I + d] = (fd < f.ndof) ? mf[fd] : (uint8_t)0;
  }
}

void inject_mask(const Grid& fine, const Grid& coarse, const uint8_t* mf, uint8_t* mc, cudaStream_t s) {
  const int bs = 256;
  k_inject_mask<<<(unsigned)((coarse.nnodes + bs - 1) / bs), bs, 0, s>>>(fine, coarse, mf, mc);
  TOPO_LAUNCH_CHECK();
}

// r_c = mask_c * P^T r_f: one thread per coarse DoF, its 27 reads issued
// together (missing ones have weight zero). On the coarsest level free DoF i
// goes to compact[index[i]] in FP64, the right-hand side of the coarsest
// solve; on the others r_c starts the level's smoother right here, d = c2 D^-1
// r_c, x = ax d (x = 0 before), which saves a launch per level. Latency bound
// on small levels: one thread per node over three nested loops took 7.5 us
// there, this 2.4 us (and the start 1.9 us as a kernel of its own).
template <typename T>
__global__ void __launch_bounds__(128) k_restrict(Grid f, Grid c, const T* rf, const uint8_t* __restrict__ mc,
                                                  SmoothStart<T> ss, const int* __restrict__ index, double* compact,
                                                  const KrylovState* st, long long vsf, long long vsc, long long vscompact) {
  chain_enter();
  if (st != nullptr && st->done) return;
  rf += blockIdx.y * vsf;  // column
  if (compact != nullptr) compact += blockIdx.y * vscompact;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= c.ndof) return;
  const long long I = i / 3;
  const int d = (int)(i - 3 * I);
  int Ix, Iy, Iz;
  node_xyz(c, I, Ix, Iy, Iz);
  T wx[3], wy[3], wz[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int x = 2 * Ix + s - 1, y = 2 * Iy + s - 1, z = 2 * Iz + s - 1;
    wx[s] = (x < 0 || x > f.nx) ? (T)0 : (T)prolong_w1(x, Ix, c.nx);
    wy[s] = (y < 0 || y > f.ny) ? (T)0 : (T)prolong_w1(y, Iy, c.ny);
    wz[s] = (z < 0 || z > f.nz) ? (T)0 : (T)prolong_w1(z, Iz, c.nz);
  }
  T v[27];
#pragma unroll
  for (int k = 0; k < 27; ++k) {
    const T w = wx[k / 9] * wy[(k / 3) % 3] * wz[k % 3];
    const long long n = ((long long)(2 * Ix + k / 9 - 1) * f.NY + (2 * Iy + (k / 3) % 3 - 1)) * f.NZ + (2 * Iz + k % 3 - 1);
    v[k] = (w != (T)0 && topo_in_range(n, f.nnodes)) ? rf[3 * n + d] : (T)0;
  }
  T a = 0;
#pragma unroll
  for (int k = 0; k < 27; ++k) a += (wx[k / 9] * wy[(k / 3) % 3] * wz[k % 3]) * v[k];
  const T r = mc[i] ? a : (T)0;
  if (compact != nullptr) {
    if (index[i] >= 0) compact[index[i]] = (double)r;
    return;
  }
  const long long o = blockIdx.y * vsc + i;
  const T d0 = ss.c2 * (ss.dinv[i] * r);
  ss.r[o] = r;
  ss.d[o] = d0;
  ss.x[o] = (T)0 + ss.ax * d0;
}

void restrict_vec(bool vec64, const Grid& fine, const Grid& coarse, const void* rf, const uint8_t* mc,
                  const SmoothStart<void>& to, const int* index, double* compact, const KrylovState* st, cudaStream_t s,
                  int nv, long long vsf, long long vsc, long long vscompact) {
  const int bs = 128;
  const dim3 nb((unsigned)((coarse.ndof + bs - 1) / bs), (unsigned)nv);
  if (vec64)
    launch_chained(k_restrict<double>, nb, bs, 0, s, fine, coarse, (const double*)rf, mc, smooth_start<double>(to), index, compact, st, vsf, vsc, vscompact);
  else
    launch_chained(k_restrict<float>, nb, bs, 0, s, fine, coarse, (const float*)rf, mc, smooth_start<float>(to), index, compact, st, vsf, vsc, vscompact);
}

// x_f += mask_f * P e_c: one thread per fine node, its (at most) 24 reads issued
// together. (One thread per DoF repeats the index arithmetic three times and is
// bound by it: 23 us on level 0 of 160x80x80, this 9 us.)
template <typename T>
__global__ void __launch_bounds__(128) k_prolong_add(Grid f, Grid c, const T* ec, const uint8_t* __restrict__ mf,
                                                     T* xf, T* e_out, const KrylovState* st,
                                                     long long vsf, long long vsc) {
  chain_enter();
  if (st != nullptr && st->done) return;
  ec += blockIdx.y * vsc;  // column
  xf += blockIdx.y * vsf;
  if (e_out) e_out += blockIdx.y * vsf;
  const long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (n >= f.nnodes) return;
  int ix, iy, iz;
  node_xyz(f, n, ix, iy, iz);
  const int px = ix >> 1, py = iy >> 1, pz = iz >> 1;
  // weights of the lower and upper parent (none: zero)
  const bool hx = (ix & 1) && px + 1 <= c.nx, hy = (iy & 1) && py + 1 <= c.ny, hz = (iz & 1) && pz + 1 <= c.nz;
  const T wx[2] = {hx ? (T)0.5 : (T)1, hx ? (T)0.5 : (T)0};
  const T wy[2] = {hy ? (T)0.5 : (T)1, hy ? (T)0.5 : (T)0};
  const T wz[2] = {hz ? (T)0.5 : (T)1, hz ? (T)0.5 : (T)0};
  T v[8][3], x[3];
  uint8_t m[3];
  const long long J0 = ((long long)px * c.NY + py) * c.NZ + pz;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const bool in = (!(k & 4) || hx) && (!(k & 2) || hy) && (!(k & 1) || hz);
    const long long J = J0 + ((k >> 2) * c.NY + ((k >> 1) & 1)) * (long long)c.NZ + (k & 1);
    const bool ok = in && topo_in_range(J, c.nnodes);
#pragma unroll
    for (int d = 0; d < 3; ++d) v[k][d] = ok ? ec[3 * J + d] : (T)0;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    x[d] = xf[3 * n + d];
    m[d] = mf[3 * n + d];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    T a = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) a += (wx[k >> 2] * wy[(k >> 1) & 1] * wz[k & 1]) * v[k][d];
    const T e = m[d] ? a : (T)0;
    xf[3 * n + d] = x[d] + e;
    if (e_out) e_out[3 * n + d] = e;
  }
}

void prolong_add(bool vec64, const Grid& fine, const Grid& coarse, const void* ec, const uint8_t* mf, void* xf,
                 void* e_out, const KrylovState* st, cudaStream_t s, int nv, long long vsf, long long vsc) {
  const int bs = 128;
  const dim3 nb((unsigned)((fine.nnodes + bs - 1) / bs), (unsigned)nv);
  if (vec64)
    launch_chained(k_prolong_add<double>, nb, bs, 0, s, fine, coarse, (const double*)ec, mf, (double*)xf, (double*)e_out, st, vsf, vsc);
  else
    launch_chained(k_prolong_add<float>, nb, bs, 0, s, fine, coarse, (const float*)ec, mf, (float*)xf, (float*)e_out, st, vsf, vsc);
}

TOPO_BOUNDS_READER(bounds_flag_coarse)

}  // namespace topo
