// design.cu - density filter, OC updates and field statistics on the device.
//
// The OC bisections keep their whole state (lambda bracket, phase, counters) in
// device memory: each pass evaluates the volume of one or several candidates
// with a deterministic grid reduction and the last block advances the
// bisection, so the host only checks a "done" flag every few passes instead of
// reading a mean per step (the reference runs the loop in NumPy on the host,
// src/topogpu/solver.py:94-117).
#include "internal.cuh"
#include "reduce.cuh"

#include <cmath>
#include <functional>
#include <stdexcept>
#include <vector>

namespace topo {

// Offsets and weights of the linear-hat filter: every element at centre
// distance d <= rmin - 1e-10 with weight rmin - d, plus the element itself with
// weight rmin (pub_simp_solver.py:215-243; kd-tree query_pairs radius).
static void set_filter(FilterStencil& fs, double rmin, cudaStream_t s) {
  if (fs.rmin == rmin) return;
  const int R = (int)std::floor(rmin);
  std::vector<int> off;
  std::vector<double> w;
  TapGroups tg;
  tg.R = R;
  const char* too_large = "filter radius too large (more than 1331 elements within rmin)";
  if (R > kMaxFilterR) throw std::runtime_error(too_large);
  for (int dz = -R; dz <= R; ++dz) {  // taps of one dz together: one z test per group
    tg.start[dz + R] = (int)w.size();
    for (int dx = -R; dx <= R; ++dx)
      for (int dy = -R; dy <= R; ++dy) {
        const double d = std::sqrt((double)(dx * dx + dy * dy + dz * dz));
        if (dx == 0 && dy == 0 && dz == 0) {
          off.insert(off.end(), {0, 0, 0});
          w.push_back(rmin);
        } else if (d <= rmin - 1e-10) {
          off.insert(off.end(), {dx, dy, dz});
          w.push_back(rmin - d);
        }
      }
  }
  tg.start[2 * R + 1] = (int)w.size();
  if ((int)w.size() > kMaxFilterOff) throw std::runtime_error(too_large);
  TOPO_CUDA_CHECK(cudaMemcpyAsync(fs.off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice, s));
  TOPO_CUDA_CHECK(cudaMemcpyAsync(fs.w, w.data(), sizeof(double) * w.size(), cudaMemcpyHostToDevice, s));
  TOPO_CUDA_CHECK(cudaStreamSynchronize(s));
  fs.rmin = rmin;
  fs.n = (int)w.size();
  fs.tg = tg;
}

// The taps of the filter in shared memory, grouped by dz: weight, distance in
// the linear element index, dx and dy as signed bytes; the groups' weight sums.
struct Tap {
  double w;
  int lin, off;
};
struct Taps {
  Tap t[kMaxFilterOff];
  double gw[2 * kMaxFilterR + 1];
  double full;  // weight sum of a row with all its taps
};

__device__ __forceinline__ void load_taps(Taps& t, const Grid& g, const TapGroups& tg, const int* __restrict__ fo,
                                          const double* __restrict__ fw) {
  const int noff = tg.start[2 * tg.R + 1];
  for (int k = threadIdx.x; k < noff; k += blockDim.x) {
    const int dx = fo[3 * k], dy = fo[3 * k + 1], dz = fo[3 * k + 2];
    t.t[k] = Tap{fw[k], (dx * g.ny + dy) * g.nz + dz, (dx & 255) | (dy & 255) << 8};
  }
  if (threadIdx.x < 2 * tg.R + 1) {
    double s = 0.0;
    for (int k = tg.start[threadIdx.x]; k < tg.start[threadIdx.x + 1]; ++k) s += fw[k];
    t.gw[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int d = 0; d < 2 * tg.R + 1; ++d) s += t.gw[d];
    t.full = s;
  }
  __syncthreads();
}

struct ElemXyz {
  int x, y, z;
};
__device__ __forceinline__ ElemXyz elem_xyz(const Grid& g, long long e) {
  ElemXyz q;
  if (g.nelem < (1LL << 31)) {  // 32-bit division
    const unsigned u = (unsigned)e, r = u / (unsigned)g.nz;
    q.z = (int)(u - r * (unsigned)g.nz);
    q.x = (int)(r / (unsigned)g.ny);
    q.y = (int)(r - (unsigned)q.x * (unsigned)g.ny);
  } else {
    q.z = (int)(e % g.nz);
    q.y = (int)((e / g.nz) % g.ny);
    q.x = (int)(e / ((long long)g.nz * g.ny));
  }
  return q;
}
// all taps in range in x and y
__device__ __forceinline__ bool xy_inside(const Grid& g, const ElemXyz& q, int R) {
  return q.x >= R && q.x < g.nx - R && q.y >= R && q.y < g.ny - R;
}
__device__ __forceinline__ bool tap_xy(const Grid& g, const ElemXyz& q, int off) {
  return (unsigned)(q.x + (int)(signed char)off) < (unsigned)g.nx && (unsigned)(q.y + (int)(signed char)(off >> 8)) < (unsigned)g.ny;
}

// Weight sum of the element's row: group sums where the row is cut in z only.
__device__ __forceinline__ double row_sum(const Grid& g, const ElemXyz& q, const TapGroups& tg, const Taps& t) {
  const bool xy = xy_inside(g, q, tg.R);
  if (xy && q.z >= tg.R && q.z < g.nz - tg.R) return t.full;
  double hs = 0.0;
  for (int d = 0; d < 2 * tg.R + 1; ++d) {
    if ((unsigned)(q.z + d - tg.R) >= (unsigned)g.nz) continue;
    if (xy) {
      hs += t.gw[d];
    } else {
      for (int k = tg.start[d]; k < tg.start[d + 1]; ++k)
        if (tap_xy(g, q, t.t[k].off)) hs += t.t[k].w;
    }
  }
  return hs;
}

// f(weight, index distance) for every tap of the element's row.
template <typename F>
__device__ __forceinline__ void each_tap(const Grid& g, const ElemXyz& q, const TapGroups& tg, const Taps& t, F f) {
  const bool xy = xy_inside(g, q, tg.R);
  for (int d = 0; d < 2 * tg.R + 1; ++d) {
    if ((unsigned)(q.z + d - tg.R) >= (unsigned)g.nz) continue;
    const int k1 = tg.start[d + 1];
    if (xy) {
#pragma unroll 4
      for (int k = tg.start[d]; k < k1; ++k) f(t.t[k].w, t.t[k].lin);
    } else {
      for (int k = tg.start[d]; k < k1; ++k)
        if (tap_xy(g, q, t.t[k].off)) f(t.t[k].w, t.t[k].lin);
    }
  }
}

// out_i = in_i / Hs_i, Hs_i the weight sum of row i
__global__ void __launch_bounds__(256) k_filter_rows(Grid g, const __grid_constant__ TapGroups tg, const int* __restrict__ fo,
                                                     const double* __restrict__ fw, const double* __restrict__ in, double* __restrict__ out) {
  __shared__ Taps t;
  load_taps(t, g, tg, fo, fw);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < g.nelem; e += (long long)gridDim.x * blockDim.x)
    out[e] = in[e] / row_sum(g, elem_xyz(g, e), tg, t);
}

// NORM: out_i = (sum_j w_ij in_j) / Hs_i; else out_i = sum_j w_ij in_j.
// One thread per element, lanes along z; weights and index distances come from
// shared memory (one 16-byte load per tap), elements whose row is not cut in x
// and y test z once per group. At 160x80x80, rmin 2 (27 taps): H x 29 us, H^T x
// 12 + 23 us, against 22 us for the row sums and 63 us with a division per tap
// before; bound by issue and L1 (16 MB of traffic would take 3 us).
template <bool NORM>
__global__ void __launch_bounds__(256) k_filter(Grid g, const __grid_constant__ TapGroups tg, const int* __restrict__ fo,
                                                const double* __restrict__ fw, const double* __restrict__ in, double* __restrict__ out) {
  __shared__ Taps t;
  load_taps(t, g, tg, fo, fw);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < g.nelem; e += (long long)gridDim.x * blockDim.x) {
    const ElemXyz q = elem_xyz(g, e);
    const double* p = in + e;
    double acc = 0.0;
    each_tap(g, q, tg, t, [&](double w, int lin) {
      if (topo_in_range(e + lin, g.nelem)) acc += w * p[lin];
    });
    out[e] = NORM ? acc / row_sum(g, q, tg, t) : acc;
  }
}

static unsigned filter_blocks(const Grid& g) {
  // one wave of the 8 CTAs an SM holds, so that the taps are loaded once per thread
  return (unsigned)std::min<long long>((g.nelem + 255) / 256, 8 * 148);
}

void filter_apply(FilterStencil& fs, const Grid& g, double rmin, const double* in, double* out, bool transpose,
                  double* work, cudaStream_t s) {
  set_filter(fs, rmin, s);
  const unsigned nb = filter_blocks(g);
  if (transpose) {
    k_filter_rows<<<nb, 256, 0, s>>>(g, fs.tg, fs.off, fs.w, in, work);
    TOPO_LAUNCH_CHECK();
    k_filter<false><<<nb, 256, 0, s>>>(g, fs.tg, fs.off, fs.w, work, out);
  } else {
    k_filter<true><<<nb, 256, 0, s>>>(g, fs.tg, fs.off, fs.w, in, out);
  }
  TOPO_LAUNCH_CHECK();
}

// ------------------------------------------------------------------- OC
// Device state of the bisection. Slots of a double[16] array:
enum OcSlot { OC_LO = 0, OC_HI, OC_EVAL, OC_MID, OC_MEAN, OC_PHASE, OC_NBIS, OC_DONE, OC_EVALS };

__device__ __forceinline__ double oc_candidate(double rho, double dc, double lam, double move, double rho_min) {
  const double dcs = fmin(dc, -1.0e-12);
  double t = -dcs / fmax(lam, 1.0e-40);
  t = fmax(t, 0.0);
  const double v = rho * sqrt(t);
  const double lo = fmax(rho - move, rho_min);
  const double hi = fmin(rho + move, 1.0);
  return fmin(fmax(v, lo), hi);
}

__global__ void k_oc_pass(long long n, const double* __restrict__ rho, const double* __restrict__ dc,
                          double volfrac, double move, double rho_min, double* st, RedWork red) {
  if (st[OC_DONE] != 0.0) return;
  const double lam = st[OC_EVAL];
  double v[1] = {0.0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v[0] += oc_candidate(rho[i], dc[i], lam, move, rho_min);
  double tot[1];
  if (grid_sum<1>(v, red, tot) && threadIdx.x == 0) {
    const double mean = tot[0] / (double)n;
    st[OC_MEAN] = mean;
    st[OC_EVALS] += 1.0;
    if (st[OC_PHASE] == 0.0) {
      // lambda_hi doubling while the candidate volume is too large
      if (mean > volfrac && st[OC_HI] < 1.0e40) {
        st[OC_LO] = st[OC_HI];
        st[OC_HI] = st[OC_HI] * 2.0;
        st[OC_EVAL] = st[OC_HI];
      } else {
        st[OC_PHASE] = 1.0;
        st[OC_EVAL] = 0.5 * (st[OC_LO] + st[OC_HI]);
      }
    } else {
      const double mid = st[OC_EVAL];
      if (mean > volfrac) st[OC_LO] = mid;
      else st[OC_HI] = mid;
      st[OC_MID] = mid;
      st[OC_NBIS] += 1.0;
      if (fabs(mean - volfrac) < 1.0e-8 || st[OC_NBIS] >= 80.0) st[OC_DONE] = 1.0;
      else st[OC_EVAL] = 0.5 * (st[OC_LO] + st[OC_HI]);
    }
  }
}

__global__ void k_oc_final(long long n, const double* __restrict__ rho, const double* __restrict__ dc, double move,
                           double rho_min, const double* st, double* __restrict__ out) {
  const double lam = st[OC_MID];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = oc_candidate(rho[i], dc[i], lam, move, rho_min);
}

__global__ void k_oc_init(double* st) {
  for (int i = 0; i < 16; ++i) st[i] = 0.0;
  st[OC_LO] = 0.0;
  st[OC_HI] = 1.0;
  st[OC_EVAL] = 1.0;
}

static int run_until_done(const std::function<void()>& pass, const double* st, int max_passes, cudaStream_t s) {
  double h[16];
  int launched = 0;
  while (launched < max_passes) {
    const int chunk = launched < 16 ? 8 : 16;
    for (int k = 0; k < chunk && launched < max_passes; ++k, ++launched) pass();
    TOPO_CUDA_CHECK(cudaMemcpyAsync(h, st, sizeof(double) * 16, cudaMemcpyDeviceToHost, s));
    TOPO_CUDA_CHECK(cudaStreamSynchronize(s));
    if (h[OC_DONE] != 0.0) return (int)h[OC_EVALS];
  }
  return -1;
}

int oc_update(long long n, const double* rho, const double* dc, double volfrac, double move, double rho_min,
              double* out, RedWork red, double* st, cudaStream_t s) {
  k_oc_init<<<1, 1, 0, s>>>(st);
  TOPO_LAUNCH_CHECK();
  const unsigned nb = (unsigned)std::min<long long>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads);
  auto pass = [&]() {
    k_oc_pass<<<nb, kRedThreads, 0, s>>>(n, rho, dc, volfrac, move, rho_min, st, red);
    TOPO_LAUNCH_CHECK();
  };
  // at most 134 doublings (1 -> 2^133 > 1e40) and 80 bisections
  const int evals = run_until_done(pass, st, 134 + 80 + 1, s);
  if (evals < 0) throw std::runtime_error("OC bisection did not terminate");
  k_oc_final<<<nb, kRedThreads, 0, s>>>(n, rho, dc, move, rho_min, st, out);
  TOPO_LAUNCH_CHECK();
  return evals;
}

// ------------------------------------------------------- filtered-volume OC
// run_simp's bisection halves [0, 1e9] until the bracket is below 1e-9: 60
// volumes. The volume falls monotonically with the multiplier, so each of its
// decisions is known once a larger multiplier was found too small or a smaller
// one too large. The search below evaluates several multipliers per sweep over
// the elements, narrows its own bracket [A, B] around the root by
// interpolation, and replays the bisection's path with the decisions the
// bracket implies; a midpoint inside the bracket is evaluated itself. The
// evaluation count, the last multiplier and the output are those of the
// sequential bisection (its volumes differ in the last bits, which could turn
// a decision only where a volume equals volfrac to 1e-15). Where the volume
// need not be monotone (negative rho or column sums), every midpoint is
// evaluated: the next three levels of the tree per sweep.
// State in a double[32]:
enum OcfSlot {
  OF_L1 = 0, OF_L2, OF_LM, OF_LAST, OF_K, OF_DONE, OF_EVALS,
  OF_A, OF_FA, OF_B, OF_FB,   // largest multiplier with too much volume, smallest without, and their volumes
  OF_TREE,                    // 1: not monotone, evaluate the tree
  OF_GUESS,                   // start value from the unclamped update
  OF_NC, OF_C,                // candidates of the next sweep: their number (at most 7), then they
  OF_T = OF_C + 7             // and their lambda^-1/2
};
constexpr int OF_SLOTS = 32, OF_MAXC = 7;

__device__ __forceinline__ double ocf_candidate(double rho, double dc, double dv, double lm, double move,
                                                double rho_min) {
  const double dcs = fmin(dc, -1e-12);
  const double dvs = fmax(dv, 1e-12);
  double rn = rho * sqrt(-dcs / (lm * dvs));
  rn = fmin(fmax(rn, rho - move), rho + move);
  rn = fmin(fmax(rn, rho_min), 1.0);
  return rn;
}

// The state in registers while one thread works on it.
struct OcfState {
  double L1, L2, LM, LAST, K, EVALS, A, FA, B, FB, GUESS;
  bool done, tree;
  int nc;
  double c[OF_MAXC];

  __device__ void load(const double* st) {
    L1 = st[OF_L1]; L2 = st[OF_L2]; LM = st[OF_LM]; LAST = st[OF_LAST]; K = st[OF_K]; EVALS = st[OF_EVALS];
    A = st[OF_A]; FA = st[OF_FA]; B = st[OF_B]; FB = st[OF_FB]; GUESS = st[OF_GUESS];
    done = st[OF_DONE] != 0.0;
    tree = st[OF_TREE] != 0.0;
    nc = (int)st[OF_NC];
#pragma unroll
    for (int q = 0; q < OF_MAXC; ++q) c[q] = st[OF_C + q];
  }
  __device__ void store(double* st) const {
    st[OF_L1] = L1; st[OF_L2] = L2; st[OF_LM] = LM; st[OF_LAST] = LAST; st[OF_K] = K; st[OF_EVALS] = EVALS;
    st[OF_A] = A; st[OF_FA] = FA; st[OF_B] = B; st[OF_FB] = FB; st[OF_GUESS] = GUESS;
    st[OF_DONE] = done ? 1.0 : 0.0;
    st[OF_TREE] = tree ? 1.0 : 0.0;
    st[OF_NC] = nc;
#pragma unroll
    for (int q = 0; q < OF_MAXC; ++q) {
      st[OF_C + q] = c[q];
      st[OF_T + q] = q < nc ? rsqrt(c[q]) : 0.0;
    }
  }
  // One decision of the bisection at its midpoint; true when it ends.
  __device__ bool decide(bool up) {
    EVALS += 1.0;
    if (up) L1 = LM;
    else L2 = LM;
    LAST = LM;
    K += 1.0;
    if (L2 - L1 < 1e-9 || K >= 100.0) {
      done = true;
      return true;
    }
    LM = 0.5 * (L1 + L2);
    return false;
  }
  __device__ void add(int nmax, double v) {
    if (nc < nmax && v > A && v < B && v != LM && v > 0.0 && v < 1e9) {
#pragma unroll
      for (int q = 1; q < OF_MAXC; ++q)  // (register indices are constants)
        if (q == nc) c[q] = v;
      ++nc;
    }
  }
  // Candidates of the next sweep (nmax of them at most): the bisection's next
  // midpoint first, then points around the interpolated root. The update scales
  // with t = lambda^-1/2 where it is not clamped, so the volume is interpolated
  // in t; the error of that is about the square of the bracket's relative width.
  __device__ void choose(int nmax, double volfrac) {
    c[0] = LM;
    nc = 1;
    if (tree) {
      if (nmax < 3) return;
      c[1] = 0.5 * (L1 + c[0]);
      c[2] = 0.5 * (c[0] + L2);
      nc = 3;
      if (nmax < 7) return;
      c[3] = 0.5 * (L1 + c[1]);
      c[4] = 0.5 * (c[1] + c[0]);
      c[5] = 0.5 * (c[0] + c[2]);
      c[6] = 0.5 * (c[2] + L2);
      nc = 7;
      return;
    }
    if (A > 0.0 && B < 1e300) {
      const double ta = rsqrt(A), tb = rsqrt(B), den = FA - FB;
      double t = den > 0.0 ? tb + (volfrac - FB) * (ta - tb) / den : 0.5 * (ta + tb);
      t = fmin(fmax(t, tb), ta);
      const double r = 1.0 / (t * t), w = (B - A) / r;
      add(nmax, r);
      if (w > 0.5) {  // wide: spread over the bracket
        for (int q = 1; q < nmax - 1; ++q) {
          const double tq = tb + (ta - tb) * q / (double)(nmax - 1);
          add(nmax, 1.0 / (tq * tq));
        }
      } else {
        const double d = fmax(0.25 * w * w, 4e-16);
        add(nmax, r * (1.0 - d));
        add(nmax, r * (1.0 + d));
        add(nmax, r * (1.0 - d * 0.0625));
        add(nmax, r * (1.0 + d * 0.0625));
        add(nmax, r * (1.0 - 16.0 * d));
        add(nmax, r * (1.0 + 16.0 * d));
      }
    } else if (A > 0.0) {  // one side open: outwards by growing factors
      for (double f = 8.0; nc < nmax && f < 1e60; f *= f) add(nmax, A * f);
    } else if (B < 1e300) {
      for (double f = 8.0; nc < nmax && f < 1e60; f *= f) add(nmax, B / f);
    } else {  // around the start value
      add(nmax, GUESS);
      add(nmax, GUESS * 0.5);
      add(nmax, GUESS * 2.0);
      add(nmax, GUESS * 0.0625);
      add(nmax, GUESS * 16.0);
      add(nmax, GUESS * 1e-3);
    }
  }
  // Volumes (as fractions) of the current candidates: update the bracket, replay
  // the bisection as far as it is decided, choose the next candidates.
  __device__ void advance(const double* vol, int nmax, double volfrac) {
    if (tree) {
      int q = 0;
      while (q < nc) {
        double vq = 0.0;
        for (int j = 0; j < OF_MAXC; ++j)
          if (j == q && j < nmax) vq = vol[j];
        const bool up = vq > volfrac;
        if (decide(up)) return;
        q = 2 * q + (up ? 2 : 1);
      }
    } else {
#pragma unroll
      for (int q = 0; q < OF_MAXC; ++q) {
        if (q >= nc || q >= nmax) continue;
        const bool up = vol[q] > volfrac;
        if (up && c[q] > A) {
          A = c[q];
          FA = vol[q];
        }
        if (!up && c[q] < B) {
          B = c[q];
          FB = vol[q];
        }
      }
      if (decide(vol[0] > volfrac)) return;  // the midpoint was evaluated itself
      while (LM <= A || LM >= B)
        if (decide(LM <= A)) return;
    }
    choose(nmax, volfrac);
  }
};

// Per-element invariants of the candidate clamp(s t): s = rho sqrt(-dc / dv)
// (the two clamps of ocf_candidate folded into one are formed on the fly), and
// the start value of the search; the sums also tell whether the volume is
// monotone.
__global__ void k_ocf_prep(long long n, const double* __restrict__ rho, const double* __restrict__ dc,
                           const double* __restrict__ dv, const double* __restrict__ colsum, double volfrac, int nmax,
                           int force_tree, double* __restrict__ sv, double* st, RedWork red) {
  double v[2] = {0.0, 0.0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double r = rho[i], cs = colsum ? colsum[i] : 1.0;
    const double s = r * sqrt(-fmin(dc[i], -1e-12) / fmax(dv[i], 1e-12));
    sv[i] = s == s ? s : -INFINITY;  // a NaN update is clamped to the lower bound
    v[0] += s == s ? fmin(fabs(s), 1e100) * cs : 0.0;
    if (!(r >= 0.0) || !(cs >= 0.0)) v[1] += 1.0;
  }
  double tot[2];
  if (grid_sum<2>(v, red, tot) && threadIdx.x == 0) {
    OcfState o;
    o.L1 = o.LAST = o.K = o.EVALS = o.A = o.FA = o.FB = 0.0;
    o.L2 = 1e9;
    o.LM = 0.5 * (0.0 + 1e9);
    o.B = INFINITY;
    o.done = false;
    o.tree = force_tree || tot[1] != 0.0;
    const double q = tot[0] / ((double)n * volfrac);
    o.GUESS = (q > 1e-15 && q < 3e4) ? q * q : 1.0;
    for (int j = 0; j < OF_MAXC; ++j) o.c[j] = 1.0;
    o.choose(nmax, volfrac);
    o.store(st);
  }
}

// One sweep: the volumes of all candidates, then the search in the last block.
// 24 B per element and at most seven clamped products (issue and the latency of
// the reduction). At 160x80x80 a call is about 5 sweeps of 18 us, against 24 of
// 28 us in the sequential form (three bisection levels per sweep, a division
// and a square root per candidate).
__global__ void __launch_bounds__(kRedThreads) k_ocf_pass(long long n, const double* __restrict__ rho, const double* __restrict__ sv,
                                                          const double* __restrict__ colsum, double volfrac, double move,
                                                          double rho_min, double* st, RedWork red) {
  if (st[OF_DONE] != 0.0) return;
  const int nc = (int)st[OF_NC];
  double t[OF_MAXC], v[OF_MAXC];
#pragma unroll
  for (int q = 0; q < OF_MAXC; ++q) {
    t[q] = st[OF_T + q];
    v[q] = 0.0;
  }
#pragma unroll 2
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double r = rho[i], s = sv[i], cs = colsum[i];
    const double lo = fmin(fmax(r - move, rho_min), 1.0), hi = fmin(fmax(r + move, rho_min), 1.0);
#pragma unroll
    for (int q = 0; q < OF_MAXC; ++q)
      if (q < nc) {
        double x = s * t[q];  // not NaN
        x = x < lo ? lo : x;
        x = x > hi ? hi : x;
        v[q] += x * cs;
      }
  }
  double tot[OF_MAXC];
  if (grid_sum<OF_MAXC>(v, red, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < OF_MAXC; ++q) tot[q] /= (double)n;
    OcfState o;
    o.load(st);
    o.advance(tot, OF_MAXC, volfrac);
    o.store(st);
  }
}

__global__ void k_ocf_final(long long n, const double* __restrict__ rho, const double* __restrict__ dc,
                            const double* __restrict__ dv, double move, double rho_min, const double* st,
                            double* __restrict__ out) {
  const double lm = st[OF_LAST];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = ocf_candidate(rho[i], dc[i], dv[i], lm, move, rho_min);
}

// Runs `pass` until the device state says done; every pass decides at least
// one of the at most 100 levels. Returns the evaluation count.
static int ocf_run(const std::function<void()>& pass, const double* st, const char* what, cudaStream_t s) {
  double h[OF_SLOTS];
  for (int launched = 0; launched < 104;) {
    const int chunk = launched ? 3 : 6;  // sweeps after the end return at entry
    for (int k = 0; k < chunk; ++k, ++launched) pass();
    TOPO_CUDA_CHECK(cudaMemcpyAsync(h, st, sizeof(double) * OF_SLOTS, cudaMemcpyDeviceToHost, s));
    TOPO_CUDA_CHECK(cudaStreamSynchronize(s));
    if (h[OF_DONE] != 0.0) return (int)h[OF_EVALS];
  }
  throw std::runtime_error(what);
}

// work: n doubles (s); st: OF_SLOTS doubles
int oc_update_filtered(long long n, const double* rho, const double* dc, const double* dv, const double* colsum,
                       double volfrac, double move, double rho_min, double* out, double* work, RedWork red, double* st,
                       cudaStream_t s) {
  const unsigned nb = (unsigned)std::min<long long>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads);
  k_ocf_prep<<<nb, kRedThreads, 0, s>>>(n, rho, dc, dv, colsum, volfrac, OF_MAXC, 0, work, st, red);
  TOPO_LAUNCH_CHECK();
  const int evals = ocf_run(
      [&]() {
        k_ocf_pass<<<nb, kRedThreads, 0, s>>>(n, rho, work, colsum, volfrac, move, rho_min, st, red);
        TOPO_LAUNCH_CHECK();
      },
      st, "filtered OC bisection did not terminate", s);
  k_ocf_final<<<nb, kRedThreads, 0, s>>>(n, rho, dc, dv, move, rho_min, st, out);
  TOPO_LAUNCH_CHECK();
  return evals;
}

// ------------------------------------------------- Heaviside projection
// Smoothed Heaviside of run_simp (pub_simp_solver.py:245-253):
//   h(x)  = (tanh(b e) + tanh(b (x - e))) / (tanh(b e) + tanh(b (1 - e)))
//   h'(x) = b (1 - tanh(b (x - e))^2) / (tanh(b e) + tanh(b (1 - e)))
// with the identity (h = x, h' = 1) unless b > 1e-6, the guard every run_simp
// call site applies (pub_simp_solver.py:331,348,366). The two tanh constants
// are computed on the host and passed in the kernel arguments.
struct Projection {
  double beta, eta, tbe, den;
  bool on;
};

static Projection make_projection(double beta, double eta) {
  Projection p{beta, eta, 0.0, 1.0, beta > 1e-6};
  if (p.on) {
    p.tbe = std::tanh(beta * eta);
    p.den = p.tbe + std::tanh(beta * (1.0 - eta));
  }
  return p;
}

__global__ void k_heaviside(long long n, const double* __restrict__ rho_f, Projection p, double* __restrict__ phys,
                            double* __restrict__ dh) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double x = rho_f[i];
    if (!p.on) {
      if (phys) phys[i] = x;
      if (dh) dh[i] = 1.0;
      continue;
    }
    const double t = tanh(p.beta * (x - p.eta));
    if (phys) phys[i] = (p.tbe + t) / p.den;
    if (dh) dh[i] = p.beta * (1.0 - t * t) / p.den;
  }
}

void heaviside_apply(long long n, const double* rho_f, double beta, double eta, double* phys, double* dh,
                     cudaStream_t s) {
  const Projection p = make_projection(beta, eta);
  if (n == 0) return;
  const unsigned nb = (unsigned)std::min<long long>(4 * kRedBlocks, (n + 255) / 256);
  k_heaviside<<<nb, 256, 0, s>>>(n, rho_f, p, phys, dh);
  TOPO_LAUNCH_CHECK();
}

// ------------------------------------------------- projected-volume OC
// run_simp's OC with Heaviside (pub_simp_solver.py:319-340): the volume of a
// candidate is sum_i h((H cand)_i) / n. The projection is nonlinear, so the
// colsum shortcut of the filtered OC does not apply. The same search runs with
// OP_NC candidates per sweep: k_ocp_cand writes them interleaved, k_ocp_vol
// filters all of them at every element with one pass over the taps, projects
// and sums. At 96x48x48 (rmin 2) a sweep is 36 us and a call takes about 6 of
// them, against 60 sequential evaluations of 26 us.
constexpr int OP_NC = kOcCandidates;

__global__ void __launch_bounds__(256) k_ocp_cand(long long n, const double* __restrict__ rho, const double* __restrict__ sv,
                                                  double move, double rho_min, const double* st, double* __restrict__ cand) {
  if (st[OF_DONE] != 0.0) return;
  const int nc = (int)st[OF_NC];
  double t[OP_NC];
#pragma unroll
  for (int q = 0; q < OP_NC; ++q) t[q] = st[OF_T + (q < nc ? q : 0)];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double r = rho[i], s = sv[i];
    const double lo = fmin(fmax(r - move, rho_min), 1.0), hi = fmin(fmax(r + move, rho_min), 1.0);
    double c[OP_NC];
#pragma unroll
    for (int q = 0; q < OP_NC; ++q) c[q] = fmin(fmax(s * t[q], lo), hi);
    double2* o = reinterpret_cast<double2*>(cand + OP_NC * i);
    o[0] = make_double2(c[0], c[1]);
    o[1] = make_double2(c[2], c[3]);
  }
}

__global__ void __launch_bounds__(kRedThreads) k_ocp_vol(Grid g, const __grid_constant__ TapGroups tg, const int* __restrict__ fo,
                                                         const double* __restrict__ fw, const double* __restrict__ cand, Projection p,
                                                         double volfrac, double* st, RedWork red) {
  if (st[OF_DONE] != 0.0) return;
  __shared__ Taps tp;
  load_taps(tp, g, tg, fo, fw);
  double v[OP_NC] = {};
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < g.nelem;
       e += (long long)gridDim.x * blockDim.x) {
    const ElemXyz x = elem_xyz(g, e);
    const double2* ce = reinterpret_cast<const double2*>(cand + OP_NC * e);
    double acc[OP_NC] = {};
    each_tap(g, x, tg, tp, [&](double w, int lin) {
      const double2 a = ce[2 * (long long)lin], b = ce[2 * (long long)lin + 1];
      acc[0] += w * a.x;
      acc[1] += w * a.y;
      acc[2] += w * b.x;
      acc[3] += w * b.y;
    });
    const double hs = row_sum(g, x, tg, tp);
#pragma unroll
    for (int q = 0; q < OP_NC; ++q) {
      const double f = acc[q] / hs;
      v[q] += p.on ? (p.tbe + tanh(p.beta * (f - p.eta))) / p.den : f;
    }
  }
  double tot[OP_NC];
  if (grid_sum<OP_NC>(v, red, tot) && threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < OP_NC; ++q) tot[q] /= (double)g.nelem;
    OcfState o;
    o.load(st);
    o.advance(tot, OP_NC, volfrac);
    o.store(st);
  }
}

// work: n doubles (s); cand: OP_NC n doubles, 16-byte aligned
int oc_update_projected(FilterStencil& fs, const Grid& g, double rmin, const double* rho, const double* dc, const double* dv,
                        double beta, double eta, double volfrac, double move, double rho_min, double* out,
                        double* work, double* cand, RedWork red, double* st, cudaStream_t s) {
  const long long n = g.nelem;
  set_filter(fs, rmin, s);
  const Projection p = make_projection(beta, eta);
  const unsigned nb = (unsigned)std::min<long long>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads);
  k_ocf_prep<<<nb, kRedThreads, 0, s>>>(n, rho, dc, dv, nullptr, volfrac, OP_NC, p.on && !(p.den > 0.0), work, st, red);
  TOPO_LAUNCH_CHECK();
  const int evals = ocf_run(
      [&]() {
        k_ocp_cand<<<nb, 256, 0, s>>>(n, rho, work, move, rho_min, st, cand);
        TOPO_LAUNCH_CHECK();
        k_ocp_vol<<<nb, kRedThreads, 0, s>>>(g, fs.tg, fs.off, fs.w, cand, p, volfrac, st, red);
        TOPO_LAUNCH_CHECK();
      },
      st, "projected OC bisection did not terminate", s);
  k_ocf_final<<<nb, kRedThreads, 0, s>>>(n, rho, dc, dv, move, rho_min, st, out);
  TOPO_LAUNCH_CHECK();
  return evals;
}

// ------------------------------------------------------------ field stats
__global__ void k_stats(long long n, const double* __restrict__ x, double* out4, RedWork red) {
  double sum = 0.0, gray = 0.0, mn = INFINITY, mx = -INFINITY;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double v = x[i];
    sum += v;
    gray += v * (1.0 - v);
    mn = fmin(mn, v);
    mx = fmax(mx, v);
  }
  __shared__ double smn[32], smx[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane == 0) {
    smn[wid] = mn;
    smx[wid] = mx;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    mn = warp_min(threadIdx.x < nw ? smn[threadIdx.x] : INFINITY);
    mx = warp_max(threadIdx.x < nw ? smx[threadIdx.x] : -INFINITY);
  }
  // min/max travel through the sum slots of a separate partial row
  double v[4] = {sum, gray, 0.0, 0.0};
  __shared__ bool s_last;
  block_sum<4>(v);
  const unsigned nb = gridDim.x;
  if (threadIdx.x == 0) {
    red.partials[(size_t)blockIdx.x * 4 + 0] = v[0];
    red.partials[(size_t)blockIdx.x * 4 + 1] = v[1];
    red.partials[(size_t)blockIdx.x * 4 + 2] = mn;
    red.partials[(size_t)blockIdx.x * 4 + 3] = mx;
    __threadfence();
    s_last = (atomicAdd(red.ticket, 1u) == nb - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the last block adds the partials: thread t those of blocks t, t + 256, ...,
  // then the same tree as above (a fixed order)
  double w[4] = {0.0, 0.0, 0.0, 0.0};
  mn = INFINITY;
  mx = -INFINITY;
  for (unsigned b = threadIdx.x; b < nb; b += blockDim.x) {
    w[0] += __ldcg(red.partials + (size_t)b * 4 + 0);
    w[1] += __ldcg(red.partials + (size_t)b * 4 + 1);
    mn = fmin(mn, __ldcg(red.partials + (size_t)b * 4 + 2));
    mx = fmax(mx, __ldcg(red.partials + (size_t)b * 4 + 3));
  }
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane == 0) {
    smn[wid] = mn;
    smx[wid] = mx;
  }
  block_sum<4>(w);
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    for (int k = 0; k < nw; ++k) {
      mn = fmin(mn, smn[k]);
      mx = fmax(mx, smx[k]);
    }
    out4[0] = w[0] / (double)n;
    out4[1] = mn;
    out4[2] = mx;
    out4[3] = 4.0 * (w[1] / (double)n);
    *red.ticket = 0u;
  }
}

void field_stats(long long n, const double* x, double* out4_dev, RedWork red, cudaStream_t s) {
  const unsigned nb = (unsigned)std::min<long long>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads);
  k_stats<<<nb, kRedThreads, 0, s>>>(n, x, out4_dev, red);
  TOPO_LAUNCH_CHECK();
}

TOPO_BOUNDS_READER(bounds_flag_design)

}  // namespace topo
