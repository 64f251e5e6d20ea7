// kmatvec_pt.cu - level-0 hex8 K.u in parity form (FP64, FP32 and BF16
// inputs), streaming along x with TMA-staged node planes.
//
// The stiffness of a cube of an isotropic (or axis-aligned orthotropic)
// material does not change under the three mirror images of the element. In
// the basis of sums and differences of the corner values along x, y and z
// (the 2x2x2 Hadamard transform of each displacement component) KE therefore
// falls apart into eight 3x3 blocks, one per parity class, and one element
// costs two separable transforms (adds) and 72 multiply-adds instead of 576.
// Along x the transform of a node plane is shared by the two layers it
// bounds, so the sums and differences in y and z are formed once per plane.
// A KE without that symmetry takes the general kernels (kmatvec_xs.cu,
// kmatvec_cc.cu): pt_prepare measures the couplings between the classes.
//
// Layout of the work. A plane is one contiguous run of nodes n = y*NZ + z. A
// thread owns the element m (lower corner at node m; the elements with
// z = nz or y = ny do not exist and have E = 0), loads the four nodes m, m+1,
// m+NZ, m+NZ+1 of the next plane from shared memory and walks the layers of
// its segment in x; the transformed previous plane (12 values) and the part
// of the next plane's result already known (12 values) stay in registers.
// Values are held as pairs over the parity in z (the z component's pair in
// the opposite order, so that a pair belongs to one pair of classes): in FP32
// each pair is one operand of the two-wide instructions (add / fma .f32x2),
// which halves the issue slots of the arithmetic.
// Back transform: in z with the neighbour lane's values (a warp covers 31
// elements, its lane 0 repeats the last element of the warp before), in y
// through shared memory: result(n) = P[n] + W[n - NZ]. The last addition and
// the epilogue run one step later over the linear range of DoFs, so every
// global access of the epilogue is coalesced, and one barrier per plane
// suffices. A CTA is one (window of nodes, segment of planes) pair. What the
// epilogue will read is prefetched to L2 two planes ahead.
//
// Staging: one cp.async.bulk (TMA, no multicast) per plane into a ring of
// three slots, completed on mbarriers; start rounded down to 16 bytes, a
// range ending in the vector's last partial 16-byte word gets that tail by
// plain loads. Every wait is bounded: a timeout raises the device's error
// flag, the copies in flight are drained (bounded) and the CTA exits.
//
// Bound: issue slots and the barrier per plane (about 280 instructions per
// element and step; 20% of the elements are halo), not HBM: at 160x80x80 FP32
// Store moves 29.4 MB (4.5 us at the copy rate), ChebR 92.8 MB (14 us), each and
// 3.2 MB of mask. Measured on a B200, rotating buffers, against the kernels it replaced there (kernel
// times): 160x80x80 FP32 Store 24.5 us (64), FP64 Store 37.9 us (130), ChebR
// with BF16 rounding 35.3 us (67, tensor cores), FP32 ChebR 35.0 us, FP32 RUpd
// 27.7 us (64); 24x12x6 FP64 4.4 us (9.6). The tensor-core form of the same operator does
// 1152 flop per element in 39 us of MMA issue; the parity form needs 312.
//
// Reference semantics: MatrixFreeKff.matvec (src/gpu_fem/solver_v2.py:1183-1223)
// and fused_matvec_bf16 (src/gpu_fem/cuda_fused_matvec.py:112-246): the BF16
// form multiplies BF16-rounded u by BF16-rounded KE and accumulates in FP32.
#include "internal.cuh"
#include "reduce.cuh"

#include <atomic>
#include <cmath>
#include <cstring>
#include <stdexcept>
#include <type_traits>
#include <vector>

namespace topo {
namespace pt {

// Class blocks K[q][c][d] of H KE H^T / 64: q = 4 qx + 2 qy + qz, member c of
// class q is component c with parity q ^ e_c.
// Stored as pairs over qz at ((2 qx + qy) * 9 + 3 c + d).
__constant__ double2 cK64[36];
__constant__ float2 cK32[36];  // of KE rounded to FP32: the FP32 operator is that of the rounded entries
__constant__ float2 cKbf[36];  // of KE rounded to BF16

constexpr int RING = 3;

// Columns share one line of planes (see the kernel): only the FP64 Chebyshev
// step, whose 255 registers have room for the loop (the others spill with it).
// 8 columns of 96x48x48: one segment per window and column keeps 264 CTAs of
// 75-node windows (of 296) or 104 of 199 (of 148) busy; equal parts fill all
// 148 with the wide ones (block solve 18.2 -> 17.0 ms).
template <typename T, Epi EPI>
constexpr bool line_split = sizeof(T) == 8 && EPI == Epi::ChebR;

template <typename T>
struct Params {
  Grid g;
  int PN, TO, nwin, nseg;  // nodes per plane, output nodes per window, windows, segments
  const void* u;
  const T* E;
  const uint8_t* mask;
  EpiDev<T> ep;
  int nv;                   // columns
  long long vs;             // column v of every vector starts v * vs entries on (u 16-byte aligned)
  int list;                 // != 0: u and y of column v are ucol[v], ycol[v]
  const void* ucol[8];
  T* ycol[8];
  KrylovState* st;
  RedWork red;
  int* err;
  int slot, off_pw, pw_n, off_bar;
  int poll, skip;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

template <typename T>
struct Pair;
template <>
struct Pair<double> {
  using V = double2;
};
template <>
struct Pair<float> {
  using V = float2;
};
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 vmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 vfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

template <typename V, bool BF>
__device__ __forceinline__ V kq(int i) {
  if constexpr (std::is_same_v<V, double2>) return cK64[i];
  else if constexpr (BF) return cKbf[i];
  else return cK32[i];
}

template <typename T, typename TU>
__device__ __forceinline__ T load_u(const TU* p) {
  if constexpr (sizeof(TU) == 2) return (T)__bfloat162float(*p);
  else return (T)*p;
}

// Hint: bring bytes [b, e) to L2 (thread 0; 16-byte granules, never past e).
__device__ __forceinline__ void prefetch_l2(const void* b, const void* e) {
  const unsigned long long a = (unsigned long long)b & ~15ULL;
  const long long n = (long long)(((unsigned long long)e & ~15ULL) - a);
  if (n > 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)n) : "memory");
}

// Threads per CTA = 32 NW. MINB: CTAs per SM the registers are sized for.
// COLS: several columns (a template flag: the column pointers cost registers
// the one-column form has no room for).
template <typename T, typename TU, bool BF, Epi EPI, bool COLS, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_level0_pt(const __grid_constant__ Params<T> P) {
  extern __shared__ __align__(128) unsigned char sm[];
  using V = typename Pair<T>::V;
  constexpr int NT = 32 * NW, SU = (int)sizeof(TU), ST = (int)sizeof(T);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Grid& g = P.g;
  const int NZ = g.NZ, PN = P.PN;
  // A CTA's output planes are segment sg of window w of column blockIdx.y; with
  // LINE, the planes of all windows of all columns are one line, cut into equal
  // parts, and a part is one or more pieces (of one window of one column each).
  constexpr bool LINE = COLS && line_split<T, EPI>;
  int count = 0, at = 0, end = 1;  // planes staged by the pieces before; the line
  if constexpr (LINE) {
    const long long all = (long long)P.nv * P.nwin * g.NX;
    at = (int)(all * blockIdx.x / gridDim.x);
    end = (int)(all * (blockIdx.x + 1) / gridDim.x);
  }
  do {
  int cv = COLS ? (int)blockIdx.y : 0, w, xa, xb;
  const int staged = LINE ? count : 0;
  if constexpr (LINE) {
    const int q = at / g.NX;
    cv = q / P.nwin;
    w = q - cv * P.nwin;
    xa = at - q * g.NX;
    xb = min(g.NX, xa + (end - at));
    at += xb - xa;
  } else {
    const int sg = (int)blockIdx.x / P.nwin;
    w = (int)blockIdx.x % P.nwin;
    xa = (int)((long long)g.NX * sg / P.nseg);
    xb = (int)((long long)g.NX * (sg + 1) / P.nseg);
  }
  const long long co = COLS ? cv * P.vs : 0LL;
  const TU* const uc = COLS && P.list ? reinterpret_cast<const TU*>(P.ucol[cv]) : reinterpret_cast<const TU*>(P.u) + co;
  T* const yc = COLS && P.list ? P.ycol[cv] : P.ep.y + co;
  const int n0 = w * P.TO, n1 = min(PN, n0 + P.TO);  // output nodes of a plane
  const int mlo = n0 - NZ - 1;                                             // first element of the window
  const int ms = max(mlo, 0), me = min(PN, mlo + 31 * NW + NZ + 2);        // staged nodes of every plane
  const int pf = max(xa - 1, 0), pl = min(xb, g.NX - 1);                   // planes read
  const uint32_t bar0 = smem_u32(sm + P.off_bar);

  for (int i = tid; i < P.off_pw / 16; i += NT) reinterpret_cast<uint4*>(sm)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0 && staged == 0) {
    for (int s = 0; s < RING; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8u * s), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  chain_wait();
  chain_release();
  if (P.st != nullptr && P.st->done) return;

  // plane p -> slot (staged + p - pf) % RING; node n of it at byte 16 + shift + 3 SU (n - mlo),
  // where shift makes the copy's source and destination agree modulo 16
  auto issue = [&](int p) {  // thread 0
    const int sl = (staged + p - pf) % RING;
    const int shift = (int)((((long long)p * PN + mlo) * (3 * SU)) & 15);
    const long long off0 = ((long long)p * PN + ms) * (3 * SU);
    const long long n = (long long)(me - ms) * (3 * SU);
    unsigned char* dst = sm + sl * P.slot + 16 + shift + (ms - mlo) * 3 * SU - (int)(off0 & 15);
    const unsigned char* src = reinterpret_cast<const unsigned char*>(uc);
    const long long a = off0 & ~15LL, vfloor = (g.ndof * (long long)SU) & ~15LL;
    long long e = (off0 + n + 15) & ~15LL;
    if (e > vfloor) {
      for (long long b = max(vfloor, a); b < off0 + n; ++b) dst[b - a] = src[b];
      e = vfloor;
    }
    const uint32_t bytes = e > a ? (uint32_t)(e - a) : 0u, bar = bar0 + 8u * (uint32_t)sl;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    if (bytes)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                   "l"(src + a), "r"(bytes), "r"(bar)
                   : "memory");
  };
  auto hint = [&](int x) {  // thread 0: what the epilogue of output plane x reads
    const long long b = 3 * ((long long)x * PN + n0), e = 3 * ((long long)x * PN + n1);
    if constexpr (EPI == Epi::Residual) prefetch_l2(P.ep.b + co + b, P.ep.b + co + e);
    if constexpr (EPI == Epi::RUpd || EPI == Epi::ChebR) prefetch_l2(P.ep.r + co + b, P.ep.r + co + e);
    if constexpr (EPI == Epi::ChebR) {
      prefetch_l2(P.ep.dinv + b, P.ep.dinv + e);
      prefetch_l2(P.ep.x + co + b, P.ep.x + co + e);
    }
    prefetch_l2(P.mask + b, P.mask + e);
  };
  int issued = pf;  // planes pf .. issued-1 have been issued (thread 0)
  if (tid == 0) {
    for (; issued <= pl && issued < pf + RING; ++issued)
      if (!(P.skip && issued == pf)) issue(issued);
    hint(xa);
  }

  // this thread's element
  const int li = 31 * warp + lane, m = mlo + li;
  const int my = m >= 0 ? m / NZ : 0, mz = m - my * NZ;
  const bool ev = m >= 0 && m < PN && my < g.ny && mz < g.nz;
  const int le = g.ny * g.nz;
  const T* Ep = P.E + (long long)pf * le + (ev ? my * g.nz + mz : 0);  // modulus of the current layer
  const unsigned char* const ucol = sm + 16 + 3 * SU * li;            // node m in slot 0, without the shift
  T* const pw = reinterpret_cast<T*>(sm + P.off_pw) + 3 * (li - 1);   // results (written by lanes >= 1): P, then W
  const T* const pr = reinterpret_cast<const T*>(sm + P.off_pw) + tid;  // read in order of the DoFs
  const int bsz = 2 * P.pw_n, cnt = 3 * (n1 - n0);

  V prev[3][2], carry[3][2], other[3][2];
  T Ecur = ev ? *Ep : (T)0;  // modulus of layer p-1 at step p
#pragma unroll
  for (int i = 0; i < 6; ++i) carry[i >> 1][i & 1].x = carry[i >> 1][i & 1].y = (T)0;
  double part = 0.0;

  // sums and differences of plane values in z and y: cur[c][py], pairs over pz
  auto transform = [&](const unsigned char* q, V (&cur)[3][2]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      V t[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const TU* q0 = reinterpret_cast<const TU*>(q + r * 3 * SU * NZ);
        T a0, a1;
        if constexpr (SU == 4 && BF) {
          const __nv_bfloat162 b0 = __floats2bfloat162_rn((float)q0[c], (float)q0[3 + c]);
          a0 = __low2float(b0);
          a1 = __high2float(b0);
        } else {
          a0 = load_u<T>(q0 + c);
          a1 = load_u<T>(q0 + 3 + c);
        }
        t[r].x = c < 2 ? a0 + a1 : a1 - a0;
        t[r].y = c < 2 ? a1 - a0 : a0 + a1;
      }
      cur[c][0] = vadd(t[0], t[1]);
      cur[c][1] = vsub(t[1], t[0]);
    }
  };
  // back transform: in z of one value pair (component c), with the neighbour lane
  auto backz = [&](int c, const V& a) -> T {
    const T even = c < 2 ? a.x : a.y, odd = c < 2 ? a.y : a.x;  // in z
    return (even - odd) + __shfl_up_sync(0xffffffffu, even + odd, 1);
  };
  // in y of component c (t0, t1: its two y-parities) into buffer b: the shares
  // of the element's lower (P) and upper (W) node row
  auto backy = [&](int c, T t0, T t1, int b) {
    if (lane > 0) {
      pw[b * bsz + c] = t0 - t1;
      pw[b * bsz + P.pw_n + c] = t0 + t1;
    }
  };
  // what the epilogue of output plane x reads; then its last addition (from
  // buffer b) and stores. Places tid + NT j of the window's DoFs.
  struct Epv {
    T r[3], d[3], x[3], u[3];
    unsigned char m[3];
  };
  auto fetch = [&](int x, Epv& v) {
    const long long base = 3 * ((long long)x * PN + n0), cb = base + co;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const unsigned i = tid + j * NT;
      if (!((int)i < cnt && topo_in_range(base + i, g.ndof))) continue;
      v.m[j] = (P.mask + base)[i];
      if constexpr (EPI == Epi::Residual) v.r[j] = (P.ep.b + cb)[i];
      if constexpr (EPI == Epi::RUpd || EPI == Epi::ChebR) v.r[j] = (P.ep.r + cb)[i];
      if constexpr (EPI == Epi::ChebR) {
        v.d[j] = (P.ep.dinv + base)[i];
        v.x[j] = (P.ep.x + cb)[i];
      }
      if constexpr (EPI == Epi::ChebR || EPI == Epi::StoreDot) v.u[j] = load_u<T>(uc + base + i);
    }
  };
  auto finish = [&](int x, int b, const Epv& v) {
    const long long base = 3 * ((long long)x * PN + n0), cb = base + co;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const unsigned i = tid + j * NT;
      if (!((int)i < cnt && topo_in_range(base + i, g.ndof))) continue;
      const bool fr = v.m[j] != 0;
      const T a = pr[b * bsz + 3 * NZ + j * NT] + pr[b * bsz + P.pw_n + j * NT];
      if constexpr (EPI == Epi::Store) {
        (yc + base)[i] = fr ? a : (T)0;
      } else if constexpr (EPI == Epi::StoreDot) {
        const T y = fr ? a : (T)0;
        (yc + base)[i] = y;
        part += (double)v.u[j] * (double)y;
      } else if constexpr (EPI == Epi::Residual) {
        (yc + base)[i] = fr ? v.r[j] - a : (T)0;
      } else if constexpr (EPI == Epi::RUpd) {
        (P.ep.r + cb)[i] = fr ? v.r[j] - P.ep.s * a : (T)0;
      } else {
        const T rv = v.r[j] - P.ep.s * a;
        const T dn = P.ep.c1 * v.u[j] + P.ep.c2 * (v.d[j] * rv);
        (P.ep.r + cb)[i] = fr ? rv : (T)0;
        (P.ep.d_out + cb)[i] = fr ? dn : (T)0;
        if (fr) (P.ep.x + cb)[i] = v.x[j] + P.ep.ax * dn;
      }
    }
  };

  int slot = staged % RING;                                          // of the current plane
  uint32_t phase = (uint32_t)((staged / RING) & 1);                  // of that slot's barrier
  int shift = (int)((((long long)pf * PN + mlo) * (3 * SU)) & 15);   // of the current plane
  const int dshift = (int)(((long long)PN * (3 * SU)) & 15);
  // wait for the current plane; also a CTA barrier: the step before has read
  // its slot and written its results
  auto arrive = [&]() -> bool {
    bool got = false;
    for (int it = 0; it < P.poll && !got; ++it) got = mbar_try(bar0 + 8u * slot, phase);
    if (!got) {
      *(volatile int*)P.err = 1;  // mapped host memory: readable without a device sync
      __threadfence_system();
    }
    return __syncthreads_and(got);
  };
  auto advance = [&]() {
    shift = (shift + dshift) & 15;
    if (++slot == RING) {
      slot = 0;
      phase ^= 1u;
    }
  };
  // step p: layer p-1 between planes p-1 (a) and p (read into b)
  auto step = [&](int p, V (&a)[3][2], V (&b)[3][2], int buf) -> bool {
    if (!arrive()) return false;
    if (tid == 0) {
      if (issued <= pl) issue(issued++);  // into the slot of plane p - 1
      if (p < xb) hint(p);
    }
    Ep += le;
    const T En = (ev && p < pl) ? *Ep : (T)0;
    // the epilogue's loads of plane p - 2 arrive behind the arithmetic of this step
    Epv ev2;
    const bool fin = p - 2 >= xa;
    if (fin) fetch(p - 2, ev2);
    transform(ucol + slot * P.slot + shift, b);
    V Ev;
    T t[3];
    Ev.x = Ev.y = Ecur;
    Ecur = En;
#pragma unroll
    for (int qy = 0; qy < 2; ++qy) {
      // the classes (0,qy,qz) and (1,qy,qz), as pairs over qz, hold both
      // x-parities of one value pair of each component
      // class (0,qy,qz): x component odd in x, y and z components even
      // class (1,qy,qz): x component even, y and z components odd
      V v0[3], v1[3];
      if constexpr (ST == 4) {
        V S[3], D[3];  // x-sum and x-difference
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int py = c == 1 ? qy ^ 1 : qy;
          S[c] = vadd(a[c][py], b[c][py]);
          D[c] = vsub(b[c][py], a[c][py]);
        }
        const V u0[3] = {D[0], S[1], S[2]}, u1[3] = {S[0], D[1], D[2]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int i0 = qy * 9 + 3 * c, i1 = (2 + qy) * 9 + 3 * c;
          v0[c] = vfma(kq<V, BF>(i0 + 2), u0[2], vfma(kq<V, BF>(i0 + 1), u0[1], vmul(kq<V, BF>(i0), u0[0])));
          v1[c] = vfma(kq<V, BF>(i1 + 2), u1[2], vfma(kq<V, BF>(i1 + 1), u1[1], vmul(kq<V, BF>(i1), u1[0])));
        }
      } else {
        // one qz after the other: half the registers
#pragma unroll
        for (int qz = 0; qz < 2; ++qz) {
          auto el = [&](const V& v) -> T { return qz ? v.y : v.x; };
          T S[3], D[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int py = c == 1 ? qy ^ 1 : qy;
            S[c] = el(a[c][py]) + el(b[c][py]);
            D[c] = el(b[c][py]) - el(a[c][py]);
          }
          const T u0[3] = {D[0], S[1], S[2]}, u1[3] = {S[0], D[1], D[2]};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int i0 = qy * 9 + 3 * c, i1 = (2 + qy) * 9 + 3 * c;
            (qz ? v0[c].y : v0[c].x) = el(kq<V, BF>(i0)) * u0[0] + el(kq<V, BF>(i0 + 1)) * u0[1] + el(kq<V, BF>(i0 + 2)) * u0[2];
            (qz ? v1[c].y : v1[c].x) = el(kq<V, BF>(i1)) * u1[0] + el(kq<V, BF>(i1 + 1)) * u1[1] + el(kq<V, BF>(i1 + 2)) * u1[2];
          }
        }
      }
      const V even[3] = {v1[0], v0[1], v0[2]}, odd[3] = {v0[0], v1[1], v1[2]};  // in x
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int py = c == 1 ? qy ^ 1 : qy;
        const T tc = backz(c, vfma(Ev, vsub(even[c], odd[c]), carry[c][py]));
        carry[c][py] = vmul(Ev, vadd(even[c], odd[c]));
        // results of plane p - 1 (not an output of this segment where p - 1 < xa)
        if (qy == 0) t[c] = tc;
        else if (c == 1) backy(c, tc, t[c], buf);
        else backy(c, t[c], tc, buf);
      }
    }
    if (fin) finish(p - 2, buf ^ 1, ev2);
    advance();
    return true;
  };

  bool ok = arrive();
  if (ok) {
    transform(ucol + slot * P.slot + shift, prev);
    advance();
  }
  // two steps per round, so that the two planes' registers swap roles
  for (int p = pf + 1; ok && p <= pl; p += 2) {
    ok = step(p, prev, other, 0);
    if (!ok || p + 1 > pl) break;
    ok = step(p + 1, other, prev, 1);
  }
  if (ok) {
    const int buf = (pl - pf) & 1;  // buffer of the next results; the other one holds plane pl - 1
    __syncthreads();
    Epv v;
    if (pl - 1 >= xa) {
      fetch(pl - 1, v);
      finish(pl - 1, buf ^ 1, v);
    }
    if (xb == g.NX) {  // the last plane has no layer above it
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T t0 = backz(c, carry[c][0]), t1 = backz(c, carry[c][1]);
        backy(c, t0, t1, buf);
      }
      fetch(g.NX - 1, v);
      __syncthreads();
      finish(g.NX - 1, buf, v);
    }
  } else if (tid == 0) {
    for (int j = max(pf, issued - RING); j < issued; ++j)
      if (!(P.skip && j == pf))
        for (int it = 0; it < P.poll && !mbar_try(bar0 + 8u * (uint32_t)((staged + j - pf) % RING),
                                                  (uint32_t)(((staged + j - pf) / RING) & 1)); ++it) {
        }
  }
  if constexpr (EPI == Epi::StoreDot) {
    double v[1] = {part};
    double tot[1];
    if (grid_sum<1>(v, P.red, tot) && tid == 0) {
      P.st->pAp = tot[0];
      P.st->alpha = P.st->rz / tot[0];
    }
  }
  if constexpr (!LINE) break;
  if (!ok) break;  // (uniform)
  count += pl - pf + 1;
  } while (at < end);
}

}  // namespace pt

// ----------------------------------------------------------------- host side
namespace {
struct PtDevice {
  // KE / KE rounded to FP32 / BF16 has the mirror symmetry (set with the device's KE)
  std::atomic<bool> sym64{false}, sym32{false}, symbf{false};
  std::atomic<int> nsm{0};
};
PerDevice<PtDevice> g_pt;

PtDevice& pt_device() {
  int dev = 0;
  TOPO_CUDA_CHECK(cudaGetDevice(&dev));
  PtDevice& d = g_pt.at(dev);
  if (d.nsm == 0) d.nsm = sm_count(dev);
  return d;
}

// Class blocks of H KE H^T / 64; false when a coupling between classes is
// above 1e-12 of the largest entry (KE then needs the general kernels). H is the
// product of three butterflies; the sums are carried in 64 bits of mantissa, so
// that a block's entry is KE's to one rounding (sums in double left up to 3.4
// ulp, which took K.u's error on a small mesh from 1.8e-16 to 4.2e-16).
bool class_blocks(const double* KE, double* K) {
  static const int corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
  static const int e[3] = {4, 2, 1};
  double top = 0.0, cross = 0.0;
  for (int c = 0; c < 3; ++c)
    for (int d = 0; d < 3; ++d) {
      long double M[8][8];  // rows and columns by corner 4 x + 2 y + z, then by parity
      for (int a = 0; a < 8; ++a)
        for (int b = 0; b < 8; ++b)
          M[4 * corner[a][0] + 2 * corner[a][1] + corner[a][2]][4 * corner[b][0] + 2 * corner[b][1] + corner[b][2]] =
              KE[(3 * a + c) * 24 + 3 * b + d];
      for (int bit = 1; bit < 8; bit *= 2)
        for (int i = 0; i < 8; ++i) {
          if (i & bit) continue;
          for (int j = 0; j < 8; ++j) {  // rows
            const long double lo = M[i][j], hi = M[i | bit][j];
            M[i][j] = lo + hi;
            M[i | bit][j] = hi - lo;
          }
        }
      for (int bit = 1; bit < 8; bit *= 2)
        for (int j = 0; j < 8; ++j) {
          if (j & bit) continue;
          for (int i = 0; i < 8; ++i) {  // columns
            const long double lo = M[i][j], hi = M[i][j | bit];
            M[i][j] = lo + hi;
            M[i][j | bit] = hi - lo;
          }
        }
      for (int p = 0; p < 8; ++p)
        for (int r = 0; r < 8; ++r) {
          const double v = (double)(M[p][r] / 64.0L);
          if (!std::isfinite(v)) return false;
          top = std::max(top, std::fabs(v));
          if ((p ^ e[c]) == (r ^ e[d])) K[(p ^ e[c]) * 9 + 3 * c + d] = v;
          else cross = std::max(cross, std::fabs(v));
        }
    }
  return cross <= 1e-12 * top;
}

// Kernel widths: the (warps per CTA, CTAs per SM) pairs an instance is
// compiled for. FP32: 512 threads per SM (128 registers each); FP64: 384 (168),
// for the Chebyshev epilogue with its five operands per DoF 256 (255). More
// threads with fewer registers spill (160x80x80: FP32 Store 24.5 us with 512
// threads per SM, 30.4 with 768, 32.5 with 1024; FP64 Chebyshev step at
// 96x48x48 18 us with 256, 23 with 384).
template <typename T, Epi EPI>
struct Width {
  static constexpr bool D = sizeof(T) == 8, C = D && EPI == Epi::ChebR;
  static constexpr int NW[3] = {4, C ? 8 : D ? 6 : 8, C ? 8 : D ? 12 : 16};
  static constexpr int PER[3] = {C ? 2 : D ? 3 : 4, C ? 1 : 2, 1};
};
constexpr int kPtSmem = 200 * 1024;  // dynamic shared memory of one CTA at most

struct PtLayout {
  int w, TO, nwin, nseg, ctas, slot, off_pw, pw_n, off_bar, total;
  double cost;  // layers times warps per SM
};

// Window width and segments. A CTA of NW warps yields 31 NW - NZ nodes per
// plane (NZ of its elements are the window's halo row) and pays one extra
// layer per segment. The three widths are compared by the layers a CTA walks
// times the warps that share its SM (at least 8: below that a step is
// latency and costs the same), over the waves of CTAs. A width that spends more
// than 3/4 of its elements on the halo is left out; with none left (NZ above
// 372, in FP64 186) the general kernels take the mesh, and where pt_pays says so.
template <typename T, Epi EPI>
bool pt_layout(const Grid& g, int s_u, bool cols, int nv, int nsm, PtLayout& best) {
  const bool line = cols && pt::line_split<T, EPI>;
  const long long PN = (long long)g.NY * g.NZ;
  if (PN >= (1 << 28) || PN * g.NX >= (1LL << 31)) return false;
  double cost = 1e300;
  for (int w = 0; w < 3; ++w) {
    const int NW = Width<T, EPI>::NW[w], TO = 31 * NW - g.NZ;
    if (TO < 31 * NW / 4) continue;
    PtLayout L;
    L.w = w;
    L.TO = TO;
    L.nwin = (int)((PN + TO - 1) / TO);
    const long long slots = (long long)nsm * Width<T, EPI>::PER[w], all = (long long)nv * L.nwin * g.NX;
    double layers, waves = 1.0;
    if (line) {
      L.nseg = 1;
      L.ctas = (int)std::max<long long>(1, std::min(slots, all / 4));
      const double part = std::ceil((double)all / L.ctas);
      layers = part + 2.0 * (1.0 + part / g.NX);  // a piece costs two: its extra layer and the start of the ring
    } else {
      const long long own = std::max<long long>(1, slots / nv);  // a column's share
      L.nseg = (int)std::max<long long>(1, std::min<long long>(g.NX, own / L.nwin));
      L.ctas = L.nwin * L.nseg;
      waves = std::ceil((double)L.ctas / (double)own);
      layers = (g.NX + L.nseg - 1) / L.nseg + 1;
    }
    const double per = std::min<double>(Width<T, EPI>::PER[w], std::ceil((double)L.ctas * (line ? 1 : nv) / nsm));
    const double c = waves * layers * std::max(8.0, per * NW);
    const auto al = [](long long x) { return (int)((x + 127) & ~127LL); };
    L.slot = al(64 + 3LL * s_u * (31 * NW + g.NZ + 3));
    L.off_pw = pt::RING * L.slot;
    L.pw_n = (3 * 31 * NW + 3) & ~3;
    L.off_bar = L.off_pw + al(4LL * L.pw_n * (int)sizeof(T));
    L.total = L.off_bar + 128;
    if (L.total <= kPtSmem / Width<T, EPI>::PER[w] && c < cost) {
      cost = L.cost = c;
      best = L;
    }
  }
  return cost < 1e300;
}

template <typename T, typename TU, bool BF, Epi EPI, int W, bool COLS>
void launch_pt_w(const PtLayout& L, const pt::Params<T>& P, cudaStream_t s) {
  auto* k = pt::k_level0_pt<T, TU, BF, EPI, COLS, Width<T, EPI>::NW[W], Width<T, EPI>::PER[W]>;
  static std::atomic<uint64_t> raised{0};  // devices where this instance's shared-memory limit is raised
  int dev = 0;
  TOPO_CUDA_CHECK(cudaGetDevice(&dev));
  if (L.total > 48 * 1024 && (dev > 63 || !(raised.load() >> dev & 1))) {
    TOPO_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtSmem));
    if (dev <= 63) raised |= 1ull << dev;
  }
  launch_chained(k, dim3((unsigned)L.ctas, COLS && !pt::line_split<T, EPI> ? (unsigned)P.nv : 1u), 32 * Width<T, EPI>::NW[W], L.total, s, P);
}

template <typename T, typename TU, bool BF, Epi EPI>
void launch_pt(const Grid& g, const void* u, const void* E, const uint8_t* mask, void* y, const EpiArgs& ea, cudaStream_t s,
               int nv = 1, long long vs = 0, const void* const* ul = nullptr, void* const* yl = nullptr) {
  PtLayout L;
  if (!pt_layout<T, EPI>(g, (int)sizeof(TU), nv > 1 || ul, nv, pt_device().nsm, L))
    throw std::runtime_error("level0 K.u: mesh not supported by the parity form");
  pt::Params<T> P;
  P.g = g;
  P.PN = g.NY * g.NZ;
  P.TO = L.TO;
  P.nwin = L.nwin;
  P.nseg = L.nseg;
  P.u = u;
  P.E = (const T*)E;
  P.mask = mask;
  P.ep = make_epi<T>(y, ea);
  P.nv = nv;
  P.vs = vs;
  P.list = ul != nullptr;
  for (int v = 0; v < 8; ++v) {
    P.ucol[v] = ul && v < nv ? ul[v] : nullptr;
    P.ycol[v] = yl && v < nv ? (T*)yl[v] : nullptr;
  }
  P.st = ea.st;
  P.red = ea.red;
  P.err = wait_error_flag();
  P.slot = L.slot;
  P.off_pw = L.off_pw;
  P.pw_n = L.pw_n;
  P.off_bar = L.off_bar;
  wait_debug(P.skip, P.poll);
  auto go = [&](auto cols) {
    constexpr bool C = decltype(cols)::value;
    switch (L.w) {
      case 0: launch_pt_w<T, TU, BF, EPI, 0, C>(L, P, s); break;
      case 1: launch_pt_w<T, TU, BF, EPI, 1, C>(L, P, s); break;
      default: launch_pt_w<T, TU, BF, EPI, 2, C>(L, P, s); break;
    }
  };
  // several columns: the V-cycle's two epilogues, and the block solve's FP64 product
  if constexpr (sizeof(TU) != 2 && (EPI == Epi::ChebR || EPI == Epi::RUpd || (EPI == Epi::Store && sizeof(T) == 8))) {
    if (nv > 1 || ul) {
      go(std::true_type{});
      return;
    }
  }
  if (nv > 1 || ul) throw std::runtime_error("level0 K.u: this form takes one column");
  go(std::false_type{});
}
}  // namespace

void pt_prepare(const double* KE) {
  double K[72] = {}, Kf[72] = {}, Kb[72] = {}, KEf[576], KEb[576];
  double2 d64[36];
  float2 f[36], fb[36];
  for (int i = 0; i < 576; ++i) {
    const float x = (float)KE[i];
    uint32_t b;
    std::memcpy(&b, &x, 4);
    b = (b + 0x7FFFu + ((b >> 16) & 1u)) & 0xFFFF0000u;
    float r;
    std::memcpy(&r, &b, 4);
    KEb[i] = r;
    KEf[i] = x;
  }
  const bool s64 = class_blocks(KE, K), s32 = class_blocks(KEf, Kf), sbf = class_blocks(KEb, Kb);
  for (int q = 0; q < 4; ++q)  // q = 2 qx + qy; class 2 q + qz
    for (int i = 0; i < 9; ++i) {
      const int e = 18 * q + i, o = e + 9;
      d64[9 * q + i] = make_double2(K[e], K[o]);
      f[9 * q + i] = make_float2((float)Kf[e], (float)Kf[o]);
      fb[9 * q + i] = make_float2((float)Kb[e], (float)Kb[o]);
    }
  TOPO_CUDA_CHECK(cudaMemcpyToSymbol(pt::cK64, d64, sizeof(d64)));
  TOPO_CUDA_CHECK(cudaMemcpyToSymbol(pt::cK32, f, sizeof(f)));
  TOPO_CUDA_CHECK(cudaMemcpyToSymbol(pt::cKbf, fb, sizeof(fb)));
  PtDevice& d = pt_device();
  d.sym64 = s64;
  d.sym32 = s32;
  d.symbf = sbf;
}

// Whether the parity form is the faster one. Its time follows pt_layout's cost c
// (B200: FP32 Store 2 us + 0.074 c, FP64 Store 5 + 0.10 c, FP64 Chebyshev step
// 3.5 + 0.168 c), which counts halo rows, the extra layer of a segment, idle SMs
// and last waves with the elements: 1.5 to 2 times the elements' own share n =
// nodes / (31 SMs) on ordinary meshes, 3 to 6 times where a window is little
// more than its halo row or barely more windows than SMs make a second wave. The
// general kernels do not pay for that. Measured with z extents from 60 to 371 at
// 60,000 and a million elements (n = 14, 225), times of the parity form against
// the other: brick kernel, FP64 Chebyshev step 114 against 115 us at c = 2.9 n,
// 207 against 123 at 5.9 n, 14.7 against 14.7 at c = 64 (n = 14), 16.8 against
// 14.6 at 80; FP32 step 62 against 62 at 3.0 n, 110 against 62 at 5.9 n.
// CUDA-core streaming kernel: 39 against 95 us at 1.5 n (FP64), 29 against 64 at
// 1.6 n (FP32), and 15 to 43 us on the small meshes against 8 to 13. Tensor-core
// kernel, whose time goes with rows and z padded to 16: plain product 37 against
// 39 us at c = 1.65 of the padded n, 37 against 35 at 1.8; Chebyshev step 47
// against 60 at 1.8.
bool pt_pays(const Grid& g, bool f64, Epi epi, int nsm, Level0Kernel other) {
  PtLayout L, narrow;
  const bool cheb = epi == Epi::ChebR;
  if (!(f64 ? pt_layout<double, Epi::ChebR>(g, 8, false, 1, nsm, narrow) : pt_layout<float, Epi::ChebR>(g, 4, false, 1, nsm, narrow)))
    return false;
  if (!f64 || cheb) L = narrow;  // (FP32: the same widths)
  else if (!pt_layout<double, Epi::Store>(g, 8, false, 1, nsm, L)) return false;
  const double n = (double)g.nnodes / (31.0 * nsm);
  switch (other) {
    case Level0Kernel::Stream: return L.cost <= 80.0 + 3.2 * n;
    case Level0Kernel::Tensor: {
      const double padded = n * ((g.NY + 15) / 16 * 16) / g.NY * ((g.NZ + 15) / 16 * 16) / g.NZ;
      return L.cost <= 48.0 + (epi == Epi::Store || epi == Epi::Residual ? 1.55 : 2.0) * padded;
    }
    default: return L.cost <= 30.0 + 2.95 * n;
  }
}

// The parity form takes this operator: the element stiffness has the mirror
// symmetry, the mesh a window layout, the copies' 16-byte alignment holds, and
// the kernel that would run instead is the slower one.
bool level0_pt_takes(const Grid& g, bool f64, bool bf, const void* u, Epi epi, Level0Kernel other) {
  const PtDevice& d = pt_device();
  return (bf ? d.symbf : f64 ? d.sym64 : d.sym32) && ((uintptr_t)u & 15) == 0 && pt_pays(g, f64, epi, d.nsm, other);
}

long long pt_dot_blocks(const Grid& g, bool f64, int nsm) {
  PtLayout L;
  const bool ok = f64 ? pt_layout<double, Epi::StoreDot>(g, 8, false, 1, nsm, L) : pt_layout<float, Epi::StoreDot>(g, 4, false, 1, nsm, L);
  return ok ? L.ctas : 0;
}

// f64: FP64 throughout; else FP32 vectors with u FP32 (bf: rounded to BF16
// where it is read) or stored BF16 (u_bf16). Epilogues as level0_apply. nv
// columns vs entries apart (u of each 16-byte aligned; ChebR and RUpd, u not
// stored BF16).
void level0_apply_pt(bool f64, bool bf, bool u_bf16, const Grid& g, const void* u, const void* E, const uint8_t* mask, void* y,
                     Epi epi, const EpiArgs& ea, cudaStream_t s, int nv, long long vs) {
#define TOPO_PT_CASE(EP)                                                                                     \
  case Epi::EP:                                                                                              \
    if (f64) launch_pt<double, double, false, Epi::EP>(g, u, E, mask, y, ea, s, nv, vs);                     \
    else if (u_bf16) launch_pt<float, __nv_bfloat16, true, Epi::EP>(g, u, E, mask, y, ea, s, nv, vs);        \
    else if (bf) launch_pt<float, float, true, Epi::EP>(g, u, E, mask, y, ea, s, nv, vs);                    \
    else launch_pt<float, float, false, Epi::EP>(g, u, E, mask, y, ea, s, nv, vs);                           \
    break;
  switch (epi) {
    TOPO_PT_CASE(Store)
    TOPO_PT_CASE(Residual)
    TOPO_PT_CASE(ChebR)
    TOPO_PT_CASE(RUpd)
    case Epi::StoreDot:
      if (nv != 1) throw std::runtime_error("level0 K.u: the dot product goes with one column");
      if (f64) launch_pt<double, double, false, Epi::StoreDot>(g, u, E, mask, y, ea, s);
      else if (!bf) launch_pt<float, float, false, Epi::StoreDot>(g, u, E, mask, y, ea, s);
      else throw std::runtime_error("level0 K.u: the dot product goes with the FP32 and FP64 operators");
      break;
  }
#undef TOPO_PT_CASE
}

// Y_v = K U_v in FP64 for nv <= 8 columns (each U_v 16-byte aligned).
void level0_columns_pt(const Grid& g, const double* const* U, const double* E, const uint8_t* mask, double* const* Y, int nv,
                       cudaStream_t s) {
  EpiArgs ea{};
  launch_pt<double, double, false, Epi::Store>(g, nullptr, E, mask, nullptr, ea, s, nv, 0, (const void* const*)U, (void* const*)Y);
}

bool pt_class_blocks(const double* KE, double* K) { return class_blocks(KE, K); }

TOPO_BOUNDS_READER(bounds_flag_pt)

}  // namespace topo
