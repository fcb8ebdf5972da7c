// Jacobi-preconditioned CG of a small level inside one thread-block cluster:
// the whole solve -- operator, DSS, inner products, updates, stop -- in one
// launch, with the level's vectors in the shared memory (or registers) of up
// to 16 SMs.
//
// A small level is latency bound, not bandwidth bound: as three launches an
// iteration (operator, DSS, update) the 4^3 periodic box at n = 8 takes
// 17.8 us an iteration, and as one cooperative launch with three grid-wide
// barriers the n = 4 level under it takes 14.8 us, for 4,096 points.  In a
// cluster a barrier is a hardware barrier over at most 16 SMs, a neighbour
// element's copy of a node is one load from L2 (the exchanged vector is the
// only one in global memory: gathered from distributed shared memory, a warp's
// scattered loads took 15 cycles each), and the sums of an iteration travel
// as one value per SM through distributed shared memory.
//
// Arithmetic: conjugate_gradient with jacobi_preconditioner
// (src/solver.c:33-81, src/precon.c:311-324) as cg_solve's kernels do it --
// the same rounding to the storage type T, the DSS in the reference's order,
// FP64 sums -- except that where p is the same in all copies of a node (the
// levels below level 0, and level 0 for a right-hand side that is; FP32 as in
// its kernels) p.(A p) is summed over the element copies before the DSS, equal
// to the weighted product, so that it is known at the same barrier as the
// operator's output; other FP64 solves take (p w).ap of the assembled ap and
// one more barrier (12 % of a Helmholtz solve).  Every block adds
// the blocks' partial sums in rank order, so all take the same alpha, beta and
// stop decision.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "kernels.cuh"
#include "ssg_internal.h"
#include "ssg_kernels.h"

namespace ssg {
namespace dev {

constexpr int kClusterMax = 16;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// address of the same shared variable in the cluster's block `rank`
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void st_cluster(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// all threads of all blocks; shared-memory writes before it are visible to
// every block of the cluster after it
__device__ __forceinline__ void cluster_sync() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n"
      "barrier.cluster.wait.acquire.aligned;\n" ::
          : "memory");
}

// Sums over the cluster, NQ values a thread: the warp, the block's warps,
// then one value per block in every block's slots.  post() ends with the
// block's sums sent; after a cluster_sync, sum() adds the blocks' values, in
// the same order in every warp of every block.  The two buffers alternate so that a block
// may post the next sums while another still reads the last.
struct ClusterRed {
  double warp[4 * 16];
  double slot[2][4 * kClusterMax];
  double max_warp[2 * 16], max_slot[2 * kClusterMax];   // red_max, once a launch
};

// sum of v over the warp, in every lane: two tensor-core products with ones
// (quad sums of the lanes as B, then the sum over the quads as A) in place of
// five dependent shuffle-and-add steps
__device__ __forceinline__ double warp_sum(double v) {
  double c0, c1;
  dmma(c0, c1, 1.0, v, 0.0, 0.0);       // C[.][n] = v[4n] + .. + v[4n + 3]
  dmma(c0, c1, c0 + c1, 1.0, 0.0, 0.0);  // lane t of a quad holds quads 2t, 2t + 1
  return c0;
}

template <int NQ>
__device__ __forceinline__ void red_post(ClusterRed& s, int buf, double (&v)[NQ], int cs,
                                         uint32_t rank) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = warp_sum(v[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) s.warp[q * 16 + wid] = v[q];
  __syncthreads();
  if (wid == 0) {   // (at most 16 warps)
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = warp_sum(lane < nw ? s.warp[q * 16 + lane] : 0.0);
    if (lane < cs)
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        st_cluster(map_rank(smem_addr(&s.slot[buf][q * kClusterMax + rank]), lane), v[q]);
  }
}

template <int NQ>
__device__ __forceinline__ void red_sum(const ClusterRed& s, int buf, int cs, double (&v)[NQ]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    v[q] = warp_sum(lane < cs ? s.slot[buf][q * kClusterMax + lane] : 0.0);
}

// The maxima of two values a thread over the cluster: post() ends with the
// block's sent, max() is for after a cluster_sync (once a launch).
__device__ __forceinline__ void max_post(ClusterRed& s, double (&v)[2], int cs, uint32_t rank) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] = fmax(v[q], __shfl_xor_sync(0xffffffffu, v[q], o));
    if (lane == 0) s.max_warp[q * 16 + wid] = v[q];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double m = 0.0;
    for (int w = 0; w < nw; ++w) m = fmax(m, s.max_warp[lane * 16 + w]);
    for (int b = 0; b < cs; ++b)
      st_cluster(map_rank(smem_addr(&s.max_slot[lane * kClusterMax + rank]), b), m);
  }
}

__device__ __forceinline__ void max_get(const ClusterRed& s, int cs, double (&v)[2]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    v[q] = 0.0;
    for (int b = 0; b < cs; ++b) v[q] = fmax(v[q], s.max_slot[q * kClusterMax + b]);
  }
}

// ---------------------------------------------------------------------------
// general order: elements in shared memory, line-form operator
// ---------------------------------------------------------------------------
template <typename T>
struct ClusterCgArgs {
  int nel = 0, epc = 0, cs = 1;   // elements, elements per block, blocks
  T* f = nullptr;                 // masked in place
  T* x = nullptr;                 // initial guess in, solution out
  T* ex = nullptr;                // exchanged operator output (global: stays in L2)
  const T* gf = nullptr;
  size_t npts = 0;
  const double* bj = nullptr;     // Helmholtz: rho J
  const double *D = nullptr, *S = nullptr;
  double lambda = 0.0;
  const T* dinv = nullptr;
  const uint8_t* mult = nullptr;
  const double* mask = nullptr;
  const int* dss = nullptr;       // DSS map (dss_map_table)
  AffGeom ag;
  int helm = 0, pressure = 0;
  int weighted = 0;               // alpha from the assembled A p (kAlpha*)
  int sgeom = 0;                  // per-point factors in shared memory
  double nunique = 1.0, eps = 0.0;
  int max_iter = 0;
  double* frame = nullptr;
  double* hist = nullptr;
  int hist_cap = 0;
};

template <int N, typename T>
struct ClusterLevel {
  static constexpr int NT = N * N * N, NN = N * N;
  // field rows of odd length: lines along i by lanes walking j hit distinct
  // banks; point q sits at q + q / N (even N) or q
  static constexpr int RS = N + 1 - N % 2, FS = NN * RS;
  static constexpr int RM = N + (N & 1);   // matrix rows (pair-aligned)
  static constexpr int MATS = (4 * N * RM + 3) / 4 * 4;
  static constexpr int RHO = (NT + 3) / 4 * 4;   // weight products (affine)
  // an element's face-interior, edge-interior nodes and their DSS sources:
  // one, three and (corners) seven a node
  static constexpr int I = N - 2, NF = 6 * I * I, NE = 12 * I, SRC = NF + 3 * NE + 56;
  __host__ __device__ static size_t values(int epc, bool aff, bool sgeom) {
    return MATS + (aff ? RHO : 0) +
           (size_t)epc * (4 * FS + 3 * NT + (aff ? 6 : (sgeom ? 6 * NT : 0)));
  }
  static size_t bytes(int epc, bool aff, bool sgeom) {
    return (sizeof(T) * values(epc, aff, sgeom) + 7) / 8 * 8 + (size_t)epc * (4 * SRC + NT);
  }
};

// y = A x with every output its own chain of multiply-adds; A rows of RM
template <int N, int RM, typename T>
__device__ __forceinline__ void line_full(const T* A, const T (&x)[N], T (&y)[N]) {
  using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
#pragma unroll
  for (int o = 0; o < N; ++o) y[o] = 0;
#pragma unroll
  for (int l = 0; l + 1 < N; l += 2)
#pragma unroll
    for (int o = 0; o < N; ++o) {
      const V2 m = *reinterpret_cast<const V2*>(A + o * RM + l);
      y[o] += m.x * x[l];
      y[o] += m.y * x[l + 1];
    }
  if (N & 1)
#pragma unroll
    for (int o = 0; o < N; ++o) y[o] += A[o * RM + N - 1] * x[N - 1];
}

template <int N, typename T>
__global__ void __launch_bounds__(512) k_cluster_cg(ClusterCgArgs<T> a) {
  using C = ClusterLevel<N, T>;
  constexpr int NN = N * N, NT = C::NT, RS = C::RS, FS = C::FS, RM = C::RM;
  constexpr int NF = C::NF, NE = C::NE, SRC = C::SRC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ClusterRed red;
  const uint32_t rank = cluster_rank();
  const int cs = a.cs, epc = a.epc;
  const int e0 = (int)rank * epc, ne = max(0, min(epc, a.nel - e0));
  // (FP32 reads its stored factors, each one rounding of the FP64 value)
  const bool aff = sizeof(T) == 8 && a.ag.c != nullptr;
  T* const sD = reinterpret_cast<T*>(smem_raw);
  T* const sDT = sD + N * RM;
  T* const sS = sDT + N * RM;
  T* const sST = sS + N * RM;
  T* const U = sD + C::MATS;            // the direction p
  T* const F1 = U + (size_t)epc * FS;   // A_e p
  T* const F2 = F1 + (size_t)epc * FS;  // its DSS
  T* const F3 = F2 + (size_t)epc * FS;
  T* const X = F3 + (size_t)epc * FS;   // natural order from here
  T* const Rv = X + (size_t)epc * NT;
  T* const DI = Rv + (size_t)epc * NT;
  T* const CG = DI + (size_t)epc * NT;                    // affine: 6 constants an element
  T* const RHO = CG + (aff ? (size_t)epc * 6 : 0);        //   and the weight products
  T* const G = CG;                                        // else 6 factors a point (sgeom)
  // sources: [ne][NF], [ne][NE][3], [ne][8][7]; then the multiplicities
  int* const src = reinterpret_cast<int*>(
      smem_raw + (sizeof(T) * C::values(epc, aff, a.sgeom != 0) + 7) / 8 * 8);
  int* const esrc = src + (size_t)ne * NF;
  int* const csrc = esrc + (size_t)ne * NE * 3;
  uint8_t* const MU = reinterpret_cast<uint8_t*>(src + (size_t)epc * SRC);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const size_t g0 = (size_t)e0 * NT;    // first point of this block
  const int np = ne * NT, nlines = ne * NN;
  // position of point q in a padded field
  auto at = [](int q) { return RS == N ? q : q + q / N; };
  for (int q = tid; q < NN; q += nthr) {
    const int r = q / N, c = q % N;
    const T d = (T)a.D[q], sv = (T)a.S[q];   // (S = D for the Laplacian)
    sD[r * RM + c] = d;
    sDT[c * RM + r] = d;
    sS[r * RM + c] = sv;
    sST[c * RM + r] = sv;
  }
  for (int q = tid; q < np; q += nthr) {
    const T xv = a.x[g0 + q];
    X[q] = xv;
    U[at(q)] = xv;
    DI[q] = a.dinv[g0 + q];
    MU[q] = a.mult[g0 + q];
    if (!aff && a.sgeom)
#pragma unroll
      for (int c = 0; c < 6; ++c) G[(size_t)c * epc * NT + q] = a.gf[c * a.npts + g0 + q];
  }
  if (aff) {
    for (int q = tid; q < ne * 6; q += nthr) CG[q] = (T)__ldg(a.ag.c + 6 * (size_t)e0 + q);
    for (int q = tid; q < NT; q += nthr)
      RHO[q] = (T)((__ldg(a.ag.w + q % N) * __ldg(a.ag.w + (q / N) % N)) * __ldg(a.ag.w + q / NN));
  }
  // the DSS map's sources of this block's boundary nodes (gather words; edge
  // and corner records), -1 for none
  {
    const int* rec0 = a.dss + dss_map_records_offset(a.npts) + (size_t)e0 * (12 * C::I * 4 + 64);
    for (int t = tid; t < ne * NF; t += nthr) {
      const int e = t / NF;
      src[t] = __ldg(a.dss + g0 + e * NT + class_ordered_node<N>(t - e * NF));
    }
    for (int t = tid; t < ne * NE * 3; t += nthr) {
      const int n = t / 3, e = n / NE;
      esrc[t] = __ldg(rec0 + (size_t)e * (12 * C::I * 4 + 64) + (n - e * NE) * 4 + t % 3);
    }
    for (int t = tid; t < ne * 56; t += nthr) {
      const int n = t / 7, e = n / 8;
      csrc[t] = __ldg(rec0 + (size_t)e * (12 * C::I * 4 + 64) + 12 * C::I * 4 + (n & 7) * 8 +
                      t % 7);
    }
  }
  const T* const gp0 = a.sgeom ? G : a.gf + g0;           // factor c at gp0 + c * gs
  const size_t gs = a.sgeom ? (size_t)epc * NT : a.npts;
  __syncthreads();
  // kAlphaAsk: the largest |f| and the largest difference between copies of a
  // node (before any block masks its f); not a number counts as infinite
  double span[2] = {0.0, 0.0};
  if (a.weighted == kAlphaAsk) {
    auto gap = [&](int q, int p) {
      if (p < 0) return;
      const double d = fabs((double)a.f[g0 + q] - (double)a.f[p]);
      span[1] = fmax(span[1], isnan(d) ? CUDART_INF : d);
    };
    for (int q = tid; q < np; q += nthr) span[0] = fmax(span[0], fabs((double)a.f[g0 + q]));
    for (int t = tid; t < ne * NF; t += nthr) {
      const int e = t / NF;
      gap(e * NT + class_ordered_node<N>(t - e * NF), src[t]);
    }
    for (int t = tid; t < ne * NE * 3; t += nthr) {
      const int n = t / 3, e = n / NE;
      gap(e * NT + class_ordered_node<N>(NF + n - e * NE), esrc[t]);
    }
    for (int t = tid; t < ne * 56; t += nthr) {
      const int n = t / 7, e = n / 8;
      gap(e * NT + corner_node(N, n & 7), csrc[t]);
    }
  }

  // the block's points four at a time: f(points, field positions, valid); the
  // four are read before any is written, so their chains overlap (one point
  // at a time a pass over 8 points a thread took 2000 cycles).  Points past
  // the end repeat the last one.
  auto points = [&](auto&& f) {
    for (int q0 = tid; q0 < np; q0 += 4 * nthr) {
      int q[4], o[4];
      bool ok[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        ok[h] = q0 + h * nthr < np;
        q[h] = ok[h] ? q0 + h * nthr : np - 1;
        o[h] = at(q[h]);
      }
      f(q, o, ok);
    }
  };

  // F2 = the exchanged vector = mask .* A_e U; returns this thread's share of U . F1
  auto op = [&]() -> double {
    // r-derivatives (S for Helmholtz) of the lines along i, s-derivatives of
    // the lines along j
    for (int t = tid; t < nlines; t += nthr) {
      const int e = t / NN, r = t - e * NN, a0 = r % N, a1 = r / N;
      T x[N], y[N];
      const int oi = t * RS, oj = e * FS + a1 * N * RS + a0;
#pragma unroll
      for (int l = 0; l < N; ++l) x[l] = U[oi + l];
      line_full<N, RM, T>(sS, x, y);
#pragma unroll
      for (int l = 0; l < N; ++l) F1[oi + l] = y[l];
#pragma unroll
      for (int l = 0; l < N; ++l) x[l] = U[oj + l * RS];
      line_full<N, RM, T>(sD, x, y);
#pragma unroll
      for (int l = 0; l < N; ++l) F2[oj + l * RS] = y[l];
    }
    __syncthreads();
    // lines along k: t-derivative, metric product, t-transposed part
    for (int t = tid; t < nlines; t += nthr) {
      const int e = t / NN, r = t - e * NN;
      const int q0 = e * FS + at(r);
      T x[N], ut[N];
#pragma unroll
      for (int l = 0; l < N; ++l) x[l] = U[q0 + l * N * RS];
      line_full<N, RM, T>(sD, x, ut);
      T cg[6];
      if (aff) {
#pragma unroll
        for (int c = 0; c < 6; ++c) cg[c] = CG[6 * e + c];
      }
      const T* gp = gp0 + (size_t)e * NT + r;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const int q = q0 + k * N * RS;
        const T ur = F1[q], us = F2[q];
        T h[6];
        if (aff) {
          const T rho = RHO[k * NN + r];
#pragma unroll
          for (int c = 0; c < 6; ++c) h[c] = cg[c] * rho;
        } else {
#pragma unroll
          for (int c = 0; c < 6; ++c) h[c] = gp[c * gs + k * NN];
        }
        F1[q] = h[0] * ur + h[1] * us + h[2] * ut[k];
        F2[q] = h[1] * ur + h[3] * us + h[4] * ut[k];
        x[k] = h[2] * ur + h[4] * us + h[5] * ut[k];
      }
      line_full<N, RM, T>(sST, x, ut);
#pragma unroll
      for (int k = 0; k < N; ++k) F3[q0 + k * N * RS] = ut[k];
    }
    __syncthreads();
    // transposed r and s parts, in place
    for (int t = tid; t < nlines; t += nthr) {
      const int e = t / NN, r = t - e * NN, a0 = r % N, a1 = r / N;
      const int oi = t * RS, oj = e * FS + a1 * N * RS + a0;
      T x[N], y[N];
#pragma unroll
      for (int l = 0; l < N; ++l) x[l] = F1[oi + l];
      line_full<N, RM, T>(sDT, x, y);
#pragma unroll
      for (int l = 0; l < N; ++l) F1[oi + l] = y[l];
#pragma unroll
      for (int l = 0; l < N; ++l) x[l] = F2[oj + l * RS];
      line_full<N, RM, T>(sST, x, y);
#pragma unroll
      for (int l = 0; l < N; ++l) F2[oj + l * RS] = y[l];
    }
    __syncthreads();
    double pap = 0.0;
    points([&](const int (&q)[4], const int (&o)[4], const bool (&ok)[4]) {
      T uv[4], out[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        uv[h] = U[o[h]];
        out[h] = (F1[o[h]] + F2[o[h]]) + F3[o[h]];
        if (a.helm) out[h] += (T)a.lambda * ((T)__ldg(a.bj + g0 + q[h]) * uv[h]);
        if (a.mask) out[h] = (T)((double)out[h] * __ldg(a.mask + g0 + q[h]));
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (ok[h]) {
          F2[o[h]] = out[h];
          a.ex[g0 + q[h]] = out[h];
          pap += (double)uv[h] * (double)out[h];
        }
    });
    return pap;
  };
  // F2 = its DSS (after a cluster_sync): each boundary node its sources in the
  // reference's order
  auto other = [&](int p) -> T { return p >= 0 ? __ldcg(a.ex + p) : T(0); };
  auto dss = [&]() {
    const int n1 = ne * NF, n2 = ne * NE, n3 = n2 + ne * 8;
    for (int t0 = tid; t0 < n1; t0 += 4 * nthr) {
      double v[4], w[4];
      int o[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int t = min(t0 + h * nthr, n1 - 1), e = t / NF;
        v[h] = (double)other(src[t]);
        o[h] = at(e * NT + class_ordered_node<N>(t - e * NF));
        w[h] = (double)F2[o[h]];
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (t0 + h * nthr < n1) F2[o[h]] = (T)(w[h] + v[h]);
    }
    for (int t = tid; t < n3; t += nthr) {
      if (t < n2) {
        const int e = t / NE;
        const int o = at(e * NT + class_ordered_node<N>(NF + t - e * NE));
        const double v0 = (double)other(esrc[3 * t]);
        const double v1 = (double)other(esrc[3 * t + 1]);
        const double v2 = (double)other(esrc[3 * t + 2]);
        F2[o] = (T)((((double)F2[o] + v0) + v1) + v2);
      } else {
        const int u = t - n2, e = u / 8;
        const int o = at(e * NT + corner_node(N, u & 7));
        double v[7];
#pragma unroll
        for (int m = 0; m < 7; ++m) v[m] = (double)other(csrc[7 * u + m]);
        double acc = (double)F2[o];
#pragma unroll
        for (int m = 0; m < 7; ++m) acc += v[m];
        F2[o] = (T)acc;
      }
    }
    __syncthreads();
  };
  int buf = 0;

  // r = f - DSS(A x); nullspace of r (pressure)
  op();
  cluster_sync();
  dss();
  {
    double s[1] = {0.0};
    for (int q = tid; q < np; q += nthr) {
      double fv = (double)a.f[g0 + q];
      if (a.mask) {
        const T fm = (T)(fv * __ldg(a.mask + g0 + q));
        a.f[g0 + q] = fm;
        fv = (double)fm;
      }
      const T rv = (T)(fv + -(double)F2[at(q)]);
      Rv[q] = rv;
      s[0] += (double)rv * inv_count(MU[q]);
    }
    red_post<1>(red, buf, s, cs, rank);
    if (a.weighted == kAlphaAsk) max_post(red, span, cs, rank);
  }
  cluster_sync();
  bool weighted = a.weighted != kAlphaPlain;
  if (a.weighted == kAlphaAsk) {
    max_get(red, cs, span);
    weighted = !(span[1] <= 1.4e-14 * span[0]);
  }
  double cz = 0.0, rdz = 0.0, beta = 0.0, err = 0.0, err0 = 0.0;
  {
    double s[1];
    red_sum<1>(red, buf, cs, s);
    buf ^= 1;
    const double nc = a.pressure ? -(s[0] / a.nunique) : 0.0;
    double z[1] = {0.0};
    for (int q = tid; q < np; q += nthr) {
      T rv = Rv[q];
      if (a.pressure) {
        rv = (T)((double)rv + nc);
        Rv[q] = rv;
      }
      const T zq = (T)((double)rv * (double)DI[q]);
      z[0] += (double)zq * inv_count(MU[q]);
    }
    red_post<1>(red, buf, z, cs, rank);
    cluster_sync();
    red_sum<1>(red, buf, cs, s);
    buf ^= 1;
    if (a.pressure) cz = s[0] / a.nunique;
  }
  int it = 0;
  for (; it < a.max_iter; ++it) {
    const bool first = it == 0;
    // p = beta p + (z - c) (first: z - c), masked
    double d[3] = {0.0, 0.0, 0.0};
    points([&](const int (&q)[4], const int (&o)[4], const bool (&ok)[4]) {
      double rv[4];
      T pt[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        rv[h] = (double)Rv[q[h]];
        const double zc = (double)(T)(rv[h] * (double)DI[q[h]]) - cz;
        double pv = first ? zc : beta * (double)U[o[h]] + zc;
        if (a.mask) pv = pv * __ldg(a.mask + g0 + q[h]);
        pt[h] = (T)pv;
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (ok[h]) {
          U[o[h]] = pt[h];
          if (first) {   // (r w).p and (r w).r
            const double rw = rv[h] * inv_count(MU[q[h]]);
            d[1] += rw * (double)pt[h];
            d[2] += rw * rv[h];
          }
        }
    });
    __syncthreads();
    d[0] = op();
    if (weighted) {
      // (p w).ap of the assembled ap: one more barrier
      cluster_sync();
      dss();
      d[0] = 0.0;
      points([&](const int (&q)[4], const int (&o)[4], const bool (&ok)[4]) {
        double pa[4];
#pragma unroll
        for (int h = 0; h < 4; ++h)
          pa[h] = ((double)U[o[h]] * inv_count(MU[q[h]])) * (double)F2[o[h]];
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (ok[h]) d[0] += pa[h];
      });
    }
    if (first) {
      red_post<3>(red, buf, d, cs, rank);
    } else {
      double s[1] = {d[0]};
      red_post<1>(red, buf, s, cs, rank);
    }
    cluster_sync();
    if (!weighted) dss();
    if (first) {
      red_sum<3>(red, buf, cs, d);
      rdz = d[1];
      err0 = sqrt(d[2]);
    } else {
      double s[1];
      red_sum<1>(red, buf, cs, s);
      d[0] = s[0];
    }
    buf ^= 1;
    const double alpha = rdz / d[0];
    // x += alpha p; r -= alpha ap; z = dinv r
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    points([&](const int (&q)[4], const int (&o)[4], const bool (&ok)[4]) {
      T xv[4], rq[4];
      double zq[4], w[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        xv[h] = (T)((double)X[q[h]] + alpha * (double)U[o[h]]);
        rq[h] = (T)((double)Rv[q[h]] + -alpha * (double)F2[o[h]]);
        zq[h] = (double)(T)((double)rq[h] * (double)DI[q[h]]);
        w[h] = ok[h] ? inv_count(MU[q[h]]) : 0.0;
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (ok[h]) {
          X[q[h]] = xv[h];
          Rv[q[h]] = rq[h];
          const double rw = (double)rq[h] * w[h];
          s[0] += rw * zq[h];
          s[1] += rw * (double)rq[h];
          s[2] += w[h] * zq[h];
          s[3] += rw;
        }
    });
    red_post<4>(red, buf, s, cs, rank);
    cluster_sync();
    red_sum<4>(red, buf, cs, s);
    buf ^= 1;
    if (a.pressure) cz = s[2] / a.nunique;
    const double rdz_new = s[0] - cz * s[3];
    beta = rdz_new / rdz;
    rdz = rdz_new;
    err = sqrt(s[1]);
    if (rank == 0 && tid == 0 && a.hist && it < a.hist_cap) a.hist[it] = err;
    if (!(err > a.eps) || it + 1 >= a.max_iter) {
      ++it;
      break;
    }
  }
  for (int q = tid; q < np; q += nthr) a.x[g0 + q] = X[q];
  if (rank == 0 && tid == 0) {
    a.frame[F_ITER] = (double)it;
    a.frame[F_ERR] = err;
    a.frame[F_ERR0] = err0;
    a.frame[F_DONE] = 1.0;
  }
  // (the last cluster_sync is after every read of another block's memory)
}

// ---------------------------------------------------------------------------
// n = 2: one to KP points a thread in registers, an element's 8 points in 8
// lanes (the operator by shuffles, as the cooperative kernel's point_op2);
// the exchanged operator output is the only vector in memory
// ---------------------------------------------------------------------------
struct ClusterCoarseArgs {
  int nel = 0, epc = 0, cs = 1;
  const double* f = nullptr;
  double* x = nullptr;
  double* ex = nullptr;   // exchanged operator output (global: stays in L2)
  const double* gf = nullptr;
  size_t npts = 0;
  const double* D = nullptr;
  const double* dinv = nullptr;
  const int2* pairs = nullptr;
  double nunique = 1.0, eps = 0.0, rel = 0.0;
  int max_iter = 0;
  double* frame = nullptr;
};

constexpr int kCoarseThreads = 512;

template <int KP>
__global__ void __launch_bounds__(kCoarseThreads) k_cluster_coarse(ClusterCoarseArgs a) {
  constexpr unsigned full = 0xffffffffu;
  // the metric in registers up to two points a thread, else in shared memory
  constexpr bool GREG = KP <= 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ClusterRed red;
  const uint32_t rank = cluster_rank();
  const int cs = a.cs, epc = a.epc, npl = epc * 8;
  double* const sg = reinterpret_cast<double*>(smem_raw);   // [6][npl] when !GREG
  const int e0 = (int)rank * epc, ne = max(0, min(epc, a.nel - e0));
  const size_t g0 = (size_t)e0 * 8;
  const int np = ne * 8, tid = threadIdx.x, q3 = tid & 7;
  const int i = q3 & 1, j = (q3 >> 1) & 1, k = q3 >> 2;
  double* const ex = a.ex + g0;
  // D rows of this lane's coordinates: own and partner entries, and columns
  double df[3][2], db[3][2];
  {
    const int c3[3] = {i, j, k};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      df[b][0] = __ldg(a.D + c3[b] * 2);
      df[b][1] = __ldg(a.D + c3[b] * 2 + 1);
      db[b][0] = __ldg(a.D + c3[b]);
      db[b][1] = __ldg(a.D + 2 + c3[b]);
    }
  }
  double x[KP], r[KP], z[KP], p[KP], di[KP], w[KP], own[KP];
  double g[GREG ? KP : 1][6];
  int src[KP][7];
#pragma unroll
  for (int s = 0; s < KP; ++s) {
    const int l = tid + s * kCoarseThreads;
    const bool ok = l < np;
    const size_t o = g0 + l;
    x[s] = ok ? a.x[o] : 0.0;
    di[s] = ok ? a.dinv[o] : 0.0;
    r[s] = z[s] = p[s] = 0.0;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const double v = ok ? __ldg(a.gf + c * a.npts + o) : 0.0;
      if (GREG)
        g[s][c] = v;
      else if (l < npl)
        sg[c * npl + l] = v;
    }
    // the node's DSS sources in the reference's order (faces x, y, z, edges
    // xy, xz, yz, corner); absent ones read a zero
    int cnt = 0;
#pragma unroll
    for (int m = 0; m < 7; ++m) src[s][m] = -1;
    if (ok) {
      const int2* pr = a.pairs + (size_t)(e0 + (l >> 3)) * 26;
      auto put = [&](int m, int2 pp, int node) {
        if (pp.x < 0) return;
        src[s][m] = pp.x * 8 + node;
        ++cnt;
      };
      int2 pp = pr[i];
      put(0, pp, face_node(2, pp.y, k, j));
      pp = pr[2 + j];
      put(1, pp, face_node(2, pp.y, k, i));
      pp = pr[4 + k];
      put(2, pp, face_node(2, pp.y, j, i));
      pp = pr[6 + (i | (j << 1))];
      put(3, pp, edge_node(2, pp.y, k));
      pp = pr[10 + (i | (k << 1))];
      put(4, pp, edge_node(2, pp.y, j));
      pp = pr[14 + (j | (k << 1))];
      put(5, pp, edge_node(2, pp.y, i));
      pp = pr[18 + q3];
      put(6, pp, corner_node(2, pp.y));
    }
    w[s] = ok ? inv_count(1u + (unsigned)cnt) : 0.0;
  }
  __syncthreads();

  // A_e v of this lane's point: two-term sums over the partner lane, metric
  // products, transposed two-term sums (m = 0 first, then m = 1)
  auto op = [&](double v, int s) -> double {
    const double vr = __shfl_xor_sync(full, v, 1), vs = __shfl_xor_sync(full, v, 2),
                 vt = __shfl_xor_sync(full, v, 4);
    auto two = [](const double (&d)[2], int c, double own, double other) {
      return fma(d[1], c ? own : other, d[0] * (c ? other : own));
    };
    const double ur = two(df[0], i, v, vr), us = two(df[1], j, v, vs), ut = two(df[2], k, v, vt);
    double h[6];
    if (GREG) {
#pragma unroll
      for (int c = 0; c < 6; ++c) h[c] = g[GREG ? s : 0][c];
    } else {
      const int l = tid + s * kCoarseThreads;
#pragma unroll
      for (int c = 0; c < 6; ++c) h[c] = l < np ? sg[c * npl + l] : 0.0;
    }
    const double w0 = h[0] * ur + h[1] * us + h[2] * ut;
    const double w1 = h[1] * ur + h[3] * us + h[4] * ut;
    const double w2 = h[2] * ur + h[4] * us + h[5] * ut;
    const double o0 = __shfl_xor_sync(full, w0, 1), o1 = __shfl_xor_sync(full, w1, 2),
                 o2 = __shfl_xor_sync(full, w2, 4);
    return (two(db[0], i, w0, o0) + two(db[1], j, w1, o1)) + two(db[2], k, w2, o2);
  };
  auto gather = [&](int s) -> double {
    const int l = tid + s * kCoarseThreads;
    double v[7];
#pragma unroll
    for (int m = 0; m < 7; ++m) v[m] = src[s][m] >= 0 ? __ldcg(a.ex + src[s][m]) : 0.0;
    double acc = l < np ? own[s] : 0.0;
#pragma unroll
    for (int m = 0; m < 7; ++m) acc += v[m];   // (adding 0.0 changes nothing)
    return acc;
  };
  int buf = 0;

#pragma unroll
  for (int s = 0; s < KP; ++s) {
    const double o = op(x[s], s);
    own[s] = o;
    if (tid + s * kCoarseThreads < np) ex[tid + s * kCoarseThreads] = o;
  }
  cluster_sync();
  double t1[1] = {0.0};
#pragma unroll
  for (int s = 0; s < KP; ++s) {
    const int l = tid + s * kCoarseThreads;
    const double acc = gather(s);
    r[s] = l < np ? a.f[g0 + l] + -acc : 0.0;
    t1[0] += r[s] * w[s];
  }
  red_post<1>(red, buf, t1, cs, rank);
  cluster_sync();
  red_sum<1>(red, buf, cs, t1);
  buf ^= 1;
  const double c0 = t1[0] / a.nunique;
  t1[0] = 0.0;
#pragma unroll
  for (int s = 0; s < KP; ++s) {
    r[s] = tid + s * kCoarseThreads < np ? r[s] + -c0 : 0.0;
    z[s] = r[s] * di[s];
    t1[0] += z[s] * w[s];
  }
  red_post<1>(red, buf, t1, cs, rank);
  cluster_sync();
  red_sum<1>(red, buf, cs, t1);
  buf ^= 1;
  double cz = t1[0] / a.nunique, rdz = 0.0, beta = 0.0, err = 0.0, err0 = 0.0;
  int it = 0;
  for (; it < a.max_iter; ++it) {
    const bool first = it == 0;
    double d[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < KP; ++s) {
      const int l = tid + s * kCoarseThreads;
      const double zc = z[s] - cz;
      p[s] = l < np ? (first ? zc : beta * p[s] + zc) : 0.0;
      const double o = op(p[s], s);
      own[s] = o;
      if (l < np) ex[l] = o;
      d[0] += p[s] * o;
      if (first) {
        const double rw = r[s] * w[s];
        d[1] += rw * p[s];
        d[2] += rw * r[s];
      }
    }
    if (first) {
      red_post<3>(red, buf, d, cs, rank);
    } else {
      double s1[1] = {d[0]};
      red_post<1>(red, buf, s1, cs, rank);
    }
    cluster_sync();
    double ap[KP];
#pragma unroll
    for (int s = 0; s < KP; ++s) ap[s] = gather(s);
    if (first) {
      red_sum<3>(red, buf, cs, d);
      rdz = d[1];
      err0 = sqrt(d[2]);
    } else {
      double s1[1];
      red_sum<1>(red, buf, cs, s1);
      d[0] = s1[0];
    }
    buf ^= 1;
    const double alpha = rdz / d[0];
    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < KP; ++s) {
      x[s] = x[s] + alpha * p[s];
      r[s] = r[s] + -alpha * ap[s];
      z[s] = r[s] * di[s];
      const double rw = r[s] * w[s];
      v[0] += rw * z[s];
      v[1] += rw * r[s];
      v[2] += w[s] * z[s];
      v[3] += rw;
    }
    red_post<4>(red, buf, v, cs, rank);
    cluster_sync();
    red_sum<4>(red, buf, cs, v);
    buf ^= 1;
    cz = v[2] / a.nunique;
    const double rdz_new = v[0] - cz * v[3];
    beta = rdz_new / rdz;
    rdz = rdz_new;
    err = sqrt(v[1]);
    if (!(err > a.eps) || !(err > a.rel * err0) || it + 1 >= a.max_iter) {
      ++it;
      break;
    }
  }
#pragma unroll
  for (int s = 0; s < KP; ++s)
    if (tid + s * kCoarseThreads < np) a.x[g0 + tid + s * kCoarseThreads] = x[s];
  if (rank == 0 && tid == 0) {
    a.frame[F_ITER] = (double)it;
    a.frame[F_ERR] = err;
    a.frame[F_ERR0] = err0;
    a.frame[F_DONE] = 1.0;
  }
}

}  // namespace dev

namespace {

constexpr int kMaxDev = 64;
constexpr size_t kSmemMax = 224 * 1024;   // dynamic shared memory of a block (the static part is 2 KB)

// Largest cluster of a kernel at full shared memory, per device: 16 where
// the device can place it, else 8 (the portable size).  Filled on first use;
// a race repeats the same queries.
struct ClusterAttr {
  std::atomic<int> most[kMaxDev] = {};
  cudaError_t ensure(const void* kern, int threads, size_t smem, int device, int* out) {
    if (device < 0 || device >= kMaxDev) return cudaErrorInvalidDevice;
    int m = most[device].load(std::memory_order_acquire);
    if (m == 0) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
      m = 8;
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = dev::kClusterMax;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(dev::kClusterMax);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0)
        m = dev::kClusterMax;
      else
        cudaGetLastError();
      most[device].store(m, std::memory_order_release);
    }
    *out = m;
    return cudaSuccess;
  }
};

template <typename Args>
cudaError_t launch_cluster(cudaStream_t s, void (*kern)(Args), int cs, int threads, size_t smem,
                           const Args& a) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kern, a);
}

// Points a block may hold: beyond it the cluster's 16 SMs are slower than the
// whole device with three launches an iteration
constexpr int kMostPoints = 4096;

// Blocks of the cluster for nel elements of order n: the fewest (1, 2, 4, 8,
// 16) whose elements are at most 128 lines a block; the largest size where
// none is.  0: the elements do not fit.
// sgeom: the per-point factors fit in shared memory beside the vectors.
template <int N, typename T>
int cluster_blocks(int nel, int most, bool aff, int* epc, bool* sgeom) {
  using C = dev::ClusterLevel<N, T>;
  for (int cs = 1; cs <= most; cs *= 2) {
    const int e = (nel + cs - 1) / cs;
    if ((cs < most && e * N * N > 128) || e * C::NT > kMostPoints) continue;
    for (bool g : {true, false})
      if (C::bytes(e, aff, g) <= kSmemMax) {
        *epc = e;
        *sgeom = g && !aff;
        return cs;
      }
  }
  return 0;
}

template <int N, typename T>
cudaError_t cluster_cg_n(cudaStream_t s, int device, const ClusterCgRun& L, bool launch,
                         bool* fits) {
  using C = dev::ClusterLevel<N, T>;
  auto kern = &dev::k_cluster_cg<N, T>;
  int epc = 0;
  bool sgeom = false;
  const bool aff = sizeof(T) == 8 && L.ag.c;
  // (too large for any cluster: the kernel is not loaded for it)
  *fits = cluster_blocks<N, T>(L.nel, dev::kClusterMax, aff, &epc, &sgeom) > 0;
  if (!*fits) return cudaSuccess;
  static ClusterAttr attr;
  int most = 0;
  cudaError_t e = attr.ensure((const void*)kern, 512, kSmemMax, device, &most);
  if (e != cudaSuccess) return e;
  const int cs = cluster_blocks<N, T>(L.nel, most, aff, &epc, &sgeom);
  *fits = cs > 0;
  if (!cs || !launch) return cudaSuccess;
  dev::ClusterCgArgs<T> a;
  a.nel = L.nel;
  a.epc = epc;
  a.cs = cs;
  a.f = (T*)L.f;
  a.x = (T*)L.x;
  a.ex = (T*)L.ex;
  a.gf = (const T*)L.gf;
  a.npts = (size_t)L.nel * C::NT;
  a.bj = L.bj;
  a.D = L.D;
  a.S = L.S;
  a.lambda = L.lambda;
  a.dinv = (const T*)L.dinv;
  a.mult = L.mult;
  a.mask = L.mask;
  a.dss = L.dss;
  a.ag = L.ag;
  a.helm = L.helm;
  a.pressure = !L.helm;
  a.weighted = L.weighted;
  a.sgeom = sgeom;
  a.nunique = L.nunique;
  a.eps = L.eps;
  a.max_iter = L.max_iter;
  a.frame = L.frame;
  a.hist = L.hist;
  a.hist_cap = L.hist_cap;
  int threads = (epc * N * N + 31) / 32 * 32;
  threads = std::min(std::max(threads, 256), 512);
  return launch_cluster(s, kern, cs, threads, C::bytes(epc, aff, sgeom), a);
}

template <typename T>
cudaError_t cluster_cg_t(cudaStream_t s, int device, int n, const ClusterCgRun& L, bool launch,
                         bool* fits) {
  *fits = false;
  switch (n) {
#define SSG_CLN(NV) \
  case NV: return cluster_cg_n<NV, T>(s, device, L, launch, fits);
    SSG_CLN(3) SSG_CLN(4) SSG_CLN(5) SSG_CLN(6) SSG_CLN(7) SSG_CLN(8) SSG_CLN(9) SSG_CLN(10)
    SSG_CLN(11) SSG_CLN(12)
#undef SSG_CLN
    default: return cudaSuccess;
  }
}

template <int KP>
cudaError_t cluster_coarse_k(cudaStream_t s, int device, dev::ClusterCoarseArgs a, bool* done) {
  *done = false;
  if ((a.nel + dev::kClusterMax - 1) / dev::kClusterMax * 8 > KP * dev::kCoarseThreads)
    return cudaSuccess;   // too large for any cluster: the kernel is not loaded for it
  auto kern = &dev::k_cluster_coarse<KP>;
  constexpr size_t most_smem = KP <= 2 ? 0 : (size_t)KP * dev::kCoarseThreads * 6 * 8;
  static ClusterAttr attr;
  int most = 0;
  cudaError_t e = attr.ensure((const void*)kern, dev::kCoarseThreads, most_smem, device, &most);
  if (e != cudaSuccess) return e;
  for (int cs = 1; cs <= most; cs *= 2) {
    const int epc = (a.nel + cs - 1) / cs;
    if (epc * 8 > KP * dev::kCoarseThreads) continue;
    a.cs = cs;
    a.epc = epc;
    *done = true;
    return launch_cluster(s, kern, cs, dev::kCoarseThreads,
                          KP <= 2 ? 0 : (size_t)epc * 8 * 6 * sizeof(double), a);
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t run_cluster_cg(cudaStream_t s, int device, int n, bool fp32, const ClusterCgRun& L,
                           bool launch, bool* fits) {
  *fits = false;
  if (fp32 && L.helm) return cudaSuccess;
  return fp32 ? cluster_cg_t<float>(s, device, n, L, launch, fits)
              : cluster_cg_t<double>(s, device, n, L, launch, fits);
}

cudaError_t run_cluster_coarse(cudaStream_t s, int device, int nel, const double* f, double* x,
                               double* ex, const double* gf, const double* D, const double* dinv,
                               const int* pairs, double nunique, double eps, double rel,
                               int max_iter, double* frame, bool* done) {
  dev::ClusterCoarseArgs a;
  a.nel = nel;
  a.f = f;
  a.x = x;
  a.ex = ex;
  a.gf = gf;
  a.npts = (size_t)nel * 8;
  a.D = D;
  a.dinv = dinv;
  a.pairs = reinterpret_cast<const int2*>(pairs);
  a.nunique = nunique;
  a.eps = eps;
  a.rel = rel;
  a.max_iter = max_iter;
  a.frame = frame;
  // one point a thread where the cluster holds them, else two, else four
  cudaError_t e = cluster_coarse_k<1>(s, device, a, done);
  if (e == cudaSuccess && !*done) e = cluster_coarse_k<2>(s, device, a, done);
  if (e == cudaSuccess && !*done) e = cluster_coarse_k<4>(s, device, a, done);
  return e;
}

}  // namespace ssg
