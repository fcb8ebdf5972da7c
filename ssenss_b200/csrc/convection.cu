// Dealiased skew-symmetric convection (convection_operator ->
// antialiased_convection_operator, src/convection.c:31-140), all in FP64:
//   1. interpolate the advecting u and advected v (3 components each) from
//      the n-point to the m = 3n/2-point GLL grid (interpolate_to_grid,
//      src/interpolation.c:136-155);
//   2. per dealiasing point, the convective form (u . grad) v_c with grad
//      through the conv-grid tinv (src/convection.c:71-93) and the
//      conservative form sum_a sum_b tinv[a][b] d_b(u_b v_c)
//      (src/convection.c:95-127), both weighted by rho J, averaged with
//      weights 1/2 (src/convection.c:129-140);
//   3. project back with (J^T)^3 (integrate_to_grid, src/interpolation.c:
//      157-176).
//
// Step 2 is regrouped per reference direction b (the same sums):
//   skew = sum_b ( A_b d_b v_c + B_b d_b(u_b v_c) ),
//   A_b = sum_a u_a W[a][b],  B_b = sum_a W[a][b],  W[a][b] = rho J tinv[a][b] / 2,
// so each direction b is one pass over the m-point lines along b.
//
// k_conv_line (m = 3n/2, n <= 12): what bounds it is the FP64 pipe and the
// shared-memory pipe together, so it is built to spend few of either.
//  - Every contraction (interpolation, derivative, projection) is one whole
//    line in one thread's registers: a line is loaded once for all its
//    outputs, and the small matrices sit in the kernel's parameter space, so
//    an entry is a constant-bank operand of the FMA.
//  - The GLL points are symmetric about 0, so the matrices are too
//    (J[M-1-o][N-1-p] = J[o][p], D[M-1-i][M-1-l] = -D[i][l]): a line is
//    split into its even and odd parts, each contracted with a matrix of a
//    quarter of the entries -- half the multiply-adds.  (The FP64 tensor
//    cores have the same peak as the FMA pipe, and their 8 x 8 x 4 tiles pad
//    m = 12 to 16 columns: the same work there is 2.6 times as many
//    operations.)
//  - Stages run in place: a thread overwrites the line it read, so the only
//    buffers are the fields themselves (U, V, SK) and all components of a
//    stage go through one sweep between two barriers.
//  - On affine elements (constant metric) the weights W reduce to nine
//    numbers an element, and the quadrature weights fold into the projection
//    matrix: no weight is read per point.
//
// Matrices without that symmetry (a caller's own arrays) and dealiasing orders
// other than 3n/2 run a runtime-order kernel of the same arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <iterator>
#include <type_traits>
#include <vector>

#include "kernels.cuh"
#include "ssg_internal.h"
#include "ssg_kernels.h"

namespace ssg {
namespace dev {

// ----------------------------------------------------------------------------
// compile-time-order kernel
// ----------------------------------------------------------------------------

// row stride of the m-wide shared fields: odd for odd m (scalar accesses),
// 2 mod 4 doubles for even m (16-byte accesses along i), so that lanes
// walking j hit distinct banks
__host__ __device__ constexpr int conv_row(int m) { return m % 2 ? m : (m % 4 == 2 ? m : m + 2); }

// A matrix entry in the kernel's parameter space, padded to 16 bytes: next
// to each other the compiler loads entries in pairs into registers, keeps
// them there across the line loop and spills (n = 8: 377 us a call on 4096
// elements); apart, each is a constant operand of its multiply-add
struct ConvEntry {
  double v, pad;
};

// even / odd halves of the three matrices (h = number of even terms)
template <int N, int M>
struct ConvMats {
  static constexpr int HN = (N + 1) / 2, HM = (M + 1) / 2;
  ConvEntry JE[HM * HN], JO[HM * HN];   // interpolation n -> m
  ConvEntry DE[HM * HM], DO[HM * HM];   // derivative on m points
  ConvEntry PE[HN * HM], PO[HN * HM];   // projection m -> n (weights folded in when affine)
};

template <int N>
struct ConvLine {
  static constexpr int M = (3 * N) / 2;
  static constexpr int RM = conv_row(M), PL = M * RM, FM = M * PL;
  // components advected together: three while the nine fields fit
  static constexpr int NB = (size_t)9 * FM * 8 <= 200 * 1024 ? 3 : 1;
  // n = 12: U, V and SK together exceed a block's shared memory by 832
  // bytes, so SK (written and read once a pass) lives in the block's part of
  // the global scratch and stays in L2
  static constexpr bool GSK = (size_t)(3 + 2 * NB) * FM * 8 > 227 * 1024;
  // per-point weights: A_b and B_b of the direction at hand as two more
  // fields, formed point by point with coalesced weight loads, once for all
  // components (lines reading the weights themselves: 143.6 us a call at
  // n = 8 on 1024 deformed elements); n >= 11 has no room for them
  static constexpr bool AB = (size_t)(5 + 2 * NB) * FM * 8 <= 227 * 1024;
  // self-convection: two such pairs by turns, the second in V's fields
  // (conv_passes), where one block has the SM to itself (1024 deformed
  // elements: n = 8 122.0 -> 116.4 us, n = 9 102.2 -> 94.7; below, the blocks
  // that share an SM already overlap: n = 5 94.1 and 96.4, n = 7 112.0 and 111.3)
  static constexpr bool TURNS = AB && NB == 3 && N >= 8;
  static constexpr size_t smem(bool aff) {
    return (size_t)(3 + (GSK ? 1 : 2) * NB + (!aff && AB ? 2 : 0)) * FM * sizeof(double);
  }
  static constexpr int TASKS = NB * M * M;
  // one line a thread, 128 registers at 512 threads; 448 threads (m = 12)
  // put four warps on two of the SM's four schedulers, so they would have the
  // registers of 512: 384 threads have 168 and the same longest scheduler
  static constexpr int FULL = (TASKS + 31) / 32 * 32;
  static constexpr int THREADS = N == 12 ? 256 : (FULL > 384 && FULL < 512 ? 384 : FULL);
  // small orders: several blocks per SM
  static constexpr int BLOCKS = THREADS <= 128 ? 4 : (THREADS <= 256 && NB == 3 ? 2 : 1);
};

// y (NO) = A x (NI), A symmetric under reversal of both indices (ANTI:
// antisymmetric), as its even / odd halves E, O
template <int NI, int NO, bool ANTI>
__device__ __forceinline__ void eo_contract(const ConvEntry* E, const ConvEntry* O,
                                            const double (&x)[NI], double (&y)[NO]) {
  constexpr int HI = NI / 2, CI = (NI + 1) / 2, HO = NO / 2, CO = (NO + 1) / 2;
  double a[CO], b[CO];
#pragma unroll
  for (int o = 0; o < CO; ++o) a[o] = b[o] = 0.0;
#pragma unroll
  for (int l = 0; l < HI; ++l) {
    const double e = x[l] + x[NI - 1 - l], d = x[l] - x[NI - 1 - l];
#pragma unroll
    for (int o = 0; o < CO; ++o) {
      a[o] = fma(E[o * CI + l].v, ANTI ? d : e, a[o]);
      if (o < HO) b[o] = fma(O[o * CI + l].v, ANTI ? e : d, b[o]);
    }
  }
  if (NI & 1) {
    // the middle entry is even: it joins the even sums (ANTI: the odd ones)
#pragma unroll
    for (int o = 0; o < CO; ++o) {
      if (!ANTI) a[o] = fma(E[o * CI + HI].v, x[HI], a[o]);
      if (ANTI && o < HO) b[o] = fma(O[o * CI + HI].v, x[HI], b[o]);
    }
  }
#pragma unroll
  for (int o = 0; o < HO; ++o) {
    y[o] = a[o] + b[o];
    y[NO - 1 - o] = a[o] - b[o];
  }
  if (NO & 1) y[HO] = a[HO];
}

template <int L>
__device__ __forceinline__ void load_line(const double* p, int stride, double (&x)[L]) {
#pragma unroll
  for (int l = 0; l < L; ++l) x[l] = p[l * stride];
}

// contiguous line (stride 1); V: at a 16-byte aligned address, even length
template <int L, bool V>
__device__ __forceinline__ void load_row(const double* p, double (&x)[L]) {
  if constexpr (V) {
#pragma unroll
    for (int l = 0; l < L; l += 2) {
      const double2 v = *reinterpret_cast<const double2*>(p + l);
      x[l] = v.x;
      x[l + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int l = 0; l < L; ++l) x[l] = p[l];
  }
}

template <int L>
__device__ __forceinline__ void store_line(double* p, int stride, const double (&x)[L]) {
#pragma unroll
  for (int l = 0; l < L; ++l) p[l * stride] = x[l];
}

template <int L, bool V>
__device__ __forceinline__ void store_row(double* p, const double (&x)[L]) {
  if constexpr (V) {
#pragma unroll
    for (int l = 0; l < L; l += 2)
      *reinterpret_cast<double2*>(p + l) = make_double2(x[l], x[l + 1]);
  } else {
#pragma unroll
    for (int l = 0; l < L; ++l) p[l] = x[l];
  }
}

// nf fields (field f at src0 for f < 3, src1 for f >= 3, components `cs`
// apart; n^3 in global) interpolated into dst (fields FM apart), in place
// stage by stage; vec: the sources start on 16-byte boundaries, where even
// orders up to 8 load pairs (n = 8 on 16^3 affine elements 314.6 us with single
// loads, 307; a caller's field may start anywhere, and from n = 10 the second
// form costs registers: n = 12 on 250 deformed elements 303.4 for 296.7); ends
// with a barrier
template <int N>
__device__ __forceinline__ void conv_interpolate(const ConvMats<N, ConvLine<N>::M>& mt, bool vec,
                                                 int nf,
                                                 const double* __restrict__ src0,
                                                 const double* __restrict__ src1, size_t cs,
                                                 double* dst) {
  using L = ConvLine<N>;
  constexpr int M = L::M, RM = L::RM, PL = L::PL, FM = L::FM;
  // x: lines (j, k) of n points in global memory -> row (k, j) of m points
  for (int t = threadIdx.x; t < nf * N * N; t += blockDim.x) {
    const int f = t / (N * N), jk = t - f * (N * N), j = jk % N, k = jk / N;
    const double* s = (f < 3 ? src0 + f * cs : src1 + (f - 3) * cs) + jk * N;
    double x[N], y[M];
    if constexpr (N % 2 == 0 && N <= 8) {
      if (vec)
        load_row<N, true>(s, x);
      else
        load_row<N, false>(s, x);
    } else {
      load_row<N, false>(s, x);
    }
    eo_contract<N, M, false>(mt.JE, mt.JO, x, y);
    store_row<M, RM % 2 == 0>(dst + f * FM + k * PL + j * RM, y);
  }
  __syncthreads();
  // y: columns (i, k) along j
  for (int t = threadIdx.x; t < nf * N * M; t += blockDim.x) {
    const int f = t / (N * M), r = t - f * (N * M), i = r % M, k = r / M;
    double* p = dst + f * FM + k * PL + i;
    double x[N], y[M];
    load_line<N>(p, RM, x);
    eo_contract<N, M, false>(mt.JE, mt.JO, x, y);
    store_line<M>(p, RM, y);
  }
  __syncthreads();
  // z: columns (i, j) along k
  for (int t = threadIdx.x; t < nf * M * M; t += blockDim.x) {
    const int f = t / (M * M), r = t - f * (M * M), i = r % M, j = r / M;
    double* p = dst + f * FM + j * RM + i;
    double x[N], y[M];
    load_line<N>(p, PL, x);
    eo_contract<N, M, false>(mt.JE, mt.JO, x, y);
    store_line<M>(p, PL, y);
  }
  __syncthreads();
}

// A_b and B_b of a direction at every point into AB (two fields) from its three
// per-point weight arrays Wb, `ws` apart; no barrier
template <int N>
__device__ __forceinline__ void conv_weights(const double* U, double* AB,
                                             const double* __restrict__ Wb, size_t ws) {
  using L = ConvLine<N>;
  constexpr int M = L::M, RM = L::RM, PL = L::PL, FM = L::FM;
  // up to six points a thread with every weight load in flight
  constexpr int MT = M * M * M, RND = (MT + L::THREADS - 1) / L::THREADS, G = RND < 6 ? RND : 6;
  for (int g0 = threadIdx.x; g0 < MT; g0 += G * L::THREADS) {
    double w[G][3];
#pragma unroll
    for (int h = 0; h < G; ++h) {
      const int g = g0 + h * L::THREADS;
#pragma unroll
      for (int c = 0; c < 3; ++c) w[h][c] = g < MT ? __ldg(Wb + c * ws + g) : 0.0;
    }
#pragma unroll
    for (int h = 0; h < G; ++h) {
      const int g = g0 + h * L::THREADS;
      if (g < MT) {
        const int i = g % M, j = (g / M) % M, k = g / (M * M), q = k * PL + j * RM + i;
        double A = w[h][0] * U[q];
        A = fma(w[h][1], U[FM + q], A);
        AB[q] = fma(w[h][2], U[2 * FM + q], A);
        AB[FM + q] = (w[h][0] + w[h][1]) + w[h][2];
      }
    }
  }
}

// direction B of the skew-symmetric form for nc advected components: SK_c
// (=, +=) A_b d_b v_c + B_b d_b(u_b v_c) at every point, one line of one
// component per thread.  AFF: Wb = the element's three constants W[.][b]
// (without the quadrature weights); else the three per-point arrays, or,
// where they are staged, conv_weights' fields in AB.  Ends with a barrier.
template <int N, int B, bool AFF>
__device__ __forceinline__ void conv_pass(const ConvMats<N, ConvLine<N>::M>& mt, int nc,
                                          const double* U, const double* V, double* SK,
                                          const double* AB, const double* __restrict__ Wb,
                                          size_t ws) {
  using L = ConvLine<N>;
  constexpr int M = L::M, RM = L::RM, PL = L::PL, FM = L::FM;
  // line step in shared memory / in the unpadded global point index
  constexpr int SS = B == 0 ? 1 : (B == 1 ? RM : PL);
  constexpr int SG = B == 0 ? 1 : (B == 1 ? M : M * M);
  for (int t = threadIdx.x; t < nc * M * M; t += blockDim.x) {
    const int c = t / (M * M), r = t - c * (M * M);
    const int a0 = r % M, a1 = r / M;   // the two coordinates across the line
    const int bs = B == 0 ? a0 * RM + a1 * PL : (B == 1 ? a0 + a1 * PL : a0 + a1 * RM);
    const double* vl = V + c * FM + bs;
    double v[M], ub[M], dv[M], dp[M];
    if constexpr (B == 0) {
      load_row<M, RM % 2 == 0>(vl, v);
      load_row<M, RM % 2 == 0>(U + bs, ub);
    } else {
      load_line<M>(vl, SS, v);
      load_line<M>(U + B * FM + bs, SS, ub);
    }
    eo_contract<M, M, true>(mt.DE, mt.DO, v, dv);
#pragma unroll
    for (int o = 0; o < M; ++o) v[o] = ub[o] * v[o];
    eo_contract<M, M, true>(mt.DE, mt.DO, v, dp);
    double* sk = SK + c * FM + bs;
    if constexpr (AFF) {
      const double w0 = Wb[0], w1 = Wb[1], w2 = Wb[2];
      const double wb = B == 0 ? w0 : (B == 1 ? w1 : w2);
      const double Bb = (w0 + w1) + w2;
      if ((B == 0 || w0 == 0.0) && (B == 1 || w1 == 0.0) && (B == 2 || w2 == 0.0)) {
        // axis-aligned element: u_b is the only component along b
#pragma unroll
        for (int o = 0; o < M; ++o) {
          const double s = wb * fma(ub[o], dv[o], dp[o]);
          if (B == 0)
            sk[o * SS] = s;
          else
            sk[o * SS] += s;
        }
      } else {
#pragma unroll
        for (int o = 0; o < M; ++o) {
          const double* q = U + bs + o * SS;
          double A = w0 * q[0];
          A = fma(w1, q[FM], A);
          A = fma(w2, q[2 * FM], A);
          double s = A * dv[o];
          s = fma(Bb, dp[o], s);
          if (B == 0)
            sk[o * SS] = s;
          else
            sk[o * SS] += s;
        }
      }
    } else if constexpr (L::AB) {
      const double* q = AB + bs;
#pragma unroll
      for (int o = 0; o < M; ++o) {
        double s = q[o * SS] * dv[o];
        s = fma(q[FM + o * SS], dp[o], s);
        if (B == 0)
          sk[o * SS] = s;
        else
          sk[o * SS] += s;
      }
    } else {
      const int bg = B == 0 ? a0 * M + a1 * M * M : (B == 1 ? a0 + a1 * M * M : a0 + a1 * M);
#pragma unroll
      for (int o = 0; o < M; ++o) {
        const double* q = U + bs + o * SS;
        const size_t g = bg + o * SG;
        const double w0 = __ldg(Wb + g), w1 = __ldg(Wb + ws + g), w2 = __ldg(Wb + 2 * ws + g);
        double A = w0 * q[0];
        A = fma(w1, q[FM], A);
        A = fma(w2, q[2 * FM], A);
        const double Bb = (w0 + w1) + w2;
        double s = A * dv[o];
        s = fma(Bb, dp[o], s);
        if (B == 0)
          sk[o * SS] = s;
        else
          sk[o * SS] += s;
      }
    }
  }
  __syncthreads();
}

// the three directions of conv_pass with staged weights: in one pair of fields,
// or (AB2) in two by turns, where a direction's weights form while the lines of
// the one before are at work
template <int N, bool AFF>
__device__ __forceinline__ void conv_passes(const ConvMats<N, ConvLine<N>::M>& mt, int nc,
                                            const double* U, const double* V, double* SK,
                                            double* AB, double* AB2,
                                            const double* __restrict__ Wb, size_t ws) {
  constexpr bool staged = !AFF && ConvLine<N>::AB;
  if (staged) {
    conv_weights<N>(U, AB, Wb, ws);
    __syncthreads();
    if (AB2) conv_weights<N>(U, AB2, Wb + 3 * ws, ws);
  }
  conv_pass<N, 0, AFF>(mt, nc, U, V, SK, AB, Wb, ws);
  if (staged) {
    conv_weights<N>(U, AB, Wb + (AB2 ? 6 : 3) * ws, ws);
    if (!AB2) __syncthreads();
  }
  conv_pass<N, 1, AFF>(mt, nc, U, V, SK, staged && AB2 ? AB2 : AB, Wb + 3 * ws, ws);
  if (staged && !AB2) {
    conv_weights<N>(U, AB, Wb + 6 * ws, ws);
    __syncthreads();
  }
  conv_pass<N, 2, AFF>(mt, nc, U, V, SK, AB, Wb + 6 * ws, ws);
}

// nc fields of SK -> out (n^3 in global, components `cs` apart) through
// (J^T)^3, in place; no barrier at the end (the last stage reads SK only)
template <int N>
__device__ __forceinline__ void conv_project(const ConvMats<N, ConvLine<N>::M>& mt, int nc,
                                             double* SK, double* __restrict__ out, size_t cs) {
  using L = ConvLine<N>;
  constexpr int M = L::M, RM = L::RM, PL = L::PL, FM = L::FM;
  // i: rows (j, k) of m points -> n points
  for (int t = threadIdx.x; t < nc * M * M; t += blockDim.x) {
    const int c = t / (M * M), r = t - c * (M * M), j = r % M, k = r / M;
    double* p = SK + c * FM + k * PL + j * RM;
    double x[M], y[N];
    load_row<M, RM % 2 == 0>(p, x);
    eo_contract<M, N, false>(mt.PE, mt.PO, x, y);
    store_line<N>(p, 1, y);
  }
  __syncthreads();
  // j: columns (i, k)
  for (int t = threadIdx.x; t < nc * N * M; t += blockDim.x) {
    const int c = t / (N * M), r = t - c * (N * M), i = r % N, k = r / N;
    double* p = SK + c * FM + k * PL + i;
    double x[M], y[N];
    load_line<M>(p, RM, x);
    eo_contract<M, N, false>(mt.PE, mt.PO, x, y);
    store_line<N>(p, RM, y);
  }
  __syncthreads();
  // k: columns (i, j) -> out
  for (int t = threadIdx.x; t < nc * N * N; t += blockDim.x) {
    const int c = t / (N * N), r = t - c * (N * N), i = r % N, j = r / N;
    double x[M], y[N];
    load_line<M>(SK + c * FM + j * RM + i, PL, x);
    eo_contract<M, N, false>(mt.PE, mt.PO, x, y);
    store_line<N>(out + c * cs + r, N * N, y);
  }
}

// Fields u, v, udv hold `nel` elements (component stride nel n^3); the
// factors hold all elements of the mesh, and field element e uses those of
// mesh element e0 + e.  W: AFF: 9 constants an element, W[9 e + 3 b + a] =
// J tinv[a][b] / 2; else 9 arrays of nel_fac m^3, W[(3b + a)][e][q] = rho J
// tinv[a][b] / 2.  u == v (self-convection): the fields are interpolated
// once.
template <int N, bool AFF>
__global__ void __launch_bounds__(ConvLine<N>::THREADS, ConvLine<N>::BLOCKS)
    k_conv_line(int nel, int e0, int nel_fac, const double* __restrict__ u,
                const double* __restrict__ v, double* __restrict__ udv,
                const double* __restrict__ W, double* __restrict__ scratch,
                const __grid_constant__ ConvMats<N, ConvLine<N>::M> mt) {
  using L = ConvLine<N>;
  constexpr int NT = N * N * N, M = L::M, FM = L::FM, NB = L::NB;
  constexpr size_t MT = (size_t)M * M * M;
  extern __shared__ __align__(16) double smem[];
  double* const U = smem;
  double* const SK = L::GSK ? scratch + (size_t)blockIdx.x * NB * FM : U + (3 + NB) * FM;
  double* const AB = U + (3 + (L::GSK ? 1 : 2) * NB) * FM;
  const bool self = u == v;
  const bool vec = ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(v)) & 15u) == 0;
  const size_t cs = (size_t)nel * NT, ws = AFF ? 1 : (size_t)nel_fac * MT;
  for (int e = blockIdx.x; e < nel; e += gridDim.x) {
    // the next element's fields (and weights) into L2 while this one
    // computes (a hint: 16-byte aligned chunks only)
    const int en = e + gridDim.x;
    if (threadIdx.x < 32 && en < nel) {
      const int lane = threadIdx.x;
      const double* p = nullptr;
      unsigned bytes = NT * sizeof(double);
      if (lane < 3) {
        p = u + (size_t)en * NT + lane * cs;
      } else if (lane < 6) {
        if (!self) p = v + (size_t)en * NT + (lane - 3) * cs;
      } else if (!AFF && lane < 15) {
        p = W + (size_t)(e0 + en) * MT + (lane - 6) * ws;
        bytes = MT * sizeof(double);
      }
      if (p && ((reinterpret_cast<uintptr_t>(p) | bytes) & 15u) == 0) bulk_prefetch_l2(p, bytes);
    }
    const double* Wb = AFF ? W + 9 * (size_t)(e0 + e) : W + (size_t)(e0 + e) * MT;
    const double* ue = u + (size_t)e * NT;
    const double* ve = v + (size_t)e * NT;
    double* oe = udv + (size_t)e * NT;
    if constexpr (NB == 3) {
      double* const V = self ? U : U + 3 * FM;
      conv_interpolate<N>(mt, vec, self ? 3 : 6, ue, ve, cs, U);
      conv_passes<N, AFF>(mt, 3, U, V, SK, AB, L::TURNS && self ? U + 3 * FM : nullptr, Wb, ws);
      conv_project<N>(mt, 3, SK, oe, cs);
    } else {
      conv_interpolate<N>(mt, vec, 3, ue, ue, cs, U);
#pragma unroll 1
      for (int c = 0; c < 3; ++c) {
        double* const V = self ? U + c * FM : U + 3 * FM;
        if (!self) conv_interpolate<N>(mt, vec, 1, ve + c * cs, ve, cs, V);
        conv_passes<N, AFF>(mt, 1, U, V, SK, AB, nullptr, Wb, ws);
        conv_project<N>(mt, 1, SK, oe + c * cs, cs);
        // the next component's first pass writes SK, its interpolation V
        if (self) __syncthreads();
      }
    }
    // the next element's interpolation writes U and V, last read before the
    // projection's barriers; its first pass writes SK after three barriers
  }
}

// ----------------------------------------------------------------------------
// runtime-order kernel (any n, m; fields in a global scratch region when they
// exceed shared memory)
// ----------------------------------------------------------------------------

// out (no^3) = (A x A x A) in (ni^3), stages x, y, z; A[o*ni + q]
// (transpose = true: A[q*no + o], the weak projection).  Block-cooperative.
__device__ void block_tensor3(int ni, int no, const double* A, bool transpose,
                              const double* in, double* t1, double* t2, double* out) {
  auto a = [&](int o, int q) { return transpose ? A[q * no + o] : A[o * ni + q]; };
  for (int q = threadIdx.x; q < ni * ni * no; q += blockDim.x) {
    const int o = q % no, kj = q / no;
    double s = 0;
    for (int r = 0; r < ni; ++r) s += a(o, r) * in[kj * ni + r];
    t1[q] = s;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < ni * no * no; q += blockDim.x) {
    const int o1 = q % no, o2 = (q / no) % no, k = q / (no * no);
    double s = 0;
    for (int r = 0; r < ni; ++r) s += a(o2, r) * t1[(k * ni + r) * no + o1];
    t2[q] = s;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < no * no * no; q += blockDim.x) {
    const int o12 = q % (no * no), o3 = q / (no * no);
    double s = 0;
    for (int r = 0; r < ni; ++r) s += a(o3, r) * t2[r * no * no + o12];
    out[q] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(512, 1) k_convection_rt(
    int nel, int e0, int nel_fac, int n, int m, const double* __restrict__ u,
    const double* __restrict__ v, double* __restrict__ udv, const double* __restrict__ W,
    const double* __restrict__ Dm, const double* __restrict__ J, double* __restrict__ gscr) {
  extern __shared__ __align__(16) double srt[];
  const int nt = n * n * n, mt = m * m * m;
  const int tmax = n * m * m > n * n * m ? n * m * m : n * n * m;
  double* sD = srt;                  // D[i*m + l]
  double* sJ = sD + m * m;           // J[i*n + p]
  double* t1 = sJ + m * n;
  double* t2 = t1 + tmax;
  double* stage = t2 + tmax;         // nt
  double* ui = gscr ? gscr + (size_t)blockIdx.x * 5 * mt : stage + nt;   // 3 x mt
  double* vc = ui + 3 * mt;
  double* sk = vc + mt;
  const size_t nptsn = (size_t)nel * nt, wstride = (size_t)nel_fac * mt;
  for (int q = threadIdx.x; q < m * m; q += blockDim.x) sD[q] = Dm[q];
  for (int q = threadIdx.x; q < m * n; q += blockDim.x) sJ[q] = J[q];
  for (size_t e = blockIdx.x; e < (size_t)nel; e += gridDim.x) {
    for (int f = 0; f < 3; ++f) {
      __syncthreads();
      for (int q = threadIdx.x; q < nt; q += blockDim.x) stage[q] = u[f * nptsn + e * nt + q];
      __syncthreads();
      block_tensor3(n, m, sJ, false, stage, t1, t2, ui + f * mt);
    }
    for (int c = 0; c < 3; ++c) {
      __syncthreads();
      for (int q = threadIdx.x; q < nt; q += blockDim.x) stage[q] = v[c * nptsn + e * nt + q];
      __syncthreads();
      block_tensor3(n, m, sJ, false, stage, t1, t2, vc);
      for (int q = threadIdx.x; q < mt; q += blockDim.x) {
        const int i = q % m, j = (q / m) % m, k = q / (m * m);
        const size_t g = (e + e0) * mt + q;
        const int base[3] = {(k * m + j) * m, k * m * m + i, j * m + i};
        const int step[3] = {1, m, m * m};
        const int at[3] = {i, j, k};
        double s = 0.0;
        for (int b = 0; b < 3; ++b) {
          double dv = 0.0, dp = 0.0;
          for (int l = 0; l < m; ++l) {
            const double d = sD[at[b] * m + l];
            const double vl = vc[base[b] + l * step[b]];
            dv = fma(d, vl, dv);
            dp = fma(d, ui[b * mt + base[b] + l * step[b]] * vl, dp);
          }
          const double w0 = W[(3 * b) * wstride + g], w1 = W[(3 * b + 1) * wstride + g],
                       w2 = W[(3 * b + 2) * wstride + g];
          double A = w0 * ui[q];
          A = fma(w1, ui[mt + q], A);
          A = fma(w2, ui[2 * mt + q], A);
          const double Bb = (w0 + w1) + w2;
          s = b == 0 ? A * dv : fma(A, dv, s);
          s = fma(Bb, dp, s);
        }
        sk[q] = s;
      }
      __syncthreads();
      block_tensor3(m, n, sJ, true, sk, t1, t2, stage);
      for (int q = threadIdx.x; q < nt; q += blockDim.x) udv[c * nptsn + e * nt + q] = stage[q];
    }
    __syncthreads();
  }
}

}  // namespace dev

static size_t convection_rt_smem(int n, int m, bool fields) {
  const size_t nt = (size_t)n * n * n, mt = (size_t)m * m * m;
  const size_t tmax = std::max((size_t)n * m * m, (size_t)n * n * m);
  return (m * m + m * n + 2 * tmax + nt + (fields ? 5 * mt : 0)) * sizeof(double);
}

static constexpr size_t kConvSmemMax = 227 * 1024;

size_t convection_scratch_doubles(int n, int m) {
  if (convection_rt_smem(n, m, true) <= kConvSmemMax) return 0;
  return (size_t)kConvScratchBlocks * 5 * m * m * m;
}

// even / odd halves of A (no x ni, A[o * ni + i]); false when A is not
// (anti)symmetric under reversal of both indices to rounding
bool conv_eo_split(int ni, int no, const double* A, bool anti, std::vector<double>& E,
                   std::vector<double>& O) {
  const int ci = (ni + 1) / 2, co = (no + 1) / 2;
  E.assign((size_t)co * ci, 0.0);
  O.assign((size_t)co * ci, 0.0);
  const double sg = anti ? -1.0 : 1.0;
  double top = 0.0;
  for (int q = 0; q < ni * no; ++q) top = std::max(top, std::fabs(A[q]));
  std::vector<double> S((size_t)ni * no);
  for (int o = 0; o < no; ++o)
    for (int i = 0; i < ni; ++i) {
      const double a = A[o * ni + i], b = sg * A[(no - 1 - o) * ni + ni - 1 - i];
      if (!(std::fabs(a - b) <= mirror_noise(std::max(ni, no)) * top)) return false;
      S[o * ni + i] = 0.5 * (a + b);
    }
  for (int o = 0; o < co; ++o)
    for (int i = 0; i < ci; ++i) {
      const double p = S[o * ni + i], q = S[o * ni + ni - 1 - i];
      const bool mid = 2 * i + 1 == ni;
      // even inputs weigh (p + q) / 2, odd ones (p - q) / 2; E multiplies the
      // part that the reversal keeps (even, or odd when antisymmetric)
      const double even = mid ? p : 0.5 * (p + q), odd = 0.5 * (p - q);
      E[o * ci + i] = anti ? odd : even;
      O[o * ci + i] = anti ? even : odd;
    }
  return true;
}

template <int N>
static cudaError_t launch_line(cudaStream_t s, int nel, int e0, int nel_fac, const double* u,
                               const double* v, double* udv, const ConvGeom& g) {
  using L = dev::ConvLine<N>;
  constexpr int M = L::M;
  dev::ConvMats<N, M> mt = {};
  auto put = [](dev::ConvEntry* dst, const double* src, size_t count) {
    for (size_t q = 0; q < count; ++q) dst[q].v = src[q];
  };
  put(mt.JE, g.eo[0], std::size(mt.JE));
  put(mt.JO, g.eo[1], std::size(mt.JO));
  put(mt.DE, g.eo[2], std::size(mt.DE));
  put(mt.DO, g.eo[3], std::size(mt.DO));
  put(mt.PE, g.eo[4], std::size(mt.PE));
  put(mt.PO, g.eo[5], std::size(mt.PO));
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  auto go = [&](auto aff) -> cudaError_t {
    constexpr bool A = decltype(aff)::value;
    auto kern = &dev::k_conv_line<N, A>;
    static SmemAttr attr;
    cudaError_t ce = attr.ensure((const void*)kern, L::smem(A));
    if (ce != cudaSuccess) return ce;
    // one wave of resident blocks walking the elements
    constexpr int fit = (int)(kConvSmemMax / L::smem(A));
    constexpr int per = fit < 1 ? 1 : (fit > 8 ? 8 : fit);
    const int grid = std::min(std::min(nel, per * sms), L::GSK ? kConvScratchBlocks : nel);
    count_launch();
    kern<<<grid, L::THREADS, L::smem(A), s>>>(nel, e0, nel_fac, u, v, udv, A ? g.aff : g.W,
                                            g.scratch, mt);
    return cudaGetLastError();
  };
  return g.aff ? go(std::true_type()) : go(std::false_type());
}

cudaError_t run_convection(cudaStream_t s, int nel, int e0, int nel_fac, int n, int m,
                           const double* u, const double* v, double* udv, const ConvGeom& g) {
  if (nel <= 0) return cudaSuccess;
  if (g.eo[0] && m == (3 * n) / 2 && (n < 12 || g.scratch)) {
    switch (n) {
#define SSG_CONVL(NV) \
  case NV:            \
    return launch_line<NV>(s, nel, e0, nel_fac, u, v, udv, g);
      SSG_CONVL(2) SSG_CONVL(3) SSG_CONVL(4) SSG_CONVL(5) SSG_CONVL(6) SSG_CONVL(7)
      SSG_CONVL(8) SSG_CONVL(9) SSG_CONVL(10) SSG_CONVL(11) SSG_CONVL(12)
#undef SSG_CONVL
      default:
        break;
    }
  }
  const bool in_smem = convection_rt_smem(n, m, true) <= kConvSmemMax;
  if (!in_smem && !g.scratch) return cudaErrorInvalidValue;
  const size_t smem = convection_rt_smem(n, m, in_smem);
  if (smem > kConvSmemMax) return cudaErrorInvalidValue;
  static SmemAttr attr;
  {
    cudaError_t e = attr.ensure((const void*)dev::k_convection_rt, kConvSmemMax);
    if (e != cudaSuccess) return e;
  }
  const int grid = in_smem ? nel : std::min(nel, kConvScratchBlocks);
  count_launch();
  dev::k_convection_rt<<<grid, 512, smem, s>>>(nel, e0, nel_fac, n, m, u, v, udv, g.W, g.Dd,
                                               g.Jd, in_smem ? nullptr : g.scratch);
  return cudaGetLastError();
}

}  // namespace ssg
