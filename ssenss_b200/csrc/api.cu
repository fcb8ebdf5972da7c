// C-ABI entry points: context, set-up/upload, operators.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "ssg_internal.h"
#include "ssg_kernels.h"

namespace ssg {

ssg_status fail(ssg_context* c, ssg_status s, const std::string& msg) {
  if (c) c->err = msg;
  return s;
}

ssg_status cuda_fail(ssg_context* c, cudaError_t e, const char* what) {
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return fail(c, SSG_ERR_NOMEM, m);
  return fail(c, SSG_ERR_CUDA, m);
}

bool is_device_ptr(const void* p) {
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

template <typename T>
static ssg_status dalloc(ssg_context* c, T** p, size_t count) {
  *p = nullptr;
  if (count == 0) return SSG_OK;
  SSG_CUDA(c, cudaMalloc((void**)p, count * sizeof(T)));
  c->dev_bytes += count * sizeof(T);
  return SSG_OK;
}

template <typename T>
static ssg_status dupload(ssg_context* c, T** p, const T* src, size_t count) {
  SSG_TRY(dalloc(c, p, count));
  if (count) SSG_CUDA(c, cudaMemcpy(*p, src, count * sizeof(T), cudaMemcpyHostToDevice));
  return SSG_OK;
}

static ssg_status upload_f32(ssg_context* c, float** p, const double* src, size_t count) {
  std::vector<float> t(count);
  const size_t blk = 1 << 14;   // converted on all host threads
  parallel_elements((int)((count + blk - 1) / blk), [&](int b0, int b1) {
    const size_t hi = std::min(count, (size_t)b1 * blk);
    for (size_t q = (size_t)b0 * blk; q < hi; ++q) t[q] = (float)src[q];
  });
  return dupload(c, p, t.data(), count);
}

static void dfree(void* p) {
  if (p) cudaFree(p);
}

static void free_level(ssg::DevLevel& d) {
  dfree(d.gf); dfree(d.bj); dfree(d.kdiag); dfree(d.dinv_p); dfree(d.dinv_h);
  dfree(d.mult); dfree(d.mask); dfree(d.D); dfree(d.S); dfree(d.Ar); dfree(d.Ap);
  dfree(d.aff); dfree(d.w);
  dfree(d.gf32); dfree(d.dinv_p32); dfree(d.dss_ec); dfree(d.det); dfree(d.rho);
  d = ssg::DevLevel();
}

static void free_conv(ssg_context* c) {
  dfree(c->conv_w); dfree(c->conv_D); dfree(c->conv_J);
  dfree(c->conv_scratch); dfree(c->conv_aff);
  c->conv_w = c->conv_D = c->conv_J = c->conv_scratch = c->conv_aff = nullptr;
  for (auto& v : c->conv_eo) v.clear();
}

static void free_mesh(ssg_context* c) {
  c->dev_bytes = 0;
  if (c->ws) {
    free_workspace(c->ws);
    c->ws = nullptr;
  }
  if (c->seg) {
    seg_scratch_free(*c->seg);
    delete c->seg;
    c->seg = nullptr;
  }
  if (c->vhist) cudaFree(c->vhist);
  if (c->rk_scratch) cudaFree(c->rk_scratch);
  c->vhist = c->rk_scratch = nullptr;
  dfree(c->flow_buf);
  dfree(c->flow_sw);
  dfree(c->flow_bc);
  c->flow_buf = c->flow_sw = nullptr;
  c->flow_bc = nullptr;
  for (int l = 0; l < 3; ++l) c->fu[l] = c->fconv[l] = c->frot[l] = c->fp[l] = nullptr;
  c->ff = c->fut = c->fa = c->fb = c->fbc = nullptr;
  c->flow_ready = false;
  for (auto& l : c->lev) free_level(l);
  dfree(c->d_pairs); c->d_pairs = nullptr;
  dfree(c->d_nbreg); c->d_nbreg = nullptr;
  dfree(c->inv_mass); c->inv_mass = nullptr;
  free_conv(c);
  c->m = 0;
  dfree(c->p_jac); dfree(c->p_tinv); dfree(c->p_ur); dfree(c->p_x);
  c->p_jac = c->p_tinv = c->p_ur = c->p_x = nullptr;
  dfree(c->d_neigh); c->d_neigh = nullptr;
  dfree(c->d_passes); c->d_passes = nullptr;
  c->has_ur = false;
  dfree(c->p_state); c->p_state = nullptr;
  if (c->p_ints) cudaFree(c->p_ints);
  c->p_ints = nullptr;
  c->p_cap = 0;
  if (c->p_order) cudaFree(c->p_order);
  if (c->p_bucket) cudaFree(c->p_bucket);
  c->p_order = c->p_bucket = nullptr;
  c->p_order_cap = 0;
  dfree(c->d_part); c->d_part = nullptr;
  for (auto& s : c->d_stage) { dfree(s); s = nullptr; }
  c->stage_cap = 0;
  c->ready = false;
}

// rho_ijk = (w_i w_j) w_k (gll_weights_array, src/basis.c:179-188)
static std::vector<double> rho3(const std::vector<double>& w) {
  const int n = (int)w.size();
  std::vector<double> r((size_t)n * n * n);
  for (int k = 0; k < n; ++k)
    for (int j = 0; j < n; ++j)
      for (int i = 0; i < n; ++i) r[(k * n + j) * n + i] = (w[i] * w[j]) * w[k];
  return r;
}

// Dealiasing-grid factors (initialise_convection_geometry, src/main.c:60-64,
// src/geometry.c): W[3b + a] = rho J tinv[a][b] / 2 at the m points (9 x nel
// x m^3: the convection kernel's per-direction weights), the m-point
// derivative matrix and the n -> m interpolation matrix.
static ssg_status upload_conv(ssg_context* c) {
  const ssg::HostMesh& H = c->host;
  const ssg::HostLevel& m = H.conv;
  const int nel = H.nel;
  free_conv(c);
  c->m = m.n;
  const size_t mp = m.nt * nel;
  const std::vector<double> rho = rho3(m.w);
  std::vector<double> wv(9 * mp);
  for (int b = 0; b < 3; ++b)
    for (int a = 0; a < 3; ++a) {
      const double* t = m.tinv[3 * a + b].data();
      double* dst = wv.data() + (size_t)(3 * b + a) * mp;
      parallel_elements(nel, [&](int e0, int e1) {
        for (int e = e0; e < e1; ++e)
          for (size_t q = 0; q < m.nt; ++q) {
            const size_t g = e * m.nt + q;
            dst[g] = 0.5 * ((rho[q] * m.det[g]) * t[g]);
          }
      });
    }
  SSG_TRY(dupload(c, &c->conv_w, wv.data(), wv.size()));
  SSG_TRY(dupload(c, &c->conv_D, m.D.data(), m.D.size()));
  SSG_TRY(dupload(c, &c->conv_J, H.jconv.data(), H.jconv.size()));
  std::vector<double> aff;
  affine_convection(m, nel, aff);
  // (the affine form folds the quadrature weights into the projection)
  std::vector<double> P((size_t)H.n * m.n);
  for (int p = 0; p < H.n; ++p)
    for (int o = 0; o < m.n; ++o)
      P[(size_t)p * m.n + o] = H.jconv[(size_t)o * H.n + p] * (aff.empty() ? 1.0 : m.w[o]);
  std::vector<double>* eo = c->conv_eo;
  if (!conv_eo_split(H.n, m.n, H.jconv.data(), false, eo[0], eo[1]) ||
      !conv_eo_split(m.n, m.n, m.D.data(), true, eo[2], eo[3]) ||
      !conv_eo_split(m.n, H.n, P.data(), false, eo[4], eo[5]))
    for (int k = 0; k < 6; ++k) eo[k].clear();
  if (!aff.empty() && !eo[0].empty()) SSG_TRY(dupload(c, &c->conv_aff, aff.data(), aff.size()));
  const size_t scr = convection_scratch_doubles(H.n, m.n);
  if (scr) SSG_TRY(dalloc(c, &c->conv_scratch, scr));
  return SSG_OK;
}

// Level-0 Jacobian and its transposed inverse for the particle walk
// (sel->geom->jac / tinv_jac, src/geometry.c).
static ssg_status upload_particle_geom(ssg_context* c) {
  const ssg::HostLevel& h = c->host.lev[0];
  const size_t np0 = h.nt * (size_t)c->host.nel;
  dfree(c->p_jac); dfree(c->p_tinv);
  c->p_jac = c->p_tinv = nullptr;
  std::vector<double> ja(9 * np0), ti(9 * np0);
  for (int a = 0; a < 9; ++a) {
    std::copy(h.jac[a].begin(), h.jac[a].end(), ja.begin() + a * np0);
    std::copy(h.tinv[a].begin(), h.tinv[a].end(), ti.begin() + a * np0);
  }
  SSG_TRY(dupload(c, &c->p_jac, ja.data(), ja.size()));
  SSG_TRY(dupload(c, &c->p_tinv, ti.data(), ti.size()));
  const std::vector<double>& px = c->host.ppoints.empty() ? h.x : c->host.ppoints;
  dfree(c->p_x);
  c->p_x = nullptr;
  SSG_TRY(dupload(c, &c->p_x, px.data(), px.size()));
  if (!c->p_ur) {
    SSG_TRY(dalloc(c, &c->p_ur, 9 * np0));
    SSG_CUDA(c, cudaMemset(c->p_ur, 0, 9 * np0 * sizeof(double)));
  }
  return SSG_OK;
}

// Upload every level (and the optional dealiasing / particle data) from
// c->host; the diagonals, multiplicities and masks are derived here as
// initialise_preconditioners does (src/precon.c:336-413).
static ssg_status upload_all(ssg_context* c) {
  ssg::HostMesh& H = c->host;
  const int nel = H.nel;
  c->n = H.n;
  c->nel = nel;
  c->nlev = H.nlev;
  c->has_walls = false;
  c->mask_same = true;
  for (int e = 0; e < nel; ++e)
    if (H.bc[e]) c->has_walls = true;
  if ((size_t)nel * H.lev[0].nt >= (size_t)INT32_MAX)
    return fail(c, SSG_ERR_ARG, "mesh exceeds 2^31 local points (32-bit node indices)");
  SSG_TRY(dupload(c, &c->d_pairs, H.pairs.data(), H.pairs.size()));
  {
    // the line-run DSS applies where every face, edge and corner is
    // paired with the opposite one of its neighbour (faces w/e, s/n, b/t;
    // edges and corners with every side flipped)
    std::vector<int> nb((size_t)nel * 26, -1);
    bool regular = true;
    for (size_t e = 0; e < (size_t)nel && regular; ++e)
      for (int sl = 0; sl < 26; ++sl) {
        const int other = H.pairs[2 * (26 * e + sl)], found = H.pairs[2 * (26 * e + sl) + 1];
        if (other < 0) continue;
        const int j = sl < 6 ? sl : (sl < 18 ? sl - 6 : sl - 18);
        const int opp = sl < 6 ? (j ^ 1) : (sl < 18 ? (j ^ 3) : (j ^ 7));
        if (found != opp) {
          regular = false;
          break;
        }
        nb[26 * e + sl] = other;
      }
    if (regular) SSG_TRY(dupload(c, &c->d_nbreg, nb.data(), nb.size()));
    c->pairs_full = dss_is_complete(H);
  }
  for (int l = 0; l < H.nlev; ++l) {
    const ssg::HostLevel& h = H.lev[l];
    ssg::DevLevel& d = c->lev[l];
    c->orders[l] = h.n;
    d.n = h.n;
    d.nt = h.nt;
    d.npts = h.nt * nel;
    const size_t np = d.npts;
    const std::vector<double> rho = rho3(h.w);
    std::vector<double> bj(np), gf(6 * np);
    parallel_elements(nel, [&](int e0, int e1) {
      for (int e = e0; e < e1; ++e)
        for (size_t q = 0; q < h.nt; ++q) {
          const size_t i = e * h.nt + q;
          bj[i] = rho[q] * h.det[i];
          for (int a = 0; a < 6; ++a) gf[a * np + i] = h.g[a][i] * bj[i];
        }
    });
    std::vector<double> kd(np);
    stiffness_diagonal(h, nel, kd.data());
    std::vector<double> dp(kd);
    host_dss(H, h.n, dp.data());
    std::vector<double> sc(np, 1.0);
    host_dss(H, h.n, sc.data());
    std::vector<uint8_t> mu(np);
    parallel_elements(nel, [&](int e0, int e1) {
      for (size_t q = e0 * h.nt; q < (size_t)e1 * h.nt; ++q) {
        dp[q] = 1.0 / dp[q];
        mu[q] = (uint8_t)std::lround(sc[q]);
        sc[q] = 1.0 / sc[q];
      }
    });
    double nun = 0.0;
    for (double v : sc) nun += v;
    d.nunique = nun;
    // FP32 copy for the mixed-precision V-cycle, natural point order (its
    // operator is the line-form kernel at every order)
    SSG_TRY(upload_f32(c, &d.gf32, gf.data(), gf.size()));
    if (h.n == 8) {
      // the FP64 tensor-core operator's fragment order (see ax8.cu)
      std::vector<double> nat(gf);
      parallel_elements(nel, [&](int e0, int e1) {
        for (int a = 0; a < 6; ++a)
          for (int e = e0; e < e1; ++e)
            for (size_t q = 0; q < h.nt; ++q) {
              const size_t i = e * h.nt + q;
              gf[a * np + e * h.nt + ax8_fragment_index((int)q)] = nat[a * np + i];
            }
      });
    }
    SSG_TRY(dupload(c, &d.gf, gf.data(), gf.size()));
    SSG_TRY(dupload(c, &d.bj, bj.data(), np));
    {
      std::vector<double> aff;
      affine_metric(h, nel, aff);
      if (!aff.empty()) {
        SSG_TRY(dupload(c, &d.aff, aff.data(), aff.size()));
        SSG_TRY(dupload(c, &d.w, h.w.data(), h.w.size()));
      }
    }
    SSG_TRY(dupload(c, &d.kdiag, kd.data(), np));
    SSG_TRY(dupload(c, &d.dinv_p, dp.data(), np));
    SSG_TRY(dalloc(c, &d.dinv_h, np));
    d.lambda_h = -1.0;
    SSG_TRY(dupload(c, &d.mult, mu.data(), np));
    if (c->has_walls) {
      std::vector<double> mk(np, 1.0);
      const int n = h.n;
      for (int e = 0; e < nel; ++e)
        for (int f = 0; f < 6; ++f)
          if (H.bc[e] & (1 << f))
            for (int k = 0; k < n; ++k)
              for (int j = 0; j < n; ++j)
                for (int i = 0; i < n; ++i) {
                  const bool on = (f == 0 && i == 0) || (f == 1 && i == n - 1) ||
                                  (f == 2 && j == 0) || (f == 3 && j == n - 1) ||
                                  (f == 4 && k == 0) || (f == 5 && k == n - 1);
                  if (on) mk[e * h.nt + (k * n + j) * n + i] = 0.0;
                }
      SSG_TRY(dupload(c, &d.mask, mk.data(), np));
      if (l == 0) {
        std::vector<double> copies(mk);   // unmasked copies of each node
        host_dss(H, n, copies.data());
        for (size_t q = 0; q < np; ++q)
          if (copies[q] != mk[q] * mu[q]) c->mask_same = false;
      }
    }
    {
      std::vector<int> ec;
      dss_map_table(H, h.n, ec);
      SSG_TRY(dupload(c, &d.dss_ec, ec.data(), ec.size()));
    }
    d.sym = true;
    for (const std::vector<double>* A : {&h.D, &h.S}) {
      const int n = h.n;
      double top = 0.0;
      for (double v : *A) top = std::max(top, std::fabs(v));
      for (int q = 0; q < n * n; ++q)
        if (!(std::fabs((*A)[q] + (*A)[n * n - 1 - q]) <= mirror_noise(n) * top)) d.sym = false;
    }
    SSG_TRY(dupload(c, &d.D, h.D.data(), h.D.size()));
    SSG_TRY(dupload(c, &d.S, h.S.data(), h.S.size()));
    SSG_TRY(upload_f32(c, &d.dinv_p32, dp.data(), np));
    if (l >= 1) {
      const int nf = H.lev[l - 1].n, nc = h.n;
      std::vector<double> Ar((size_t)nc * nf);
      for (int i = 0; i < nf; ++i)
        for (int p = 0; p < nc; ++p) Ar[p * nf + i] = h.jf[i * nc + p];
      SSG_TRY(dupload(c, &d.Ar, Ar.data(), Ar.size()));
      SSG_TRY(dupload(c, &d.Ap, h.jf.data(), h.jf.size()));
    }
    if (l == 0) {
      SSG_TRY(dupload(c, &d.det, h.det.data(), np));
      SSG_TRY(dupload(c, &d.rho, rho.data(), rho.size()));
      std::vector<double> im(bj);
      host_dss(H, h.n, im.data());
      for (auto& v : im) v = 1.0 / v;
      SSG_TRY(dupload(c, &c->inv_mass, im.data(), np));
    }
  }
  const size_t np0 = c->lev[0].npts;
  if (H.has_conv) SSG_TRY(upload_conv(c));
  if (H.has_particle_geom) SSG_TRY(upload_particle_geom(c));
  if (!c->p_x) SSG_TRY(dupload(c, &c->p_x, H.lev[0].x.data(), H.lev[0].x.size()));
  SSG_TRY(dupload(c, &c->d_neigh, H.neigh.data(), H.neigh.size()));
  SSG_TRY(dalloc(c, &c->d_passes, 1));
  // reduction partials: enough for 10 dot products over the largest grid
  // sized for the largest grids the autotuner may pick: 64 blocks per SM
  // for the vector kernels (up to 16 partial sums each) and for the DSS (up
  // to 4)
  const size_t vb = std::min((np0 + 255) / 256, (size_t)148 * 64);
  const size_t db = (size_t)148 * 64;
  c->part_cap = std::max(16 * vb, 4 * db) + 64;
  SSG_TRY(dalloc(c, &c->d_part, c->part_cap));
  // staging for host arguments: up to three vector fields
  // (one field unless the dealiasing grid is set up: convection stages
  // three-component fields)
  c->stage_cap = H.has_conv ? 3 * np0 : np0;
  for (auto& s : c->d_stage) SSG_TRY(dalloc(c, &s, c->stage_cap));
  // (uploads are synchronous copies; no device-wide synchronisation, which
  // would collide with another thread's stream capture)
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  c->ready = true;
  return SSG_OK;
}

// Helmholtz Jacobi inverse for lambda = (11/6)/(dt visc) at level 0
// (initialise_diagonal_precon, src/precon.c:336-359, with
// helmholtz_diagonal, src/helmholtz.c:51-68): DSS(kdiag + (lambda rho) J),
// reciprocal -- on the device, from the stored stiffness diagonal.
ssg_status helmholtz_diag_update(ssg_context* c) {
  const double lam = (11.0 / 6.0) * 1.0 / (c->dt * c->visc);
  ssg::DevLevel& d = c->lev[0];
  if (d.lambda_h == lam) return SSG_OK;
  SSG_TRY(ensure_workspace(c));
  double* tmp = workspace_scratch(c);
  SSG_CUDA(c, run_helm_diag(c->stream, d.npts, d.nt, d.kdiag, d.rho, d.det, lam, tmp));
  SSG_CUDA(c, run_dss(c->stream, DSS_PLAIN, false, d.n, c->nel, tmp, d.dinv_h, c->d_nbreg,
                      d.dss_ec, nullptr, nullptr, nullptr, nullptr));
  SSG_CUDA(c, run_recip(c->stream, d.npts, d.dinv_h));
  d.lambda_h = lam;
  return SSG_OK;
}

// ---- staging ------------------------------------------------------------

// Device view of a caller field: the pointer itself when it is device
// memory, else a staging slot filled from the host.
static ssg_status stage_in(ssg_context* c, int slot, const double* p, size_t count,
                           const double** out) {
  if (!p) return fail(c, SSG_ERR_ARG, "null field pointer");
  if (is_device_ptr(p)) {
    *out = p;
    return SSG_OK;
  }
  if (count > c->stage_cap) return fail(c, SSG_ERR_ARG, "field larger than staging");
  SSG_CUDA(c, cudaMemcpyAsync(c->d_stage[slot], p, count * sizeof(double),
                              cudaMemcpyHostToDevice, c->stream));
  *out = c->d_stage[slot];
  return SSG_OK;
}

static ssg_status stage_out(ssg_context* c, int slot, double* p, size_t count,
                            double** out) {
  if (!p) return fail(c, SSG_ERR_ARG, "null field pointer");
  if (is_device_ptr(p)) {
    *out = p;
    return SSG_OK;
  }
  if (count > c->stage_cap) return fail(c, SSG_ERR_ARG, "field larger than staging");
  *out = c->d_stage[slot];
  return SSG_OK;
}

static ssg_status stage_back(ssg_context* c, double* host, const double* dev, size_t count) {
  if (host != dev)
    SSG_CUDA(c, cudaMemcpyAsync(host, dev, count * sizeof(double), cudaMemcpyDeviceToHost,
                                c->stream));
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  return SSG_OK;
}

static ssg_status need_ready(ssg_context* c) {
  if (!c) return SSG_ERR_ARG;
  if (!c->ready) return fail(c, SSG_ERR_STATE, "no mesh set up on this context");
  SSG_CUDA(c, cudaSetDevice(c->device));
  return SSG_OK;
}

}  // namespace ssg

using namespace ssg;

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

static ssg_status create_impl(int device, void* stream, ssg_context** out) {
  if (!out) return SSG_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return SSG_ERR_CUDA;
  }
  if (device < 0 || device >= ndev) return SSG_ERR_ARG;
  ssg_context* c = new ssg_context();
  c->device = device;
  if (cudaSetDevice(device) != cudaSuccess) {
    delete c;
    return SSG_ERR_CUDA;
  }
  if (stream) {
    c->stream = (cudaStream_t)stream;
    c->own_stream = false;
  } else {
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete c;
      return SSG_ERR_CUDA;
    }
    c->own_stream = true;
  }
  if (cudaMalloc(&c->d_sums, 16 * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&c->d_counter, sizeof(unsigned)) != cudaSuccess ||
      cudaMemset(c->d_counter, 0, sizeof(unsigned)) != cudaSuccess ||
      cudaMalloc(&c->d_sc, FR_COUNT * F_SIZE * sizeof(double)) != cudaSuccess ||
      cudaMallocHost(&c->h_pin, 64 * sizeof(double)) != cudaSuccess ||
      cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess) {
    ssg_destroy(c);
    return SSG_ERR_CUDA;
  }
  cudaMemset(c->d_sc, 0, FR_COUNT * F_SIZE * sizeof(double));
  *out = c;
  return SSG_OK;
}

ssg_status ssg_create(int device, ssg_context** out) { return create_impl(device, nullptr, out); }

ssg_status ssg_create_on_stream(int device, void* cuda_stream, ssg_context** out) {
  return create_impl(device, cuda_stream, out);
}

void ssg_destroy(ssg_context* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  free_mesh(c);
  dfree(c->d_sums);
  dfree(c->d_counter);
  dfree(c->d_sc);
  if (c->h_pin) cudaFreeHost(c->h_pin);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->own_stream && c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

const char* ssg_status_string(ssg_status s) {
  switch (s) {
    case SSG_OK: return "ok";
    case SSG_ERR_ARG: return "invalid argument";
    case SSG_ERR_CUDA: return "CUDA failure or no device";
    case SSG_ERR_NOMEM: return "device allocation failed";
    case SSG_ERR_BUDGET: return "request exceeds the HBM budget";
    case SSG_MAXITER: return "iteration cap reached";
    case SSG_NONFINITE: return "non-finite residual";
    case SSG_ERR_MESH: return "inconsistent mesh connectivity";
    case SSG_ERR_STATE: return "call out of order";
    case SSG_ERR_TIMEOUT: return "deadline expired";
    case SSG_ERR_CANCELLED: return "cancelled";
  }
  return "unknown status";
}

const char* ssg_last_error(const ssg_context* c) { return c ? c->err.c_str() : ""; }

void* ssg_stream(const ssg_context* c) { return c ? (void*)c->stream : nullptr; }

ssg_status ssg_set_parameters(ssg_context* c, double dt, double visc, double dens) {
  if (!c) return SSG_ERR_ARG;
  if (!(dt > 0.0) || !(visc > 0.0)) return fail(c, SSG_ERR_ARG, "dt and visc must be > 0");
  c->dt = dt;
  c->visc = visc;
  c->dens = dens;
  return SSG_OK;
}

ssg_status ssg_set_precision(ssg_context* c, int precision) {
  if (!c) return SSG_ERR_ARG;
  if (precision != SSG_PRECISION_FP64 && precision != SSG_PRECISION_MIXED)
    return fail(c, SSG_ERR_ARG, "unknown precision");
  c->precision = precision;
  return SSG_OK;
}

ssg_status ssg_set_graphs(ssg_context* c, int enable) {
  if (!c) return SSG_ERR_ARG;
  c->graphs = enable != 0;
  return SSG_OK;
}

ssg_status ssg_setup_mesh(ssg_context* c, int n, int nel, const double* vertices,
                          const int* neigh) {
  if (!c || !vertices || !neigh) return SSG_ERR_ARG;
  SSG_CUDA(c, cudaSetDevice(c->device));
  free_mesh(c);
  c->host = ssg::HostMesh();
  ssg_status st = build_mesh(c->host, n, nel, vertices, neigh, c->err, c->setup_opts,
                             c->svvn, c->svva);
  if (st != SSG_OK) return st;
  return upload_all(c);
}

ssg_status ssg_gll(int n, double* points, double* weights) {
  if (n < 2 || n > SSG_MAXN || !points || !weights) return SSG_ERR_ARG;
  gll_basis(n, points, weights);
  return SSG_OK;
}

ssg_status ssg_set_setup_options(ssg_context* c, unsigned flags) {
  if (!c) return SSG_ERR_ARG;
  if (flags & ~(SSG_SETUP_NO_DEALIAS | SSG_SETUP_NO_PARTICLES | SSG_SETUP_OPPOSITE_PAIRING))
    return fail(c, SSG_ERR_ARG, "unknown set-up option");
  c->setup_opts = flags;
  return SSG_OK;
}

ssg_status ssg_set_svv(ssg_context* c, int svvn, double svva) {
  if (!c) return SSG_ERR_ARG;
  if (!std::isfinite(svva) || svva < 0.0)
    return fail(c, SSG_ERR_ARG, "svva must be finite and >= 0");
  c->svvn = svvn;
  c->svva = svva;
  return SSG_OK;
}

ssg_status ssg_memory_info(const ssg_context* c, size_t* bytes) {
  if (!c || !bytes) return SSG_ERR_ARG;
  *bytes = c->dev_bytes;
  return SSG_OK;
}

ssg_status ssg_setup_connectivity(ssg_context* c, int nel, const int* neigh) {
  if (!c || !neigh || nel <= 0) return SSG_ERR_ARG;
  SSG_CUDA(c, cudaSetDevice(c->device));
  free_mesh(c);
  c->host = ssg::HostMesh();
  c->host.nel = nel;
  c->host.neigh.assign(neigh, neigh + 26 * (size_t)nel);
  return build_pairs(c->host, c->err);
}

ssg_status ssg_setup_level(ssg_context* c, int level, int n, const double* deriv,
                           const double* svv_deriv, const double* weights,
                           const double* geom, const double* jac_det,
                           const double* interp) {
  if (!c || !deriv || !weights || !geom || !jac_det) return SSG_ERR_ARG;
  ssg::HostMesh& H = c->host;
  if (H.nel <= 0) return fail(c, SSG_ERR_STATE, "ssg_setup_connectivity first");
  if (level < 0 || level >= SSG_MAXLEV || n < 2 || n > 12)
    return fail(c, SSG_ERR_ARG, "bad level or order");
  if (level > 0 && (!interp || H.lev[level - 1].n == 0))
    return fail(c, SSG_ERR_STATE, "levels must be set in order, with interp");
  ssg::HostLevel& L = H.lev[level];
  L = ssg::HostLevel();
  L.n = n;
  L.nt = (size_t)n * n * n;
  const size_t np = L.nt * H.nel;
  L.x.resize(n);
  L.w.assign(weights, weights + n);
  gll_basis(n, L.x.data(), std::vector<double>(n).data());
  L.D.resize(n * n);
  L.S.resize(n * n);
  // stored d[j][i] = D_ij  ->  D[i*n+j]
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      L.D[i * n + j] = deriv[j * n + i];
      L.S[i * n + j] = (svv_deriv ? svv_deriv : deriv)[j * n + i];
    }
  for (int a = 0; a < 6; ++a) L.g[a].assign(geom + a * np, geom + (a + 1) * np);
  L.det.assign(jac_det, jac_det + np);
  if (level > 0) {
    const int nf = H.lev[level - 1].n;
    L.jf.resize((size_t)nf * n);
    // stored interp[p][i] (p coarse, i fine) -> jf[i*n+p]
    for (int p = 0; p < n; ++p)
      for (int i = 0; i < nf; ++i) L.jf[i * n + p] = interp[p * nf + i];
  }
  if (level == 0) H.n = n;
  if (level + 1 > H.nlev) H.nlev = level + 1;
  return SSG_OK;
}

ssg_status ssg_setup_finish(ssg_context* c) {
  if (!c) return SSG_ERR_ARG;
  if (c->host.nlev < 1) return fail(c, SSG_ERR_STATE, "no levels set");
  if (c->host.lev[c->host.nlev - 1].n != 2)
    return fail(c, SSG_ERR_STATE, "the coarsest level must have order 2");
  SSG_CUDA(c, cudaSetDevice(c->device));
  return upload_all(c);
}

ssg_status ssg_mesh_info(const ssg_context* c, int* n, int* nel, int* nlevels, int* orders) {
  if (!c) return SSG_ERR_ARG;
  if (n) *n = c->n;
  if (nel) *nel = c->nel;
  if (nlevels) *nlevels = c->nlev;
  if (orders)
    for (int l = 0; l < c->nlev; ++l) orders[l] = c->orders[l];
  return c->ready ? SSG_OK : SSG_ERR_STATE;
}

ssg_status ssg_level_data(ssg_context* c, int level, int which, double* dst) {
  SSG_TRY(need_ready(c));
  if (level < 0 || level >= c->nlev || !dst) return fail(c, SSG_ERR_ARG, "bad level");
  const ssg::DevLevel& d = c->lev[level];
  const size_t np = d.npts;
  const double* src = nullptr;
  std::vector<double> tmp;
  if (which >= 0 && which < 6) {
    SSG_CUDA(c, cudaStreamSynchronize(c->stream));
    SSG_CUDA(c, cudaMemcpy(dst, d.gf + which * np, np * sizeof(double), cudaMemcpyDeviceToHost));
    if (d.n == 8) {
      // back from the tensor-core operator's fragment order
      std::vector<double> frag(dst, dst + np);
      for (size_t e = 0; e < np / d.nt; ++e)
        for (size_t q = 0; q < d.nt; ++q)
          dst[e * d.nt + q] = frag[e * d.nt + ax8_fragment_index((int)q)];
    }
    return SSG_OK;
  } else if (which == 6)
    src = d.bj;
  else if (which == 7)
    src = d.dinv_p;
  else if (which == 8) {
    SSG_TRY(helmholtz_diag_update(c));
    src = d.dinv_h;
  } else if (which == 9) {
    std::vector<uint8_t> mu(np);
    SSG_CUDA(c, cudaMemcpy(mu.data(), d.mult, np, cudaMemcpyDeviceToHost));
    for (size_t q = 0; q < np; ++q) dst[q] = 1.0 / (double)mu[q];
    return SSG_OK;
  } else if (which == 10) {
    if (d.mask)
      src = d.mask;
    else {
      std::fill(dst, dst + np, 1.0);
      return SSG_OK;
    }
  } else if (which == 11 && level == 0)
    src = c->inv_mass;
  else if (which >= 12 && which <= 14) {
    const auto& g = c->host.lev[level].grid[which - 12];
    if (g.size() != np) return fail(c, SSG_ERR_STATE, "grid not available");
    std::copy(g.begin(), g.end(), dst);
    return SSG_OK;
  } else
    return fail(c, SSG_ERR_ARG, "bad selector");
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  SSG_CUDA(c, cudaMemcpy(dst, src, np * sizeof(double), cudaMemcpyDeviceToHost));
  return SSG_OK;
}

ssg_status ssg_global_opeval(ssg_context* c, int var, const double* p, double* ap) {
  SSG_TRY(need_ready(c));
  const size_t np = c->lev[0].npts;
  const double* dp;
  double* dap;
  SSG_TRY(stage_in(c, 0, p, np, &dp));
  SSG_TRY(stage_out(c, 1, ap, np, &dap));
  SSG_TRY(op_apply(c, 0, var, false, dp, dap, true));
  return stage_back(c, ap, dap, np);
}

ssg_status ssg_local_opeval(ssg_context* c, int var, const double* p, double* ap) {
  SSG_TRY(need_ready(c));
  const size_t np = c->lev[0].npts;
  const double* dp;
  double* dap;
  SSG_TRY(stage_in(c, 0, p, np, &dp));
  SSG_TRY(stage_out(c, 1, ap, np, &dap));
  SSG_TRY(op_apply(c, 0, var, false, dp, dap, false));
  return stage_back(c, ap, dap, np);
}

ssg_status ssg_direct_stiffness_summation(ssg_context* c, double* u) {
  SSG_TRY(need_ready(c));
  const size_t np = c->lev[0].npts;
  const double* du;
  SSG_TRY(stage_in(c, 0, u, np, &du));
  // DSS is out of place: gather from a copy
  double* tmp = c->d_stage[1];
  SSG_CUDA(c, cudaMemcpyAsync(tmp, du, np * sizeof(double), cudaMemcpyDeviceToDevice,
                              c->stream));
  double* dout = (double*)du;
  if (!is_device_ptr(u)) dout = c->d_stage[0];
  SSG_CUDA(c, run_dss(c->stream, DSS_PLAIN, false, c->n, c->nel, tmp, dout, c->d_nbreg,
                      c->lev[0].dss_ec,
                      nullptr, nullptr, nullptr, nullptr));
  return stage_back(c, u, dout, np);
}

ssg_status ssg_global_dot_product(ssg_context* c, const double* x, const double* y,
                                  double* out) {
  SSG_TRY(need_ready(c));
  if (!out) return SSG_ERR_ARG;
  const size_t np = c->lev[0].npts;
  const double *dx, *dy;
  SSG_TRY(stage_in(c, 0, x, np, &dx));
  SSG_TRY(stage_in(c, 1, y, np, &dy));
  const int nb = vec_blocks(np);
  PtrList pl;
  pl.p[0] = dy;
  ScalarOp op;
  op.sums = c->d_sums;
  op.counter = c->d_counter;
  SSG_CUDA(c, run_dots(c->stream, false, np, dx, pl, 1, c->lev[0].mult, c->d_part, nb, &op));
  SSG_CUDA(c, cudaMemcpyAsync(c->h_pin, c->d_sums, sizeof(double), cudaMemcpyDeviceToHost,
                              c->stream));
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  *out = c->h_pin[0];
  return SSG_OK;
}

ssg_status ssg_inverse_mass(ssg_context* c, double* u) {
  SSG_TRY(need_ready(c));
  const size_t np = c->lev[0].npts;
  const double* du;
  SSG_TRY(stage_in(c, 0, u, np, &du));
  SSG_CUDA(c, run_mul(c->stream, false, np, (void*)du, c->inv_mass));
  return stage_back(c, u, du, np);
}

static void timing_begin(ssg_context* c) { cudaEventRecord(c->ev0, c->stream); }

static double timing_end(ssg_context* c) {
  cudaEventRecord(c->ev1, c->stream);
  cudaEventSynchronize(c->ev1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  return ms;
}

ssg_status ssg_solve_poisson_cg(ssg_context* c, const double* f, double* u, double eps,
                                int max_iter, ssg_solve_info* info) {
  SSG_TRY(need_ready(c));
  if (max_iter <= 0) return fail(c, SSG_ERR_ARG, "max_iter must be positive");
  const size_t np = c->lev[0].npts;
  const double* df;
  const double* du0;
  SSG_TRY(stage_in(c, 0, f, np, &df));
  SSG_TRY(stage_in(c, 1, u, np, &du0));
  SSG_TRY(ensure_workspace(c));
  timing_begin(c);
  ssg_status st = fcg_solve(c, df, (double*)du0, eps, max_iter, info);
  const double ms = timing_end(c);
  if (info) info->solve_ms = ms;
  if (st != SSG_OK && st != SSG_MAXITER) return st;
  ssg_status st2 = stage_back(c, u, du0, np);
  return st2 != SSG_OK ? st2 : st;
}

ssg_status ssg_conjugate_gradient(ssg_context* c, int var, const double* f, double* u,
                                  double eps, int max_iter, ssg_solve_info* info) {
  SSG_TRY(need_ready(c));
  if (max_iter <= 0) return fail(c, SSG_ERR_ARG, "max_iter must be positive");
  if (var < SSG_PRESSURE || var > SSG_Z_VELOCITY) return fail(c, SSG_ERR_ARG, "bad var");
  const size_t np = c->lev[0].npts;
  const double* df;
  const double* du0;
  SSG_TRY(stage_in(c, 0, f, np, &df));
  SSG_TRY(stage_in(c, 1, u, np, &du0));
  SSG_TRY(ensure_workspace(c));
  // the reference masks f in place; work on a copy so the caller's f stays
  double* fc = c->d_stage[2];
  SSG_CUDA(c, cudaMemcpyAsync(fc, df, np * sizeof(double), cudaMemcpyDeviceToDevice,
                              c->stream));
  if (var != SSG_PRESSURE) SSG_TRY(helmholtz_diag_update(c));
  double* hist_d = nullptr;
  int cap = 0;
  if (info && info->history && info->history_cap > 0) {
    cap = std::min(info->history_cap, max_iter);
    SSG_CUDA(c, cudaMalloc(&hist_d, cap * sizeof(double)));
  }
  timing_begin(c);
  ssg_status st = cg_solve(c, 0, var, false, fc, (double*)du0, eps, max_iter, FR_HELM,
                           hist_d, cap, true);
  const double ms = timing_end(c);
  if (info) {
    double* fr = c->d_sc + FR_HELM * F_SIZE;
    double h[F_SIZE];
    cudaMemcpy(h, fr, sizeof(h), cudaMemcpyDeviceToHost);
    info->iterations = (int)h[F_ITER];
    info->residual = h[F_ERR];
    info->initial_residual = h[F_ERR0];
    info->solve_ms = ms;
    info->history_len = std::min((int)h[F_ITER], cap);
    if (hist_d) {
      cudaMemcpy(info->history, hist_d, info->history_len * sizeof(double),
                 cudaMemcpyDeviceToHost);
    }
  }
  if (hist_d) cudaFree(hist_d);
  if (st != SSG_OK && st != SSG_MAXITER) return st;
  ssg_status st2 = stage_back(c, u, du0, np);
  return st2 != SSG_OK ? st2 : st;
}

ssg_status ssg_solve_helmholtz_cg(ssg_context* c, int var, const double* f, double* u,
                                  double eps, int max_iter, ssg_solve_info* info) {
  if (var < SSG_X_VELOCITY || var > SSG_Z_VELOCITY)
    return ssg::fail(c, SSG_ERR_ARG, "Helmholtz var must be a velocity component");
  return ssg_conjugate_gradient(c, var, f, u, eps, max_iter, info);
}

ssg_status ssg_multigrid_preconditioner(ssg_context* c, const double* r, double* z,
                                        double eps) {
  SSG_TRY(need_ready(c));
  const size_t np = c->lev[0].npts;
  const double* dr;
  double* dz;
  SSG_TRY(stage_in(c, 0, r, np, &dr));
  SSG_TRY(stage_out(c, 1, z, np, &dz));
  SSG_TRY(ensure_workspace(c));
  SSG_TRY(mg_apply(c, dr, dz, eps));
  return stage_back(c, z, dz, np);
}

ssg_status ssg_jacobi_preconditioner(ssg_context* c, int var, const double* r, double* z) {
  SSG_TRY(need_ready(c));
  if (var < SSG_PRESSURE || var > SSG_Z_VELOCITY) return fail(c, SSG_ERR_ARG, "bad var");
  const DevLevel& L = c->lev[0];
  const size_t np = L.npts;
  const double* dr;
  double* dz;
  SSG_TRY(stage_in(c, 0, r, np, &dr));
  SSG_TRY(stage_out(c, 1, z, np, &dz));
  SSG_TRY(ensure_workspace(c));
  if (var != SSG_PRESSURE) SSG_TRY(helmholtz_diag_update(c));
  // z = r .* diag^-1 of the variable's operator (the partial sums of w z the
  // kernel also forms are not used here)
  SSG_CUDA(c, run_jacobi(c->stream, false, np, dr, var == SSG_PRESSURE ? L.dinv_p : L.dinv_h,
                         L.mult, dz, c->d_part, vec_blocks(np)));
  return stage_back(c, z, dz, np);
}

ssg_status ssg_setup_dealias(ssg_context* c, int m, const double* deriv,
                             const double* weights, const double* tinv_jac,
                             const double* jac_det, const double* interp) {
  if (!c || !deriv || !weights || !tinv_jac || !jac_det || !interp) return SSG_ERR_ARG;
  ssg::HostMesh& H = c->host;
  if (H.nel <= 0 || H.lev[0].n == 0)
    return fail(c, SSG_ERR_STATE, "connectivity and level 0 first");
  if (m < 2 || m > SSG_MAXN) return fail(c, SSG_ERR_ARG, "bad dealiasing order");
  const int n = H.lev[0].n;
  ssg::HostLevel& L = H.conv;
  L = ssg::HostLevel();
  L.n = m;
  L.nt = (size_t)m * m * m;
  const size_t mp = L.nt * H.nel;
  L.x.resize(m);
  gll_basis(m, L.x.data(), std::vector<double>(m).data());
  L.w.assign(weights, weights + m);
  L.D.resize((size_t)m * m);
  // stored d[j][i] = D_ij  ->  D[i*m+j]
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) L.D[i * m + j] = deriv[j * m + i];
  for (int a = 0; a < 9; ++a) L.tinv[a].assign(tinv_jac + a * mp, tinv_jac + (a + 1) * mp);
  L.det.assign(jac_det, jac_det + mp);
  // stored interp[p][i] (p: n-point node, i: m-point node) -> jconv[i*n+p]
  H.jconv.resize((size_t)m * n);
  for (int p = 0; p < n; ++p)
    for (int i = 0; i < m; ++i) H.jconv[i * n + p] = interp[p * m + i];
  H.has_conv = true;
  if (!c->ready) return SSG_OK;
  SSG_CUDA(c, cudaSetDevice(c->device));
  return upload_conv(c);
}

ssg_status ssg_setup_particle_geometry(ssg_context* c, const double* points,
                                       const double* jac, const double* tinv_jac) {
  if (!c || !jac || !tinv_jac) return SSG_ERR_ARG;
  ssg::HostMesh& H = c->host;
  if (H.nel <= 0 || H.lev[0].n == 0)
    return fail(c, SSG_ERR_STATE, "connectivity and level 0 first");
  ssg::HostLevel& L = H.lev[0];
  const size_t np = L.nt * H.nel;
  for (int a = 0; a < 9; ++a) {
    L.jac[a].assign(jac + a * np, jac + (a + 1) * np);
    L.tinv[a].assign(tinv_jac + a * np, tinv_jac + (a + 1) * np);
  }
  if (points)
    H.ppoints.assign(points, points + L.n);
  else
    H.ppoints.clear();
  H.has_particle_geom = true;
  if (!c->ready) return SSG_OK;
  SSG_CUDA(c, cudaSetDevice(c->device));
  return upload_particle_geom(c);
}

ssg_status ssg_convection_operator(ssg_context* c, const double* u, const double* v,
                                   double* udv) {
  SSG_TRY(need_ready(c));
  if (!c->conv_w) return fail(c, SSG_ERR_STATE, "no dealiasing grid set up");
  const size_t np = 3 * c->lev[0].npts;
  const double *du, *dv;
  double* dout;
  SSG_TRY(stage_in(c, 0, u, np, &du));
  // a field advecting itself is staged once (the self-convection kernel
  // keys on the two pointers being equal)
  if (v == u)
    dv = du;
  else
    SSG_TRY(stage_in(c, 1, v, np, &dv));
  SSG_TRY(stage_out(c, 2, udv, np, &dout));
  SSG_CUDA(c, run_convection(c->stream, c->nel, 0, c->nel, c->n, c->m, du, dv, dout,
                             conv_geom(c)));
  return stage_back(c, udv, dout, np);
}

ssg_status ssg_convection_elements(ssg_context* c, int first, int count, const double* u,
                                   const double* v, double* udv) {
  SSG_TRY(need_ready(c));
  if (!c->conv_w) return fail(c, SSG_ERR_STATE, "no dealiasing grid set up");
  if (first < 0 || count < 0 || first > c->nel || count > c->nel - first)
    return fail(c, SSG_ERR_ARG, "element range outside the mesh");
  if (count == 0) return SSG_OK;
  const size_t np = 3 * (size_t)count * c->lev[0].nt;
  const double *du, *dv;
  double* dout;
  SSG_TRY(stage_in(c, 0, u, np, &du));
  if (v == u)
    dv = du;
  else
    SSG_TRY(stage_in(c, 1, v, np, &dv));
  SSG_TRY(stage_out(c, 2, udv, np, &dout));
  SSG_CUDA(c, run_convection(c->stream, count, first, c->nel, c->n, c->m, du, dv, dout,
                             conv_geom(c)));
  return stage_back(c, udv, dout, np);
}

ssg_status ssg_set_particle_velocity(ssg_context* c, const double* ur) {
  SSG_TRY(need_ready(c));
  if (!ur) return fail(c, SSG_ERR_ARG, "null velocity");
  if (!c->p_jac) return fail(c, SSG_ERR_STATE, "no particle geometry set up");
  const size_t count = 9 * c->lev[0].npts;
  SSG_CUDA(c, cudaMemcpyAsync(c->p_ur, ur, count * sizeof(double), cudaMemcpyDefault,
                              c->stream));
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  c->has_ur = true;
  return SSG_OK;
}

ssg_status ssg_integrate_particle_equations(ssg_context* c, size_t np, double* state,
                                            int* ints, double t, double dt, int* passes) {
  SSG_TRY(need_ready(c));
  if (!c->p_jac) return fail(c, SSG_ERR_STATE, "no particle geometry set up");
  if (!c->has_ur) return fail(c, SSG_ERR_STATE, "ssg_set_particle_velocity first");
  if (!(dt > 0.0)) return fail(c, SSG_ERR_ARG, "dt must be > 0");
  if (np > 0 && (!state || !ints)) return fail(c, SSG_ERR_ARG, "null particle arrays");
  const bool dev_state = np > 0 && is_device_ptr(state);
  const bool dev_ints = np > 0 && is_device_ptr(ints);
  double* ds = state;
  int* di = ints;
  if (np > 0 && (!dev_state || !dev_ints) && np > c->p_cap) {
    dfree(c->p_state);
    if (c->p_ints) cudaFree(c->p_ints);
    c->p_state = nullptr;
    c->p_ints = nullptr;
    c->p_cap = 0;
    SSG_TRY(dalloc(c, &c->p_state, 8 * np));
    if (cudaMalloc(&c->p_ints, 3 * np * sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      return fail(c, SSG_ERR_NOMEM, "particle staging");
    }
    c->p_cap = np;
  }
  if (np > 0 && !dev_state) {
    ds = c->p_state;
    SSG_CUDA(c, cudaMemcpyAsync(ds, state, 8 * np * sizeof(double), cudaMemcpyHostToDevice,
                                c->stream));
  }
  if (np > 0 && !dev_ints) {
    di = c->p_ints;
    SSG_CUDA(c, cudaMemcpyAsync(di, ints, 3 * np * sizeof(int), cudaMemcpyHostToDevice,
                                c->stream));
  }
  if (np > c->p_order_cap) {
    if (c->p_order) cudaFree(c->p_order);
    c->p_order = nullptr;
    c->p_order_cap = 0;
    if (cudaMalloc(&c->p_order, np * sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      c->p_order = nullptr;
      return fail(c, SSG_ERR_NOMEM, "particle order");
    }
    c->p_order_cap = np;
  }
  if (!c->p_bucket) {
    if (cudaMalloc(&c->p_bucket, 2 * ((size_t)c->nel + 1) * sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      c->p_bucket = nullptr;
      return fail(c, SSG_ERR_NOMEM, "particle buckets");
    }
  }
  SSG_CUDA(c, cudaMemsetAsync(c->d_passes, 0, sizeof(int), c->stream));
  SSG_CUDA(c, run_particles(c->stream, c->n, c->nel, c->lev[0].npts, c->p_x, c->p_ur,
                            c->p_jac, c->p_tinv, c->d_neigh, t, dt, np, ds, di, c->d_passes,
                            np > 0 ? c->p_order : nullptr, c->p_bucket));
  if (np > 0 && !dev_state)
    SSG_CUDA(c, cudaMemcpyAsync(state, ds, 8 * np * sizeof(double), cudaMemcpyDeviceToHost,
                                c->stream));
  if (np > 0 && !dev_ints)
    SSG_CUDA(c, cudaMemcpyAsync(ints, di, 3 * np * sizeof(int), cudaMemcpyDeviceToHost,
                                c->stream));
  int hp = 0;
  SSG_CUDA(c, cudaMemcpyAsync(c->h_pin, c->d_passes, sizeof(int), cudaMemcpyDeviceToHost,
                              c->stream));
  SSG_CUDA(c, cudaStreamSynchronize(c->stream));
  std::memcpy(&hp, c->h_pin, sizeof(int));
  // the reference's pass loop runs at least once, also without particles
  if (passes) *passes = hp > 1 ? hp : 1;
  return SSG_OK;
}

}  // extern "C"
