// reno_lanczos_expm: the Lanczos exponential psi <- exp(dt H_eff) psi of
// renormalizer/lib/krylov/krylov.py:27-84 (expm_krylov with hop_expr as the
// operator) behind one C call, so that a host without Python can drive the
// local updates of a sweep.
//
// Every matvec (reno_heff_apply) and vector operation (norm, the Lanczos
// step, the combination V c, allclose) runs on the device in FP64.  The host
// reads the Lanczos scalars only where the reference makes a decision with
// them: at its convergence tests (every even j > 5; its first approximation,
// at j = 4, has none to be compared with), where the breakdown test
// beta_i < 100 n eps is also applied to every beta since the previous one --
// the Krylov vectors up to a breakdown do not depend on what came after it,
// so the result and the count are the reference's.  The
// small tridiagonal eigenproblem of krylov.py:15-24 is solved on the host by
// implicit QL iterations with shifts (the EISPACK tql2 method of Bowdler,
// Martin, Reinsch and Wilkinson, Numer. Math. 11, 1968).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>
#include "reno_common.cuh"

using namespace reno;

namespace {

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

int64_t psi_elems(const reno_heff_desc* d) {
  if (d->nsite == 0) return (int64_t)d->ml * d->mr;
  if (d->nsite == 1) return (int64_t)d->ml * d->d1 * d->mr;
  return (int64_t)d->ml * d->d1 * d->d2 * d->mr;
}

// scal: the start norm, the allclose flag, then (alpha_0, beta_0, alpha_1, ...)
struct LzLayout {
  size_t V, w, scal, coef, heff, vec, total;
};

int lz_layout(const reno_heff_desc* d, int kmax, LzLayout& L) {
  size_t hb = 0, vb = 0;
  if (reno_heff_workspace_bytes(d, &hb) != RENO_OK) return RENO_ERR_INVALID;
  const int64_t n = psi_elems(d);
  if (reno_vec_grouped_workspace_bytes(1, &vb) != RENO_OK) return RENO_ERR_INVALID;
  const size_t vbytes = (size_t)n * 16;
  size_t o = 0;
  L.V = o;
  o = al256(o + (size_t)(kmax + 1) * vbytes);
  L.w = o;
  o = al256(o + vbytes);
  L.scal = o;
  o = al256(o + (2 * (size_t)kmax + 4) * sizeof(double));
  L.coef = o;
  o = al256(o + 4 * ((size_t)kmax + 1) * sizeof(double));
  L.heff = o;
  o = al256(o + hb);
  L.vec = o;
  o = al256(o + vb);
  L.total = o;
  return RENO_OK;
}

// Eigenvalues (d, overwritten) and eigenvectors (Z, k x k row-major, column j
// = eigenvector j) of the symmetric tridiagonal matrix with diagonal d and
// off-diagonal e[0..k-2].  Implicit QL with a shift from the leading 2 x 2
// block, one plane rotation at a time, accumulated into Z.
bool tridiag_eig(int k, std::vector<double>& d, std::vector<double> e, std::vector<double>& Z) {
  Z.assign((size_t)k * k, 0.0);
  for (int i = 0; i < k; ++i) Z[(size_t)i * k + i] = 1.0;
  e.resize(k, 0.0);
  e[k - 1] = 0.0;
  for (int l = 0; l < k; ++l) {
    for (int iter = 0;; ++iter) {
      int m = l;
      for (; m < k - 1; ++m) {
        const double dd = std::fabs(d[m]) + std::fabs(d[m + 1]);
        if (std::fabs(e[m]) <= DBL_EPSILON * dd) break;
      }
      if (m == l) break;
      if (iter >= 64) return false;
      // shift: the eigenvalue of the leading 2 x 2 block nearer to d[l]
      double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
      double r = std::hypot(g, 1.0);
      g = d[m] - d[l] + e[l] / (g + std::copysign(r, g));
      double s = 1.0, c = 1.0, p = 0.0;
      bool deflated = false;
      for (int i = m - 1; i >= l; --i) {
        const double f = s * e[i], b = c * e[i];
        r = std::hypot(f, g);
        e[i + 1] = r;
        if (r == 0.0) {  // split: the rotation chain stops here
          d[i + 1] -= p;
          e[m] = 0.0;
          deflated = true;
          break;
        }
        s = f / r;
        c = g / r;
        g = d[i + 1] - p;
        r = (d[i] - g) * s + 2.0 * c * b;
        p = s * r;
        d[i + 1] = g + p;
        g = c * r - b;
        for (int q = 0; q < k; ++q) {
          double* zq = &Z[(size_t)q * k];
          const double t = zq[i + 1];
          zq[i + 1] = s * zq[i] + c * t;
          zq[i] = c * zq[i] - s * t;
        }
      }
      if (deflated) continue;
      d[l] -= p;
      e[l] = g;
      e[m] = 0.0;
    }
  }
  return true;
}

// krylov.py:15-24: coefficients u (nrmv exp(dt w) u[0]) of the Krylov vectors
// for the leading tridiagonal block of order k, as (re, im) pairs
// (ab = alpha_0, beta_0, alpha_1, ...)
bool tridiag_coeffs(int k, const double* ab, double nrmv, double dt_re, double dt_im, double* coef) {
  std::vector<double> d(k), e(k > 0 ? k - 1 : 0), Z;
  for (int i = 0; i < k; ++i) {
    d[i] = ab[2 * i];
    if (i + 1 < k) e[i] = ab[2 * i + 1];
  }
  for (double x : d)
    if (!std::isfinite(x)) return false;
  for (double x : e)
    if (!std::isfinite(x)) return false;
  if (!tridiag_eig(k, d, e, Z)) return false;
  std::fill(coef, coef + 2 * (size_t)k, 0.0);
  for (int j = 0; j < k; ++j) {
    const double mag = nrmv * std::exp(dt_re * d[j]) * Z[j];  // Z[0][j]
    const double cr = mag * std::cos(dt_im * d[j]), ci = mag * std::sin(dt_im * d[j]);
    for (int i = 0; i < k; ++i) {
      coef[2 * i] += Z[(size_t)i * k + j] * cr;
      coef[2 * i + 1] += Z[(size_t)i * k + j] * ci;
    }
  }
  return true;
}

}  // namespace

extern "C" int reno_lanczos_workspace_bytes(const reno_heff_desc* desc, int32_t kmax, size_t* bytes) {
  if (!desc || !bytes || kmax < 1) return RENO_ERR_INVALID;
  LzLayout L;
  const int rc = lz_layout(desc, kmax, L);
  if (rc != RENO_OK) return rc;
  *bytes = L.total;
  return RENO_OK;
}

extern "C" int reno_lanczos_coefficients(int32_t count, const int32_t* k, const double* scal, int64_t ld,
                                         const double* dt, double* coef) {
  if (count < 0 || (count > 0 && (!k || !scal || !dt || !coef))) return RENO_ERR_INVALID;
  for (int i = 0; i < count; ++i) {
    if (k[i] < 1 || ld < 2 * (int64_t)k[i]) return RENO_ERR_INVALID;
    const double* s = scal + i * ld;
    if (!tridiag_coeffs(k[i], s + 1, s[0], dt[2 * i], dt[2 * i + 1], coef)) return RENO_ERR_NONFINITE;
    coef += 2 * (size_t)k[i];
  }
  return RENO_OK;
}

// The host's share of an exponential is one read of the scalars, one upload
// of coefficients and one read of the flag per convergence test, and tests
// begin at j = 6: the reference's first approximation (j = 4) is only compared
// at j = 6, where RENO_VOP_CHECK forms both from one read of the vectors.
// (Pageable host memory: the copies return once it has been read or staged, and a
// pinned block would have to be allocated in a hot call.)
// The tests write their approximation to out; in place they write it to w,
// free between a step and the next matvec, so that psi is still the start
// vector when the call fails.
// With prev, a call with k0 vectors went before and ended with
// RENO_ERR_WORKSPACE: its vectors and scalars are taken over from its workspace
// and the recurrence goes on at j = k0.  No decision looks further back than
// the scalars (both approximations of a test are formed from the vectors), so the result
// is bit for bit that of one call with enough vectors.
static int lanczos_run(reno_ctx* ctx, const reno_heff_desc* desc, const void* L, const void* W1, const void* W2,
                       const void* R, double dt_re, double dt_im, const void* psi, void* out, int32_t kmax, int32_t k0,
                       const void* prev, int32_t* out_k, void* ws, size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (!desc || !(psi || prev) || !out || !out_k || !ws || kmax < 1 || (prev && (k0 < 1 || k0 >= kmax)))
    return set_error(ctx, RENO_ERR_INVALID, "reno_lanczos_expm: null argument or bad vector count");
  if (desc->psi_dtype != RENO_C128)
    return set_error(ctx, RENO_ERR_INVALID, "reno_lanczos_expm: psi must be complex128");
  *out_k = 0;
  LzLayout Lz;
  if (lz_layout(desc, kmax, Lz) != RENO_OK) return set_error(ctx, RENO_ERR_INVALID, "reno_lanczos_expm: bad descriptor");
  if (ws_bytes < Lz.total) return set_error(ctx, RENO_ERR_WORKSPACE, "reno_lanczos_expm: workspace too small");
  const int64_t n = psi_elems(desc);
  char* base = static_cast<char*>(ws);
  double2* V = reinterpret_cast<double2*>(base + Lz.V);
  double2* w = reinterpret_cast<double2*>(base + Lz.w);
  void* approx = out == psi ? static_cast<void*>(w) : out;
  double* scal = reinterpret_cast<double*>(base + Lz.scal);
  double* ab = scal + 2;
  double* dcoef = reinterpret_cast<double*>(base + Lz.coef);
  void* hws = base + Lz.heff;
  void* vws = base + Lz.vec;
  size_t hbytes = 0, vbytes = 0;
  reno_heff_workspace_bytes(desc, &hbytes);
  reno_vec_grouped_workspace_bytes(1, &vbytes);
  cudaStream_t st = ctx->stream;
  const double thresh = 100.0 * (double)n * DBL_EPSILON;
  int rc;
#define LZ_TRY(call)              \
  do {                            \
    rc = (call);                  \
    if (rc != RENO_OK) return rc; \
  } while (0)
  std::vector<double> host(2 * (size_t)kmax + 4), hcoef(4 * ((size_t)kmax + 1));  // read / sent
  reno_vec_item it{};
  it.n = n;
  it.dtype = RENO_C128;
  it.ldv = n;
  auto read = [&](const double* from, size_t count) -> int {
    int r = check_cuda(ctx, cudaMemcpyAsync(host.data() + (from - scal), from, count * sizeof(double),
                                            cudaMemcpyDeviceToHost, st), "reno_lanczos_expm: scalars");
    return r != RENO_OK ? r : check_cuda(ctx, cudaStreamSynchronize(st), "reno_lanczos_expm: sync");
  };
  auto send = [&](size_t count) -> int {
    return check_cuda(ctx, cudaMemcpyAsync(dcoef, hcoef.data(), count * sizeof(double), cudaMemcpyHostToDevice, st),
                      "reno_lanczos_expm: coefficients");
  };
  auto coefficients = [&](int k, double* to) -> int {
    return tridiag_coeffs(k, host.data() + 2, host[0], dt_re, dt_im, to)
               ? RENO_OK
               : set_error(ctx, RENO_ERR_NONFINITE, "reno_lanczos_expm: Lanczos scalars are not finite");
  };
  const int j0 = prev ? k0 : 0;
  if (prev) {
    LzLayout P;
    lz_layout(desc, k0, P);
    const char* from = static_cast<const char*>(prev);
    cudaError_t e = cudaMemcpyAsync(V, from + P.V, ((size_t)k0 + 1) * n * sizeof(double2), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(scal, from + P.scal, (2 + 2 * (size_t)k0) * sizeof(double), cudaMemcpyDeviceToDevice, st);
    LZ_TRY(check_cuda(ctx, e, "reno_lanczos_expm_resume: copy"));
  } else {
    LZ_TRY(reno_vec_norm(ctx, n, RENO_C128, psi, scal, vws, vbytes));
    LZ_TRY(reno_vec_scale_inv(ctx, n, RENO_C128, psi, scal, V));
  }
  int checked = j0;  // a call that ran out of vectors looked at every beta it has
  for (int j = j0; j < n; ++j) {
    if (j >= kmax) {
      *out_k = kmax;
      return set_error(ctx, RENO_ERR_WORKSPACE, "reno_lanczos_expm: no convergence within kmax = " +
                                                    std::to_string(kmax) + " Krylov vectors; raise kmax");
    }
    double2* vj = V + (size_t)j * n;
    LZ_TRY(heff_apply_prepared(ctx, desc, L, W1, W2, R, vj, w, hws, hbytes, j > j0));
    const bool exhausted = (j == n - 1);
    it.j = j;
    it.scalars = ab;
    if (exhausted) {
      LZ_TRY(reno_krylov_alpha(ctx, n, RENO_C128, w, vj, ab, j, vws, vbytes));
    } else {
      it.x = vj;
      it.y = j > 0 ? vj - n : nullptr;
      it.out = w;
      LZ_TRY(reno_vec_grouped(ctx, RENO_VOP_STEP, 1, &it, 0.0, 0.0, vws, vbytes));
    }
    const bool last_chance = j + 1 >= kmax;  // a breakdown before kmax is still found
    if (!(exhausted || (j > 5 && j % 2 == 0) || last_chance)) continue;
    LZ_TRY(read(scal, 2 + 2 * (size_t)j + (exhausted ? 1 : 2)));
    if (!(host[0] > 0.0) || !std::isfinite(host[0]))
      return set_error(ctx, RENO_ERR_NONFINITE, "reno_lanczos_expm: start vector is zero or not finite");
    int k = exhausted ? j + 1 : 0;  // vectors of the final result, 0 = not known yet
    const int upto = exhausted ? j : j + 1;
    for (int i = checked; i < upto; ++i)
      if (host[2 + 2 * i + 1] < thresh) {  // the Krylov space closed at i; nothing after it is used
        k = i + 1;
        break;
      }
    checked = upto;
    if (k > 0) {
      LZ_TRY(coefficients(k, hcoef.data()));
      LZ_TRY(send(2 * (size_t)k));
      LZ_TRY(reno_vec_lincomb(ctx, n, k, RENO_C128, V, n, dcoef, out));
      *out_k = k;
      return RENO_OK;
    }
    if (!(j > 5 && j % 2 == 0)) continue;
    LZ_TRY(coefficients(j + 1, hcoef.data()));
    LZ_TRY(coefficients(j - 1, hcoef.data() + 2 * (size_t)(j + 1)));
    LZ_TRY(send(4 * (size_t)j));
    it.j = j + 1;
    it.x = V;
    it.y = nullptr;
    it.s = dcoef;
    it.out = approx;
    it.scalars = scal + 1;
    LZ_TRY(reno_vec_grouped(ctx, RENO_VOP_CHECK, 1, &it, 1e-5, 1e-8, vws, vbytes));
    it.s = nullptr;
    LZ_TRY(read(scal + 1, 1));
    if (host[1] == 1.0) {
      if (approx != out)
        LZ_TRY(check_cuda(ctx, cudaMemcpyAsync(out, approx, (size_t)n * sizeof(double2), cudaMemcpyDeviceToDevice, st),
                          "reno_lanczos_expm: copy out"));
      *out_k = j + 1;
      return RENO_OK;
    }
  }
#undef LZ_TRY
  return set_error(ctx, RENO_ERR_INVALID, "reno_lanczos_expm: empty vector");
}

extern "C" int reno_lanczos_expm(reno_ctx* ctx, const reno_heff_desc* desc, const void* L, const void* W1,
                                 const void* W2, const void* R, double dt_re, double dt_im, void* psi, int32_t kmax,
                                 int32_t* out_k, void* ws, size_t ws_bytes) {
  return reno_lanczos_expm_to(ctx, desc, L, W1, W2, R, dt_re, dt_im, psi, psi, kmax, out_k, ws, ws_bytes);
}

extern "C" int reno_lanczos_expm_to(reno_ctx* ctx, const reno_heff_desc* desc, const void* L, const void* W1,
                                    const void* W2, const void* R, double dt_re, double dt_im, const void* psi,
                                    void* out, int32_t kmax, int32_t* out_k, void* ws, size_t ws_bytes) {
  return lanczos_run(ctx, desc, L, W1, W2, R, dt_re, dt_im, psi, out, kmax, 0, nullptr, out_k, ws, ws_bytes);
}

extern "C" int reno_lanczos_expm_resume(reno_ctx* ctx, const reno_heff_desc* desc, const void* L, const void* W1,
                                        const void* W2, const void* R, double dt_re, double dt_im, void* out,
                                        int32_t kmax, int32_t prev_kmax, const void* prev_ws, int32_t* out_k, void* ws,
                                        size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (!prev_ws) return set_error(ctx, RENO_ERR_INVALID, "reno_lanczos_expm_resume: null previous workspace");
  return lanczos_run(ctx, desc, L, W1, W2, R, dt_re, dt_im, nullptr, out, kmax, prev_kmax, prev_ws, out_k, ws, ws_bytes);
}
