// Hermitian eigensolver for the truncation's Gram blocks: the leading kt
// eigenpairs of an n x n Hermitian matrix G (the QN-block Gram matrices of
// svd_qn.py:12-49 / mp.py:693-778, which the reference factorises with
// LAPACK gesdd), entirely on the device.
//
//   1. hetrd_kernel   Householder reduction G = Q T Q^H to a real symmetric
//                     tridiagonal T (d, e), one persistent cooperative launch.
//                     Step k forms reflector k from row k of the trailing
//                     matrix, then every CTA streams its rows of the trailing
//                     matrix once: it applies the rank-2 update of step k-1
//                     (lagged by one step) and accumulates y = A v_k in the
//                     same pass.  The only inter-CTA dependency per column is
//                     the sum of y^H v_k, so there is one grid barrier per
//                     column; each CTA recomputes v_k and w_k itself from
//                     row k and y (bitwise identical in every CTA: same data,
//                     same reduction order).  Reflector k is stored in row k.
//                     Matrices that fit the shared memory of a cluster
//                     (n <= 424) are reduced there (hetrd_cluster_kernel).
//   2. bisect_kernel  eigenvalues of T by Sturm-count multisection, one warp
//                     per eigenvalue, 32 points per round, signs of the leading
//                     minors without a division.
//   3. inviter_kernel eigenvectors of T by inverse iteration, one thread per
//                     eigenvalue: LU of T - lambda I with partial pivoting,
//                     three solves from a hashed start vector, in shared
//                     memory (inviter_smem_kernel) but for the largest.  The host
//                     orthonormalises the block (Householder QR) and checks the
//                     residuals ||T z - lambda z||.
//   4. back-transformation K = Q Z in blocks of 64 reflectors (compact WY
//                     form, three FP64 GEMMs per block, last block first).
//
// Every grid-barrier wait is bounded (2 s of wall clock by default, see
// reno_set_wait_limit_ns): on timeout the
// CTA raises the abort flag and a status word in the caller's workspace and
// returns; the others return at their next barrier.
#include <algorithm>
#include <cfloat>
#include <cstdlib>
#include <vector>
#include <cstddef>
#include "reno_common.cuh"
#include "gemm_fp64.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace reno {
namespace heev {

constexpr int THREADS = 256, WARPS = THREADS / 32;
constexpr int MAX_N = 4096;

struct Sync {
  unsigned count, gen;
  int abort, status;
};

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 conjg(double2 a) { return make_double2(a.x, -a.y); }

__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block sum in a fixed order (shuffle tree, then warps 0..NW-1); every
// thread gets the result
template <int NW>
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < NW; ++w) s += red[w];
  return s;
}

// grid barrier over the nblocks CTAs that share `s`: a monotonic arrival
// counter (no reset between columns), released by each CTA's thread 0 after
// a CTA barrier and acquired by polling, the ordering pattern of CUTLASS's
// generic barrier.  false when this or another CTA gave up (abort raised).
// skip_arrival (test hook only): this CTA does not arrive, so every wait of
// this barrier runs out after wait_ns.
__device__ bool grid_sync(Sync* s, unsigned nblocks, unsigned& epoch, int* ok_sh, uint64_t wait_ns,
                          bool skip_arrival) {
  __syncthreads();
  if (threadIdx.x == 0) {
    epoch += 1u;
    const unsigned target = epoch * nblocks;
    bool good = true;
    if (!skip_arrival) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&s->count) : "memory");
    volatile int* va = &s->abort;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0;; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&s->count) : "memory");
      if (v >= target) break;
      if ((it & 63u) == 63u) {
        if (*va) {
          good = false;
          break;
        }
        if (global_ns() - t0 > wait_ns) {
          atomicExch(&s->abort, 1);
          atomicCAS(&s->status, 0, 1);
          good = false;
          break;
        }
      }
    }
    *ok_sh = good && !*va;
  }
  __syncthreads();
  return *ok_sh != 0;
}

constexpr int HT = 512, HW = HT / 32;  // reduction kernel: 16 warps, one CTA per SM
constexpr int U1 = 4;                  // loads in flight per thread (rows k, y)
constexpr int U2 = 6;                  // loads in flight per lane per item (trailing rows)
constexpr int MAXM = 32;               // matrices per batched launch

// One matrix of a batched reduction: CTAs first .. first + nblk - 1 of the
// cooperative grid work on it, with their own barrier word and buffers.
struct HetrdProb {
  double2* A;
  int n;
  double* d;
  double* e;
  double2* tau;
  double2* Y;
  double2* P;
  Sync* sync;
  int first, nblk;
  double2* YP;  // lower-triangle reduction: YP_G x n partial sums of y (nullptr: not available)
};
// One matrix of the batched small-matrix reduction and of the batched
// eigenvalue / eigenvector stages (blockIdx.y = entry).
struct EigProb {
  double2* a;
  double2* tau;
  double* d;
  double* e;
  int n, kt;
  double* w;
  double* z;
  double* bnd;
  double* scr;
};
struct EigTable {
  int count;
  EigProb p[MAXM];
};

struct HetrdTable {
  int count;
  int skip_column;      // test hook: CTA 0 of matrix 0 skips its arrival after this column (-1: none)
  uint64_t wait_ns;     // limit of every grid-barrier wait
  HetrdProb p[MAXM];
};

// A: n x n row-major Hermitian (both triangles), overwritten: row k holds
// reflector k from column k+1 on.  Y: 2n, P: 2 * nblk scratch.  Every
// matrix of the table is reduced by its own share of the grid.
//
// Per column k (lagged: update k-1 is applied while column k is processed):
//   phase 1 (every CTA)  row k with update k-1 applied, reflector k;
//   phase 2              the trailing rows r > k are dealt round-robin to the
//                        matrix's CTAs (r = k + 1 + bid + j G); each CTA splits
//                        its rows into chunks of HCH columns and spreads the
//                        (row, chunk) items over its warps, two items in
//                        flight per warp: update k-1 applied and stored, the
//                        chunk's share of y_r = (A v_k)_r kept in shared
//                        memory and summed per row in chunk order;
//   grid barrier;
//   phase 3 (every CTA)  w_k from y and the CTA partials of y^H v_k, issued
//                        together with the loads of row k+1 for the next
//                        phase 1 (one round trip to L2 for both).
constexpr int HCH = 32 * U2;    // columns per phase-2 item
constexpr int PARTS = 1024;     // per-CTA (row, chunk) partial sums held at once

// one phase-2 item: update k-1 on U2 x 32 entries of a row (a: their loaded
// values), stored back; returns the lane's share of the row's y
__device__ __forceinline__ double2 hetrd_item(double2* __restrict__ row, int cbase, int n, double2 vpr, double2 wpr,
                                              const double2* vp, const double2* wp, const double2* vc,
                                              const double2 (&a)[U2]) {
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int u = 0; u < U2; ++u) {
    const int c = cbase + 32 * u;
    if (c < n) {
      const double2 x = csub(csub(a[u], cmulc(vpr, wp[c])), cmulc(wpr, vp[c]));
      __stcg(&row[c], x);
      acc = cadd(acc, cmul(x, vc[c]));
    }
  }
  return acc;
}

__global__ void __launch_bounds__(HT, 1) hetrd_kernel(const __grid_constant__ HetrdTable tab) {
  int pi = 0;
  while (pi + 1 < tab.count && (int)blockIdx.x >= tab.p[pi + 1].first) ++pi;
  const HetrdProb& PR = tab.p[pi];
  double2* __restrict__ A = PR.A;
  const int n = PR.n;
  double* __restrict__ d = PR.d;
  double* __restrict__ e = PR.e;
  double2* __restrict__ tau = PR.tau;
  double2* __restrict__ Y = PR.Y;
  double2* __restrict__ P = PR.P;
  Sync* sync = PR.sync;
  const int bid = (int)blockIdx.x - PR.first;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* vp = reinterpret_cast<double2*>(smem_raw);  // v of step k-1 (pending update)
  double2* wp = vp + n;                                // w of step k-1
  double2* vc = wp + n;                                // v of step k
  double2* parts = vc + n;                             // PARTS (row, chunk) partial sums of y
  __shared__ double red[HW];
  __shared__ double2 redc[HW];
  __shared__ double s_akk;
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = PR.nblk;
  unsigned gen = 0;
  for (int i = tid; i < n; i += HT) {
    vp[i] = make_double2(0.0, 0.0);
    wp[i] = make_double2(0.0, 0.0);
    vc[i] = make_double2(0.0, 0.0);
  }
  // row 0, the part phase 1 reads in its first pass (c = tid + u HT)
  double2 pre[U1];
#pragma unroll
  for (int u = 0; u < U1; ++u) {
    const int c = tid + u * HT;
    pre[u] = c < n ? __ldcg(&A[c]) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  // Shared-memory discipline: in phases 1 and 3 thread t owns the entries
  // c = k + t + j HT of vc (phase 1 of column k) and c = k + 1 + t + j HT of
  // vp, wp (phase 3 of column k), i.e. the same entries as phase 1 of column
  // k + 1, so those phases need no block barrier between them; every thread
  // recomputes the scalars that more than one thread needs (the Householder
  // scalars, the dot y^H v and the pending pivot entries v_{k-1}[k] = 1,
  // w_{k-1}[k]) with the same operations, so they agree bit for bit.
  double2 tk_prev = make_double2(0.0, 0.0), alph_prev = make_double2(0.0, 0.0), yk_prev = make_double2(0.0, 0.0);
  for (int k = 0; k < n - 1; ++k) {
    // ---- phase 1 (every CTA): row k with update k-1 applied, reflector k
    double2 vpk = make_double2(0.0, 0.0), wpk = make_double2(0.0, 0.0);
    if (k > 0) {
      vpk = make_double2(1.0, 0.0);
      wpk = cadd(cmul(tk_prev, yk_prev), cmul(alph_prev, vpk));
    }
    const double2* rowk = A + (size_t)k * n;
    double ss = 0.0;
    for (int base = k + tid; base < n; base += U1 * HT) {
      double2 a[U1];
      if (base == k + tid) {
#pragma unroll
        for (int u = 0; u < U1; ++u) a[u] = pre[u];
      } else {
#pragma unroll
        for (int u = 0; u < U1; ++u) {
          const int c = base + u * HT;
          a[u] = c < n ? __ldcg(&rowk[c]) : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int c = base + u * HT;
        if (c < n) {
          const double2 x = csub(csub(a[u], cmulc(vpk, wp[c])), cmulc(wpk, vp[c]));
          if (c == k) {
            s_akk = x.x;
          } else {
            const double2 xc = conjg(x);  // column k below the diagonal
            vc[c] = xc;
            if (c >= k + 2) ss += xc.x * xc.x + xc.y * xc.y;
          }
        }
      }
    }
    // block sum of ss; alpha = vc[k+1] is read by every thread between the two
    // barriers, before its writer can rescale it below
    ss = warp_sum(ss);
    __syncthreads();
    if (lane == 0) red[warp] = ss;
    const double2 alpha = vc[k + 1];
    __syncthreads();
    ss = 0.0;
#pragma unroll
    for (int w = 0; w < HW; ++w) ss += red[w];
    double beta;
    double2 tk, sc;
    if (ss == 0.0 && alpha.y == 0.0) {
      tk = make_double2(0.0, 0.0);
      sc = make_double2(0.0, 0.0);
      beta = alpha.x;
    } else {
      beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + ss), alpha.x);
      tk = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      const double2 den = make_double2(alpha.x - beta, alpha.y);
      const double m2 = den.x * den.x + den.y * den.y;
      sc = make_double2(den.x / m2, -den.y / m2);
    }
    if (bid == 0 && tid == 0) {
      d[k] = s_akk;
      e[k] = beta;
      tau[k] = tk;
    }
    // own entries of vc: v_k; reflector k-1 (own entries of vp) into row k-1,
    // which no CTA reads any more
    for (int c = k + tid; c < n; c += HT) {
      if (c > k) vc[c] = (c == k + 1) ? make_double2(1.0, 0.0) : cmul(vc[c], sc);
      if (bid == 0 && k > 0) __stcg(&A[(size_t)(k - 1) * n + c], vp[c]);
    }
    __syncthreads();

    // ---- phase 2: update k-1 on this CTA's trailing rows, y = A v_k
    const int nrow = n - k - 1;
    const int nr_c = nrow > bid ? (nrow - bid + G - 1) / G : 0;
    const int nch = (nrow + HCH - 1) / HCH;
    const int rb = max(1, PARTS / nch);
    double2 pdot = make_double2(0.0, 0.0);
    for (int j0 = 0; j0 < nr_c; j0 += rb) {
      const int jn = min(rb, nr_c - j0);
      const int nit = jn * nch;
      for (int it = warp; it < nit; it += 2 * HW) {
        const int it2 = it + HW;
        const int jl1 = it / nch, ch1 = it - jl1 * nch;
        const int r1 = k + 1 + bid + (j0 + jl1) * G;
        const int cb1 = k + 1 + ch1 * HCH + lane;
        double2* row1 = A + (size_t)r1 * n;
        double2 a1[U2], a2[U2];
#pragma unroll
        for (int u = 0; u < U2; ++u) {
          const int c = cb1 + 32 * u;
          a1[u] = c < n ? __ldcg(&row1[c]) : make_double2(0.0, 0.0);
        }
        int jl2 = 0, ch2 = 0, r2 = 0, cb2 = 0;
        double2* row2 = row1;
        if (it2 < nit) {
          jl2 = it2 / nch;
          ch2 = it2 - jl2 * nch;
          r2 = k + 1 + bid + (j0 + jl2) * G;
          cb2 = k + 1 + ch2 * HCH + lane;
          row2 = A + (size_t)r2 * n;
#pragma unroll
          for (int u = 0; u < U2; ++u) {
            const int c = cb2 + 32 * u;
            a2[u] = c < n ? __ldcg(&row2[c]) : make_double2(0.0, 0.0);
          }
        }
        double2 acc = hetrd_item(row1, cb1, n, vp[r1], wp[r1], vp, wp, vc, a1);
        acc = warp_sum(acc);
        if (lane == 0) parts[jl1 * nch + ch1] = acc;
        if (it2 < nit) {
          acc = hetrd_item(row2, cb2, n, vp[r2], wp[r2], vp, wp, vc, a2);
          acc = warp_sum(acc);
          if (lane == 0) parts[jl2 * nch + ch2] = acc;
        }
      }
      __syncthreads();
      for (int jl = tid; jl < jn; jl += HT) {
        double2 y = make_double2(0.0, 0.0);
        for (int ch = 0; ch < nch; ++ch) y = cadd(y, parts[jl * nch + ch]);
        const int r = k + 1 + bid + (j0 + jl) * G;
        __stcg(&Y[(size_t)(k & 1) * n + r], y);
        pdot = cadd(pdot, cmulc(vc[r], y));  // v_r conj(y_r)
      }
      __syncthreads();  // parts is refilled by the next row group
    }
    pdot = warp_sum(pdot);
    if (lane == 0) redc[warp] = pdot;
    __syncthreads();
    if (tid == 0) {
      double2 s = make_double2(0.0, 0.0);
      for (int w = 0; w < HW; ++w) s = cadd(s, redc[w]);
      __stcg(&P[(size_t)(k & 1) * G + bid], s);
    }
    if (!grid_sync(sync, (unsigned)G, gen, &s_ok, tab.wait_ns, pi == 0 && bid == 0 && k == tab.skip_column)) return;

    // ---- phase 3 (every CTA): w_k = tau y - (|tau|^2 / 2)(y^H v) v; every
    // warp sums the CTA partials itself.  The loads of y, of the partials, of
    // y_{k+1} and of row k+1 (phase 1 of the next column) go out together.
    const bool next = k + 2 < n;
    const double2* rown = A + (size_t)(k + 1) * n;
    double2 yv[U1];
#pragma unroll
    for (int u = 0; u < U1; ++u) {
      const int c = k + 1 + tid + u * HT;
      yv[u] = c < n ? __ldcg(&Y[(size_t)(k & 1) * n + c]) : make_double2(0.0, 0.0);
      pre[u] = (next && c < n) ? __ldcg(&rown[c]) : make_double2(0.0, 0.0);
    }
    const double2 yk1 = __ldcg(&Y[(size_t)(k & 1) * n + k + 1]);
    double2 dot = make_double2(0.0, 0.0);
    for (int base = lane; base < G; base += 32 * U1) {
      double2 pp[U1];
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int b = base + 32 * u;
        pp[u] = b < G ? __ldcg(&P[(size_t)(k & 1) * G + b]) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) dot = cadd(dot, pp[u]);
    }
    dot = warp_sum(dot);
    const double t2 = tk.x * tk.x + tk.y * tk.y;
    const double2 alph = make_double2(-0.5 * t2 * dot.x, -0.5 * t2 * dot.y);
    for (int base = k + 1 + tid; base < n; base += U1 * HT) {
      double2 y[U1];
      if (base == k + 1 + tid) {
#pragma unroll
        for (int u = 0; u < U1; ++u) y[u] = yv[u];
      } else {
#pragma unroll
        for (int u = 0; u < U1; ++u) {
          const int c = base + u * HT;
          y[u] = c < n ? __ldcg(&Y[(size_t)(k & 1) * n + c]) : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int c = base + u * HT;
        if (c < n) {
          const double2 v = vc[c];
          wp[c] = cadd(cmul(tk, y[u]), cmul(alph, v));
          vp[c] = v;
        }
      }
    }
    tk_prev = tk;
    alph_prev = alph;
    yk_prev = yk1;
  }
  if (bid == 0 && tid == 0) {
    if (n == 1) {
      d[0] = __ldcg(&A[0]).x;
    } else {
      double2 a = __ldcg(&A[(size_t)(n - 1) * n + (n - 1)]);
      a = csub(csub(a, cmulc(vp[n - 1], wp[n - 1])), cmulc(wp[n - 1], vp[n - 1]));
      d[n - 1] = a.x;
      __stcg(&A[(size_t)(n - 2) * n + (n - 1)], vp[n - 1]);
    }
  }
}

// ---------------------------------------------------------------- large matrices (n >= 3072), lower triangle
// The same lagged one-column-at-a-time reduction for large n, reading and
// updating only the lower triangle of A: half the bytes per column, and a
// 3584^2 complex matrix (205 MB in full) then stays in the 126 MB L2 instead
// of streaming from HBM twice per column.  Element (r, c), c < r, adds
// x v_c to y_r and conj(x) v_r to y_c; the diagonal adds x v_r to y_r.
//   phase 1 (every CTA)  "row" k is column k of the lower triangle (strided
//                        loads), update k-1 applied, reflector k;
//   phase 2              the trailing rows dealt round-robin to the CTAs; each
//                        warp owns column chunks of LCH columns (assigned in a
//                        snake order for balance) and walks the CTA's rows
//                        through them, two rows in flight: update k-1 stored,
//                        the row's chunk share of y kept in shared memory and
//                        the column contributions in the lanes' registers;
//                        the CTA writes its partial y (columns, plus its rows'
//                        sums in chunk order) to YP[bid][.];
//   grid barrier;
//   phase 2b             CTA b sums YP[0..G-1][i] for its slice of i (one warp
//                        per entry, lanes over the CTAs, fixed shuffle tree),
//                        writes y and its share of y^H v;
//   grid barrier;
//   phase 3 (every CTA)  w_k as before, with column k+1 loaded for phase 1.
// Every reduction has a fixed order, so the result is the same on every run.
constexpr int LU2 = 4;                 // loads in flight per lane per row of a chunk
constexpr int LCH = 32 * LU2;          // columns per chunk
constexpr int LPARTS = 2048;           // (row, chunk) partial sums per CTA
constexpr int YP_G = 256;              // largest CTA count per matrix (YP rows)
constexpr int LOWER_MIN_N = 3072;      // the lower-triangle kernel runs when the batch's largest n reaches this

// one row of a phase-2 chunk: update k-1 on its lower-triangle entries
// (a: their loaded values), stored back; the row's y share (warp-summed) is
// returned and the column contributions added to col
__device__ __forceinline__ double2 lower_row(double2* __restrict__ A, int r, int cs, int lane, int n,
                                             const double2* vp, const double2* wp, const double2* vc,
                                             const double2 (&a)[LU2], double2 (&col)[LU2]) {
  const double2 vpr = vp[r], wpr = wp[r], vr = vc[r];
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int u = 0; u < LU2; ++u) {
    const int c = cs + lane + 32 * u;
    if (c <= r && c < n) {
      const double2 x = csub(csub(a[u], cmulc(vpr, wp[c])), cmulc(wpr, vp[c]));
      __stcg(&A[(size_t)r * n + c], x);
      acc = cadd(acc, cmul(x, vc[c]));
      if (c < r) col[u] = cadd(col[u], cmul(conjg(x), vr));
    }
  }
  return warp_sum(acc);
}

__global__ void __launch_bounds__(HT, 1) hetrd_lower_kernel(const __grid_constant__ HetrdTable tab) {
  int pi = 0;
  while (pi + 1 < tab.count && (int)blockIdx.x >= tab.p[pi + 1].first) ++pi;
  const HetrdProb& PR = tab.p[pi];
  double2* __restrict__ A = PR.A;
  const int n = PR.n;
  double* __restrict__ d = PR.d;
  double* __restrict__ e = PR.e;
  double2* __restrict__ tau = PR.tau;
  double2* __restrict__ Y = PR.Y;
  double2* __restrict__ P = PR.P;
  double2* __restrict__ YP = PR.YP;
  Sync* sync = PR.sync;
  const int bid = (int)blockIdx.x - PR.first;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* vp = reinterpret_cast<double2*>(smem_raw);  // v of step k-1 (pending update)
  double2* wp = vp + n;                                // w of step k-1
  double2* vc = wp + n;                                // v of step k
  double2* parts = vc + n;                             // LPARTS (row, chunk) partial sums of y
  __shared__ double red[HW];
  __shared__ double2 redc[HW];
  __shared__ double s_akk;
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = PR.nblk;
  unsigned gen = 0;
  for (int i = tid; i < n; i += HT) {
    vp[i] = make_double2(0.0, 0.0);
    wp[i] = make_double2(0.0, 0.0);
    vc[i] = make_double2(0.0, 0.0);
  }
  // column 0 of the lower triangle, the part phase 1 reads in its first pass
  double2 pre[U1];
#pragma unroll
  for (int u = 0; u < U1; ++u) {
    const int c = tid + u * HT;
    pre[u] = c < n ? conjg(__ldcg(&A[(size_t)c * n])) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  double2 tk_prev = make_double2(0.0, 0.0), alph_prev = make_double2(0.0, 0.0), yk_prev = make_double2(0.0, 0.0);
  for (int k = 0; k < n - 1; ++k) {
    // ---- phase 1 (every CTA): row k = conj(column k) with update k-1, reflector k
    double2 vpk = make_double2(0.0, 0.0), wpk = make_double2(0.0, 0.0);
    if (k > 0) {
      vpk = make_double2(1.0, 0.0);
      wpk = cadd(cmul(tk_prev, yk_prev), cmul(alph_prev, vpk));
    }
    double ss = 0.0;
    for (int base = k + tid; base < n; base += U1 * HT) {
      double2 a[U1];
      if (base == k + tid) {
#pragma unroll
        for (int u = 0; u < U1; ++u) a[u] = pre[u];
      } else {
#pragma unroll
        for (int u = 0; u < U1; ++u) {
          const int c = base + u * HT;
          a[u] = c < n ? conjg(__ldcg(&A[(size_t)c * n + k])) : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int c = base + u * HT;
        if (c < n) {
          const double2 x = csub(csub(a[u], cmulc(vpk, wp[c])), cmulc(wpk, vp[c]));
          if (c == k) {
            s_akk = x.x;
          } else {
            const double2 xc = conjg(x);
            vc[c] = xc;
            if (c >= k + 2) ss += xc.x * xc.x + xc.y * xc.y;
          }
        }
      }
    }
    ss = warp_sum(ss);
    __syncthreads();
    if (lane == 0) red[warp] = ss;
    const double2 alpha = vc[k + 1];
    __syncthreads();
    ss = 0.0;
#pragma unroll
    for (int w = 0; w < HW; ++w) ss += red[w];
    double beta;
    double2 tk, sc;
    if (ss == 0.0 && alpha.y == 0.0) {
      tk = make_double2(0.0, 0.0);
      sc = make_double2(0.0, 0.0);
      beta = alpha.x;
    } else {
      beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + ss), alpha.x);
      tk = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      const double2 den = make_double2(alpha.x - beta, alpha.y);
      const double m2 = den.x * den.x + den.y * den.y;
      sc = make_double2(den.x / m2, -den.y / m2);
    }
    if (bid == 0 && tid == 0) {
      d[k] = s_akk;
      e[k] = beta;
      tau[k] = tk;
    }
    // own entries of vc: v_k; reflector k-1 into row k-1 (upper triangle, which
    // this kernel never reads)
    for (int c = k + tid; c < n; c += HT) {
      if (c > k) vc[c] = (c == k + 1) ? make_double2(1.0, 0.0) : cmul(vc[c], sc);
      if (bid == 0 && k > 0) __stcg(&A[(size_t)(k - 1) * n + c], vp[c]);
    }
    __syncthreads();

    // ---- phase 2: update k-1 on the lower triangle of this CTA's rows; partial y
    const int nrow = n - k - 1;
    const int nr_c = nrow > bid ? (nrow - bid + G - 1) / G : 0;
    const int nch = (nrow + LCH - 1) / LCH;
    double2* yp = YP + (size_t)bid * n;
    // chunk ch of warp w: ch = w + 2 HW t or 2 HW - 1 - w + 2 HW t
    for (int t = 0; 2 * HW * t + warp < nch; ++t) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int ch = q == 0 ? 2 * HW * t + warp : 2 * HW * t + 2 * HW - 1 - warp;
        if (ch >= nch) continue;
        const int cs = k + 1 + ch * LCH;
        double2 col[LU2];
#pragma unroll
        for (int u = 0; u < LU2; ++u) col[u] = make_double2(0.0, 0.0);
        // first own row reaching this chunk: r_j >= cs
        const int j0 = cs - (k + 1 + bid) > 0 ? (cs - (k + 1 + bid) + G - 1) / G : 0;
        for (int j = j0; j < nr_c; j += 2) {
          const int r1 = k + 1 + bid + j * G;
          const bool two = j + 1 < nr_c;
          const int r2 = two ? r1 + G : r1;
          double2 a1[LU2], a2[LU2];
#pragma unroll
          for (int u = 0; u < LU2; ++u) {
            const int c = cs + lane + 32 * u;
            a1[u] = (c <= r1 && c < n) ? __ldcg(&A[(size_t)r1 * n + c]) : make_double2(0.0, 0.0);
            a2[u] = (two && c <= r2 && c < n) ? __ldcg(&A[(size_t)r2 * n + c]) : make_double2(0.0, 0.0);
          }
          double2 acc = lower_row(A, r1, cs, lane, n, vp, wp, vc, a1, col);
          if (lane == 0) parts[j * nch + ch] = acc;
          if (two) {
            acc = lower_row(A, r2, cs, lane, n, vp, wp, vc, a2, col);
            if (lane == 0) parts[(j + 1) * nch + ch] = acc;
          }
        }
#pragma unroll
        for (int u = 0; u < LU2; ++u) {
          const int c = cs + lane + 32 * u;
          if (c < n) __stcg(&yp[c], col[u]);
        }
      }
    }
    __syncthreads();
    // this CTA's rows: add their sums over the chunks they reach, in chunk order
    for (int j = tid; j < nr_c; j += HT) {
      const int r = k + 1 + bid + j * G;
      const int chmax = (r - k - 1) / LCH;
      double2 s = __ldcg(&yp[r]);
      double2 rs = make_double2(0.0, 0.0);
      for (int ch = 0; ch <= chmax; ++ch) rs = cadd(rs, parts[j * nch + ch]);
      __stcg(&yp[r], cadd(s, rs));
    }
    if (!grid_sync(sync, (unsigned)G, gen, &s_ok, tab.wait_ns, pi == 0 && bid == 0 && k == tab.skip_column)) return;

    // ---- phase 2b: y_i = sum over the CTAs' partials, one warp per entry of this CTA's slice
    const int sl = (nrow + G - 1) / G;
    const int i0 = k + 1 + bid * sl, i1 = min(n, i0 + sl);
    double2 pdot = make_double2(0.0, 0.0);
    for (int i = i0 + warp; i < i1; i += HW) {
      // G <= YP_G = 8 x 32: every lane's partials are loaded before any is summed
      double2 part[YP_G / 32];
#pragma unroll
      for (int u = 0; u < YP_G / 32; ++u) {
        const int b = lane + 32 * u;
        part[u] = b < G ? __ldcg(&YP[(size_t)b * n + i]) : make_double2(0.0, 0.0);
      }
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < YP_G / 32; ++u) acc = cadd(acc, part[u]);
      acc = warp_sum(acc);
      if (lane == 0) {
        __stcg(&Y[(size_t)(k & 1) * n + i], acc);
        pdot = cadd(pdot, cmulc(vc[i], acc));
      }
    }
    if (lane == 0) redc[warp] = pdot;
    __syncthreads();
    if (tid == 0) {
      double2 sum = make_double2(0.0, 0.0);
      for (int w = 0; w < HW; ++w) sum = cadd(sum, redc[w]);
      __stcg(&P[(size_t)(k & 1) * G + bid], sum);
    }
    if (!grid_sync(sync, (unsigned)G, gen, &s_ok, tab.wait_ns, false)) return;

    // ---- phase 3 (every CTA): w_k; column k+1 loaded for the next phase 1
    const bool next = k + 2 < n;
    double2 yv[U1];
#pragma unroll
    for (int u = 0; u < U1; ++u) {
      const int c = k + 1 + tid + u * HT;
      yv[u] = c < n ? __ldcg(&Y[(size_t)(k & 1) * n + c]) : make_double2(0.0, 0.0);
      pre[u] = (next && c < n) ? conjg(__ldcg(&A[(size_t)c * n + k + 1])) : make_double2(0.0, 0.0);
    }
    const double2 yk1 = __ldcg(&Y[(size_t)(k & 1) * n + k + 1]);
    double2 dot = make_double2(0.0, 0.0);
    for (int base = lane; base < G; base += 32 * U1) {
      double2 pp[U1];
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int b = base + 32 * u;
        pp[u] = b < G ? __ldcg(&P[(size_t)(k & 1) * G + b]) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) dot = cadd(dot, pp[u]);
    }
    dot = warp_sum(dot);
    const double t2 = tk.x * tk.x + tk.y * tk.y;
    const double2 alph = make_double2(-0.5 * t2 * dot.x, -0.5 * t2 * dot.y);
    for (int base = k + 1 + tid; base < n; base += U1 * HT) {
      double2 y[U1];
      if (base == k + 1 + tid) {
#pragma unroll
        for (int u = 0; u < U1; ++u) y[u] = yv[u];
      } else {
#pragma unroll
        for (int u = 0; u < U1; ++u) {
          const int c = base + u * HT;
          y[u] = c < n ? __ldcg(&Y[(size_t)(k & 1) * n + c]) : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < U1; ++u) {
        const int c = base + u * HT;
        if (c < n) {
          const double2 v = vc[c];
          wp[c] = cadd(cmul(tk, y[u]), cmul(alph, v));
          vp[c] = v;
        }
      }
    }
    tk_prev = tk;
    alph_prev = alph;
    yk_prev = yk1;
  }
  if (bid == 0 && tid == 0) {
    if (n == 1) {
      d[0] = __ldcg(&A[0]).x;
    } else {
      double2 a = __ldcg(&A[(size_t)(n - 1) * n + (n - 1)]);
      a = csub(csub(a, cmulc(vp[n - 1], wp[n - 1])), cmulc(wp[n - 1], vp[n - 1]));
      d[n - 1] = a.x;
      __stcg(&A[(size_t)(n - 2) * n + (n - 1)], vp[n - 1]);
    }
  }
}

// ---------------------------------------------------------------- small matrices
// The same lagged reduction on one thread-block cluster of CL CTAs whose
// shared memories hold the matrix (row r in CTA r % CL, slot r / CL): 8 CTAs up
// to n = 256 (one each for many small matrices, see cluster_of), 16 up to
// NMAX_C16 = 424 (27 rows beside the vectors fill the shared memory) where the
// device can place such a cluster.  Thread c owns entry c of v_k and w_k in
// every CTA and keeps it in registers.  Per column:
//   1  row k (loaded from its owner through distributed shared memory while
//      phase 3 of the column before still ran), update k-1 applied, the norm of
//      its tail; a CTA barrier
//   2  the owned rows: update k-1 and (row . unscaled reflector, entry k+1),
//      pushed to every CTA (double-buffered by column parity, so a CTA that runs
//      ahead never overwrites a buffer another is still reading); 3, 2 or 1
//      rows per warp at a time share the loads of w, v and the reflector.  The
//      last warp computes tau, beta and the reflector's scale meanwhile.  Then
//      the hardware cluster barrier, which every CTA executes the same number
//      of times
//   3  y_k and v_k scaled, y^H v (a CTA barrier), w_k
// Bound by that chain of latencies (2 us a column at n = 32), with the rows' traffic in
// shared memory beside it from n = 200 on: 58 / 274 / 727 us at n = 32 / 128 /
// 256 on 8 CTAs, 942 / 1703 at 300 / 424 on 16 (which a first form found slower than
// 8 up to 256: 997 against 916); with a barrier
// for each of the scalars, the reflector and w_k, and one row per warp at a time,
// n = 240 took 821 us (623 now), and the grid 2830 for n = 416.
// Reflector k is written to row k of Aout (which may alias Gin: all of Gin is
// read before the first barrier).  blockIdx.y = matrix.
constexpr int CT = 512, CW = CT / 32, NMAX_C1 = 64, NMAX_C8 = 256, NMAX_C16 = 424;

inline size_t cluster_smem_bytes(int n, int cl) {
  return ((size_t)ceil_div(n, cl) * n + 7 * (size_t)n) * sizeof(double2);
}

// update k-1 of the CTA's rows from slot s0 on and their sums with the
// reflector, RB rows per warp at a time, by all warps but the last
template <int CL, int RB>
__device__ __forceinline__ void cluster_rows(cg::cluster_group& cluster, int rank, int n, int k, int s0, int act,
                                             double2* rows, const double2* vp, const double2* wp, const double2* vc,
                                             double2* ya, double2* yf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int g = warp * RB; g < act; g += (CW - 1) * RB) {
    double2* row[RB];
    double2 vpr[RB], wpr[RB], acc[RB], first[RB];
#pragma unroll
    for (int u = 0; u < RB; ++u) {
      const int sl = s0 + min(g + u, act - 1);  // past the end: the last row again, not written
      row[u] = rows + (size_t)sl * n;
      vpr[u] = vp[sl * CL + rank];
      wpr[u] = wp[sl * CL + rank];
      acc[u] = first[u] = make_double2(0.0, 0.0);
    }
    for (int c = k + 1 + lane; c < n; c += 32) {
      const double2 w = wp[c], v = vp[c], q = vc[c];
#pragma unroll
      for (int u = 0; u < RB; ++u) {
        const double2 x = csub(csub(row[u][c], cmulc(vpr[u], w)), cmulc(wpr[u], v));
        if (g + u < act) row[u][c] = x;
        if (c == k + 1) first[u] = x;  // the reflector is 1 there
        else acc[u] = cadd(acc[u], cmul(x, q));
      }
    }
#pragma unroll
    for (int u = 0; u < RB; ++u) {
      if (g + u >= act) break;
      const int r = (s0 + g + u) * CL + rank;
      const double2 f = make_double2(__shfl_sync(0xffffffffu, first[u].x, 0), __shfl_sync(0xffffffffu, first[u].y, 0));
      const double2 y = warp_sum(acc[u]);
      if (lane < CL) {
        cluster.map_shared_rank(ya, lane)[r] = y;
        cluster.map_shared_rank(yf, lane)[r] = f;
      }
    }
  }
}

// sum of CW values in shared memory, pairwise: four dependent additions
template <typename T, int N>
__device__ __forceinline__ T tree_sum(const T* x) {
  T t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) t[i] = x[i];
#pragma unroll
  for (int h = N / 2; h > 0; h /= 2)
#pragma unroll
    for (int i = 0; i < h; ++i) t[i] = cadd(t[i], t[i + h]);
  return t[0];
}

template <int CL>
__global__ void __launch_bounds__(CT, 1) hetrd_cluster_kernel(const __grid_constant__ EigTable tab) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const EigProb& PR = tab.p[blockIdx.y];
  const double2* Gin = PR.a;
  double2* Aout = PR.a;
  const int n = PR.n;
  const int nslots = (n - rank + CL - 1) / CL;  // rows this CTA holds
  double* __restrict__ d = PR.d;
  double* __restrict__ e = PR.e;
  double2* __restrict__ tau = PR.tau;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* vp = reinterpret_cast<double2*>(smem_raw);
  double2* wp = vp + n;
  double2* vc = wp + n;
  double2* yb = vc + n;        // 2 x (row . reflector, entry k+1) x n
  double2* rows = yb + 4 * n;  // slots x n
  __shared__ __align__(16) double red[CW];
  __shared__ double2 redc[CW];
  __shared__ double2 s_sc, s_tk;
  __shared__ double s_akk;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = tid;  // n <= 424 < CT
  for (int sl = 0; sl < nslots; ++sl)
    if (c < n) rows[(size_t)sl * n + c] = Gin[(size_t)(sl * CL + rank) * n + c];
  if (c < n) vp[c] = wp[c] = make_double2(0.0, 0.0);
  cluster.sync();
  const double2 zero = make_double2(0.0, 0.0), one = make_double2(1.0, 0.0);
  double2 v_c = zero, w_c = zero, vpk = zero, wpk = zero;  // entries c and k of v_{k-1}, w_{k-1}
  double2 nx = c < n ? cluster.map_shared_rank(rows, 0)[c] : zero;  // row k
  for (int k = 0; k < n - 1; ++k) {
    // ---- phase 1
    double ss = 0.0;
    double2 xc = zero;
    if (c >= k && c < n) {
      const double2 x = csub(csub(nx, cmulc(vpk, w_c)), cmulc(wpk, v_c));
      if (c == k) {
        s_akk = x.x;
      } else {
        xc = conjg(x);
        vc[c] = xc;
        if (c >= k + 2) ss = xc.x * xc.x + xc.y * xc.y;
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();  // vc, red, and v_{k-1}, w_{k-1} of phase 3
    // ---- phase 2
    double2* ya = yb + (size_t)(k & 1) * 2 * n;
    double2* yf = ya + n;
    const int s0 = (k + CL - rank) / CL;  // the first owned row >= k + 1
    const int act = nslots - s0;
    if (warp == CW - 1) {
      const double2 part = tree_sum<double2, CW / 2>(reinterpret_cast<const double2*>(red));
      ss = part.x + part.y;
      const double2 alpha = vc[k + 1];
      double2 sc = zero, tk = zero;
      double beta = alpha.x;
      if (ss != 0.0 || alpha.y != 0.0) {
        beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + ss), alpha.x);
        const double2 den = make_double2(alpha.x - beta, alpha.y);
        // one division for both: even lanes take 1 / beta, odd ones 1 / |alpha - beta|^2
        const double r = 1.0 / ((lane & 1) ? den.x * den.x + den.y * den.y : beta);
        const double rb = __shfl_sync(0xffffffffu, r, 0), rm = __shfl_sync(0xffffffffu, r, 1);
        tk = make_double2((beta - alpha.x) * rb, -alpha.y * rb);
        sc = make_double2(den.x * rm, -den.y * rm);
      }
      if (lane == 0) {
        s_sc = sc;
        s_tk = tk;
        if (rank == 0) {
          d[k] = s_akk;
          e[k] = beta;
          tau[k] = tk;
        }
      }
    } else if (act > 2 * (CW - 1)) {
      cluster_rows<CL, 3>(cluster, rank, n, k, s0, act, rows, vp, wp, vc, ya, yf);
    } else if (act > CW - 1) {
      cluster_rows<CL, 2>(cluster, rank, n, k, s0, act, rows, vp, wp, vc, ya, yf);
    } else {
      cluster_rows<CL, 1>(cluster, rank, n, k, s0, act, rows, vp, wp, vc, ya, yf);
    }
    cluster.sync();
    // ---- phase 3: w_k = tau y - (|tau|^2 / 2)(y^H v) v
    double2 pdot = zero, y = zero;
    const double2 sc = s_sc, tk = s_tk;
    if (c > k && c < n) {
      nx = cluster.map_shared_rank(rows + (size_t)((k + 1) / CL) * n, (k + 1) % CL)[c];
      y = cadd(cmul(ya[c], sc), yf[c]);
      v_c = c == k + 1 ? one : cmul(xc, sc);
      pdot = cmulc(v_c, y);
    }
    const double2 yk1 = cadd(cmul(ya[k + 1], sc), yf[k + 1]);
    pdot = warp_sum(pdot);
    if (lane == 0) redc[warp] = pdot;
    __syncthreads();
    const double2 dot = tree_sum<double2, CW>(redc);
    const double t2 = tk.x * tk.x + tk.y * tk.y;
    const double2 alph = make_double2(-0.5 * t2 * dot.x, -0.5 * t2 * dot.y);
    if (c > k && c < n) {
      w_c = cadd(cmul(tk, y), cmul(alph, v_c));
      vp[c] = v_c;
      wp[c] = w_c;
      if (rank == 0) Aout[(size_t)k * n + c] = v_c;
    }
    vpk = one;
    wpk = cadd(cmul(tk, yk1), alph);
  }
  if (rank == 0 && c == n - 1) d[n - 1] = csub(csub(nx, cmulc(v_c, w_c)), cmulc(w_c, v_c)).x;
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// ---------------------------------------------------------------- eigenvalues
// Sign changes of the leading principal minors p_i of T - x I = eigenvalues of T
// below x (Givens 1953): p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}.  The recurrence
// has one fused multiply-add on its chain, the pivot form q_i = d_i - x - e^2 / q
// a division.  T comes scaled by a power of two to norm <= 1, and e^2 is at least
// E2MIN = 2^-236 (eigenvalues move by 2^-117 of the norm at most).  A step takes
// the larger of two neighbouring minors up by at most 3 and down by at most E2MIN / 4:
// a smaller p_i leaves p_{i+1} above E2MIN / 2 of p_{i-1}.  Four steps from a pair
// scaled to [1, 2) therefore stay in FP64's range.  A minor that is exactly 0
// counts once whatever its sign, as the one after it has the opposite sign of the one before.
constexpr int SCH = 4;  // steps between rescalings; the arrays are padded to a multiple
constexpr double E2MIN = 0x1p-236;
__device__ __forceinline__ int sturm_count(const double2* t, int n, double x) {
  double p0 = 1.0, p1 = t[0].x - x;  // t[i] = (d_i, e_{i-1}^2)
  int cnt = __double2hiint(p1) < 0;
  for (int i0 = 1; i0 < n; i0 += SCH) {
    double2 c[SCH];
#pragma unroll
    for (int u = 0; u < SCH; ++u) c[u] = t[i0 + u];
    const int m = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
    const double f = __hiloint2double((2046 << 20) - m, 0);  // 2^-exponent of the larger
    p0 *= f;
    p1 *= f;
#pragma unroll
    for (int u = 0; u < SCH; ++u) {
      const double p2 = fma(c[u].x - x, p1, -c[u].y * p0);
      if (i0 + u < n) cnt += (uint32_t)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
      p0 = p1;
      p1 = p2;
    }
  }
  return cnt;
}

// The same count from the pivots, for x so near 0 that E2MIN would show: e as
// it is (s = 2^-exponent of T's norm), LAPACK dstebz's guard |q| >= pivmin.
__device__ __forceinline__ int sturm_count_pivots(const double2* t, const double* e, int ex, int n, double x) {
  double q = t[0].x - x;
  if (fabs(q) < DBL_MIN) q = -DBL_MIN;
  int cnt = q < 0.0;
  for (int i = 1; i < n; ++i) {
    const double s = ldexp(e[i - 1], -ex);
    q = (t[i].x - x) - s * s / q;
    if (fabs(q) < DBL_MIN) q = -DBL_MIN;
    cnt += q < 0.0;
  }
  return cnt;
}

// Gershgorin bounds and pivmin of T into out[0..2] (one block)
__global__ void __launch_bounds__(THREADS) bounds_kernel(const __grid_constant__ EigTable tab) {
  const EigProb& PR = tab.p[blockIdx.y];
  const double* __restrict__ d = PR.d;
  const double* __restrict__ e = PR.e;
  const int n = PR.n;
  double* __restrict__ out = PR.bnd;
  __shared__ double rmin[WARPS], rmax[WARPS], re2[WARPS];
  double lo = DBL_MAX, hi = -DBL_MAX, m2 = 0.0;
  for (int i = threadIdx.x; i < n; i += THREADS) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    if (i < n - 1) m2 = fmax(m2, e[i] * e[i]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    rmin[warp] = lo;
    rmax[warp] = hi;
    re2[warp] = m2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < WARPS; ++w) {
      lo = fmin(lo, rmin[w]);
      hi = fmax(hi, rmax[w]);
      m2 = fmax(m2, re2[w]);
    }
    lo = fmin(lo, rmin[0]);
    hi = fmax(hi, rmax[0]);
    m2 = fmax(m2, re2[0]);
    const double tn = fmax(fabs(lo), fabs(hi));
    const double pivmin = DBL_MIN * fmax(1.0, m2);
    out[0] = lo - 2.0 * DBL_EPSILON * tn - 2.0 * pivmin;
    out[1] = hi + 2.0 * DBL_EPSILON * tn + 2.0 * pivmin;
    out[2] = pivmin;
  }
}

// the binary exponent that brings the Gershgorin interval into [-1, 1]
__device__ __forceinline__ int norm_exponent(const double* bnd) {
  const double tn = fmax(fabs(bnd[0]), fabs(bnd[1]));
  int ex = 0;
  frexp(tn, &ex);
  return tn > 0.0 && isfinite(tn) ? ex : 0;
}

// eigenvalue i0 + j (ascending) of T for j < cnt, one warp each: the bracket is
// cut into 33 parts per round, down to 2 ulp of the eigenvalue.  Those below
// 2^-60 of the norm (blocks of exact zeros, graded diagonals) take their last
// rounds with the pivot form.  Bound by the latency of the minors' chain (one
// warp per scheduler where the matrices are small): the top half of an n = 240
// spectrum whose last values lie at 2^-53 of the norm (21 rounds) takes 79 us, 415
// with a division on the chain; 37 with rounds only down to 2^-64 of the norm.
constexpr int BW = 4, BT = 32 * BW;
__global__ void __launch_bounds__(BT) bisect_kernel(const __grid_constant__ EigTable tab) {
  const EigProb& PR = tab.p[blockIdx.y];
  const double* __restrict__ d = PR.d;
  const double* __restrict__ e = PR.e;
  const int n = PR.n, i0 = PR.n - PR.kt, cnt = PR.kt;
  if (blockIdx.x * BW >= cnt) return;
  const double* __restrict__ bnd = PR.bnd;
  double* __restrict__ w = PR.w;
  extern __shared__ double sh[];
  double2* t = reinterpret_cast<double2*>(sh);
  const int ex = norm_exponent(bnd);
  for (int i = threadIdx.x; i < n + SCH; i += BT) {
    double2 c = make_double2(0.0, 0.0);
    if (i < n) {
      c.x = ldexp(d[i], -ex);
      if (i > 0) {
        const double s = ldexp(e[i - 1], -ex);
        c.y = fmax(s * s, E2MIN);
      }
    }
    t[i] = c;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * BW + (threadIdx.x >> 5);
  if (j >= cnt) return;
  const int idx = i0 + j;
  double lo = ldexp(bnd[0], -ex), hi = ldexp(bnd[1], -ex);
  bool pivots = false;
  for (int round = 0; round < 40; ++round) {
    const double ulps = 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi));
    if (hi - lo <= ulps + (pivots ? DBL_MIN : 0x1p-112)) {
      if (pivots || ulps >= 0x1p-111) break;
      pivots = true;  // the bracket holds the eigenvalue to 2^-117
      lo -= 0x1p-114;
      hi += 0x1p-114;
    }
    const double x = lo + (hi - lo) * ((double)(lane + 1) / 33.0);
    const int c = pivots ? sturm_count_pivots(t, e, ex, n, x) : sturm_count(t, n, x);
    // count(x) > idx  <=>  eigenvalue idx < x
    const unsigned above = __ballot_sync(0xffffffffu, c > idx);
    const int first = above ? __ffs(above) - 1 : 32;
    const double xl = __shfl_sync(0xffffffffu, x, first > 0 ? first - 1 : 0);
    const double xh = __shfl_sync(0xffffffffu, x, first < 32 ? first : 31);
    const double nlo = first == 0 ? lo : xl;
    const double nhi = first == 32 ? hi : xh;
    if (nlo == lo && nhi == hi) break;
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) w[j] = ldexp(0.5 * (lo + hi), ex);
}

// ---------------------------------------------------------------- eigenvectors
__device__ __forceinline__ double hash_unit(uint32_t a, uint32_t b) {
  uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return (double)h * (2.0 / 4294967296.0) - 1.0;
}

// The three recurrences of a vector, in fixed operations, so that both kernels
// below round alike: which of them a matrix gets depends on what else is in the
// call, and its vectors must not.
//
// Row k of the LU factors of T - lambda I with partial pivoting.  The current
// row has entries (ak, ck) at columns (k, k+1), the next original row (bk, ak1,
// ck1) at (k, k+1, k+2); U's row is 1 / inv, p1, p2, and ml the multiplier (+4
// when the two were swapped, |multiplier| <= 1 either way).  A pivot below tiny becomes tiny.
struct IvRow {
  double inv, p1, p2, ml;
};
__device__ __forceinline__ IvRow iv_eliminate(double& ak, double& ck, double bk, double ak1, double ck1, double tiny) {
  const bool swap = fabs(ak) < fabs(bk);
  IvRow r;
  r.p1 = swap ? ak1 : ck;
  r.p2 = swap ? ck1 : 0.0;
  const double q = swap ? ak : bk, q1 = swap ? ck : ak1, q2 = swap ? 0.0 : ck1;
  double p = swap ? bk : ak;
  if (fabs(p) < tiny) p = copysign(tiny, p);
  r.inv = 1.0 / p;
  const double m = __dmul_rn(q, r.inv);
  r.ml = swap ? m + 4.0 : m;
  ak = __fma_rn(-m, r.p1, q1);
  ck = __fma_rn(-m, r.p2, q2);
  return r;
}
// the last pivot's reciprocal
__device__ __forceinline__ double iv_last(double ak, double tiny) {
  return 1.0 / (fabs(ak) < tiny ? copysign(tiny, ak) : ak);
}
// L^-1 at row k: returns entry k, zk moves on to k+1, whose entry is zn
__device__ __forceinline__ double iv_forward(double ml, double zn, double& zk) {
  const bool swap = ml > 2.0;
  const double m = swap ? ml - 4.0 : ml;
  const double out = swap ? zn : zk;
  zk = __fma_rn(-m, out, swap ? zk : zn);
  return out;
}
// U^-1 at row k, entries k+1 and k+2 in z1 and z2; adds to the squared norm
__device__ __forceinline__ double iv_backward(double z, double p1, double p2, double inv, double& z1, double& z2,
                                              double& nrm) {
  const double v = __dmul_rn(__fma_rn(-p1, z1, __fma_rn(-p2, z2, z)), inv);
  z2 = z1;
  z1 = v;
  nrm = __fma_rn(v, v, nrm);
  return v;
}

constexpr int IV_THREADS = 128, CH = 8, IV_WAVES = 4;

// The same iteration with every array of a vector in shared memory, V vectors
// (lanes) per warp-sized CTA: a pass over n rows then costs the chains of its
// arithmetic, not trips to L2 (each row 0.3 us against 1.2).  Laid out [row][lane],
// so the lanes never share a bank.  1 / |z| is applied by the next pass.
// 95 us for the top half of n = 240 where the form below takes 240.
constexpr int IV_SMEM = 227 * 1024;
inline size_t inviter_smem_bytes(int n, int V) { return ((size_t)2 * n + 5 * (size_t)n * V) * sizeof(double); }

__global__ void __launch_bounds__(32) inviter_smem_kernel(const __grid_constant__ EigTable tab, int V) {
  const EigProb& PR = tab.p[blockIdx.y];
  const double* __restrict__ d = PR.d;
  const double* __restrict__ e = PR.e;
  const int n = PR.n, cnt = PR.kt;
  const int lane = threadIdx.x, j = blockIdx.x * V + lane;
  if (blockIdx.x * V >= cnt) return;
  extern __shared__ double sh_iv[];
  double* sd = sh_iv;
  double* se = sd + n;
  const int ex = norm_exponent(PR.bnd);  // T and lambda scaled to norm <= 1: the vectors' squares stay finite
  for (int i = lane; i < n; i += 32) {
    sd[i] = ldexp(d[i], -ex);
    se[i] = i < n - 1 ? ldexp(e[i], -ex) : 0.0;
  }
  __syncwarp();
  if (lane >= V || j >= cnt) return;
  const size_t step = (size_t)n * V;
  double* ua = se + n + lane;  // 1 / u_kk
  double* uc = ua + step;      // u_{k,k+1}
  double* uc2 = uc + step;     // u_{k,k+2}
  double* ml = uc2 + step;     // multiplier (+4 when rows k, k+1 were swapped)
  double* z = ml + step;
  const double lam = ldexp(PR.w[j], -ex);
  const double tn = ldexp(fmax(fabs(PR.bnd[0]), fabs(PR.bnd[1])), -ex);
  const double tiny = DBL_EPSILON * fmax(tn, DBL_MIN);
  double ak = sd[0] - lam;
  double ck = se[0];
  for (int k = 0; k < n - 1; ++k) {
    const IvRow r = iv_eliminate(ak, ck, se[k], sd[k + 1] - lam, se[k + 1], tiny);
    ua[k * V] = r.inv;
    uc[k * V] = r.p1;
    uc2[k * V] = r.p2;
    ml[k * V] = r.ml;
  }
  ua[(n - 1) * V] = iv_last(ak, tiny);
  uc[(n - 1) * V] = 0.0;
  uc2[(n - 1) * V] = 0.0;
  for (int i = 0; i < n; ++i) z[i * V] = hash_unit((uint32_t)j + 1u, (uint32_t)i);
  double inv = 1.0;
  for (int it = 0; it < 3; ++it) {
    // forward: L^-1 with the row swaps
    double zk = __dmul_rn(z[0], inv);
    for (int k0 = 0; k0 < n - 1; k0 += CH) {
      double mm[CH], zn[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = min(k0 + u, n - 2);
        mm[u] = ml[k * V];
        zn[u] = __dmul_rn(z[(k + 1) * V], inv);
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        if (k0 + u < n - 1) z[(k0 + u) * V] = iv_forward(mm[u], zn[u], zk);
      }
    }
    z[(n - 1) * V] = zk;
    // backward: U with two super-diagonals
    double z1 = 0.0, z2 = 0.0, nrm = 0.0;
    for (int k0 = n - 1; k0 >= 0; k0 -= CH) {
      double zz[CH], c1[CH], c2[CH], ia[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = max(k0 - u, 0);
        zz[u] = z[k * V];
        c1[u] = uc[k * V];
        c2[u] = uc2[k * V];
        ia[u] = ua[k * V];
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        if (k0 - u >= 0) z[(k0 - u) * V] = iv_backward(zz[u], c1[u], c2[u], ia[u], z1, z2, nrm);
      }
    }
    inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
  }
  for (int i = 0; i < n; ++i) PR.z[(size_t)i * cnt + j] = z[i * V] * inv;
}

// column j of Z (n x cnt row-major) = eigenvector of T for w[j], for tables whose
// vectors would take more than IV_WAVES turns of the shared-memory form; scratch:
// 4 * n * cnt doubles laid out [i * cnt + j] (coalesced across threads).
// d, e are staged in shared memory; every sequential loop loads the next CH
// steps' independent inputs before running their dependent chain.
__global__ void __launch_bounds__(IV_THREADS) inviter_kernel(const __grid_constant__ EigTable tab) {
  const EigProb& PR = tab.p[blockIdx.y];
  const double* __restrict__ d = PR.d;
  const double* __restrict__ e = PR.e;
  const int n = PR.n, cnt = PR.kt;
  const double* __restrict__ w = PR.w;
  const double* __restrict__ bnd = PR.bnd;
  double* __restrict__ Z = PR.z;
  double* __restrict__ scr = PR.scr;
  extern __shared__ double sh_de[];
  double* sd = sh_de;
  double* se = sh_de + n;
  const int ex = norm_exponent(bnd);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    sd[i] = ldexp(d[i], -ex);
    se[i] = i < n - 1 ? ldexp(e[i], -ex) : 0.0;
  }
  __syncthreads();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cnt) return;
  const size_t S = (size_t)cnt;
  double* ua = scr;                       // 1 / u_kk
  double* uc = scr + 1 * (size_t)n * S;   // u_{k,k+1}
  double* uc2 = scr + 2 * (size_t)n * S;  // u_{k,k+2}
  double* ml = scr + 3 * (size_t)n * S;   // multiplier (+4 when rows k, k+1 were swapped)
  const double lam = ldexp(w[j], -ex);
  const double tn = ldexp(fmax(fabs(bnd[0]), fabs(bnd[1])), -ex);
  const double tiny = DBL_EPSILON * fmax(tn, DBL_MIN);
  double ak = sd[0] - lam;
  double ck = se[0];
  for (int k = 0; k < n - 1; ++k) {
    const IvRow r = iv_eliminate(ak, ck, se[k], sd[k + 1] - lam, se[k + 1], tiny);
    ua[(size_t)k * S + j] = r.inv;
    uc[(size_t)k * S + j] = r.p1;
    uc2[(size_t)k * S + j] = r.p2;
    ml[(size_t)k * S + j] = r.ml;
  }
  ua[(size_t)(n - 1) * S + j] = iv_last(ak, tiny);
  uc[(size_t)(n - 1) * S + j] = 0.0;
  uc2[(size_t)(n - 1) * S + j] = 0.0;
  double* z = Z;
#pragma unroll 8
  for (int i = 0; i < n; ++i) z[(size_t)i * S + j] = hash_unit((uint32_t)j + 1u, (uint32_t)i);
  for (int it = 0; it < 3; ++it) {
    // forward: L^-1 with the row swaps
    double zk = z[j];
    for (int k0 = 0; k0 < n - 1; k0 += CH) {
      double mm[CH], zn[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = k0 + u;
        mm[u] = k < n - 1 ? ml[(size_t)k * S + j] : 0.0;
        zn[u] = k < n - 1 ? z[(size_t)(k + 1) * S + j] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = k0 + u;
        if (k < n - 1) z[(size_t)k * S + j] = iv_forward(mm[u], zn[u], zk);
      }
    }
    z[(size_t)(n - 1) * S + j] = zk;
    // backward: U with two super-diagonals
    double z1 = 0.0, z2 = 0.0, nrm = 0.0;
    for (int k0 = n - 1; k0 >= 0; k0 -= CH) {
      double zz[CH], c1[CH], c2[CH], ia[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = k0 - u;
        const bool ok = k >= 0;
        zz[u] = ok ? z[(size_t)k * S + j] : 0.0;
        c1[u] = ok ? uc[(size_t)k * S + j] : 0.0;
        c2[u] = ok ? uc2[(size_t)k * S + j] : 0.0;
        ia[u] = ok ? ua[(size_t)k * S + j] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int k = k0 - u;
        if (k >= 0) z[(size_t)k * S + j] = iv_backward(zz[u], c1[u], c2[u], ia[u], z1, z2, nrm);
      }
    }
    const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
#pragma unroll 8
    for (int i = 0; i < n; ++i) z[(size_t)i * S + j] *= inv;
  }
}

// ---------------------------------------------------------------- back-transformation
// K = Q K with Q = H_0 ... H_{n-2} in blocks of NB reflectors (compact WY:
// H_k0 ... H_k0+kb-1 = I - V T V^H, LAPACK's forward columnwise larft), the
// blocks applied from the last to the first, each as three FP64 GEMMs.
constexpr int NB = 64;

// rows 0..n-2 of A become the reflectors (0 before column k+1, 1 at k+1) and
// row n-1 becomes 0, so that every reflector row can be read over all n columns
__global__ void clean_v_kernel(double2* __restrict__ A, int n) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)n * n) return;
  const int k = (int)(idx / n), c = (int)(idx % n);
  if (k == n - 1 || c <= k) A[idx] = make_double2(0.0, 0.0);
  else if (c == k + 1) A[idx] = make_double2(1.0, 0.0);
}

// minus the NB x NB upper-triangular T of block b from S = V^H V and tau, by
// doubling: two neighbouring factors T1, T2 of h reflectors join into
// [[T1, -T1 S12 T2], [0, T2]], for h = 1, 2, .. NB / 2, all pairs of a level at once in
// shared memory.  12 barriers in the place of the 128 of a column-by-column form,
// whose row sums also ran one after the other.  22 us a call; the
// column form took 105 per matrix.
constexpr int LT = 256;
constexpr int LARFT_SMEM = (2 * NB * NB + NB * NB / 4) * (int)sizeof(double2);
struct LarftProb {
  const double2* S;
  const double2* tau;
  double2* T;
  int n, first;  // first block of the grid
};
struct LarftTable {
  int count = 0, blocks = 0;
  LarftProb p[MAXM];
  void add(const double2* S, const double2* tau, double2* T, int n) {
    p[count++] = LarftProb{S, tau, T, n, blocks};
    blocks += (int)ceil_div(n - 1, NB);
  }
};
__global__ void __launch_bounds__(LT) larft_kernel(const __grid_constant__ LarftTable tab) {
  int pi = 0;
  while (pi + 1 < tab.count && (int)blockIdx.x >= tab.p[pi + 1].first) ++pi;
  const double2* __restrict__ Sg = tab.p[pi].S;
  const double2* __restrict__ tau = tab.p[pi].tau;
  double2* __restrict__ Tg = tab.p[pi].T;
  const int n = tab.p[pi].n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* S = reinterpret_cast<double2*>(smem_raw);
  double2* T = S + NB * NB;
  double2* W = T + NB * NB;  // S12 T2 of every pair of a level: 32 h <= NB^2 / 4 entries
  const int b = blockIdx.x - tab.p[pi].first, k0 = b * NB, kb = min(NB, n - 1 - k0);
  for (int i = threadIdx.x; i < NB * NB; i += LT) {
    const int r = i / NB, c = i % NB;
    S[i] = Sg[(size_t)b * NB * NB + i];
    T[i] = r == c && r < kb ? tau[k0 + r] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  for (int h = 1; h < NB; h *= 2) {
    const int total = NB / 2 * h;
    for (int i = threadIdx.x; i < total; i += LT) {
      const int c = i % h, r = i / h % h, o = i / (h * h) * 2 * h;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int l = 0; l <= c; ++l) acc = cadd(acc, cmul(S[(o + r) * NB + o + h + l], T[(o + h + l) * NB + o + h + c]));
      W[i] = acc;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < total; i += LT) {
      const int c = i % h, r = i / h % h, o = i / (h * h) * 2 * h, w0 = i / (h * h) * h * h + c;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int l = r; l < h; ++l) acc = cadd(acc, cmul(T[(o + r) * NB + o + l], W[w0 + l * h]));
      T[(o + r) * NB + o + h + c] = make_double2(-acc.x, -acc.y);
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < NB * NB; i += LT) Tg[(size_t)b * NB * NB + i] = make_double2(-T[i].x, -T[i].y);
}

}  // namespace heev
}  // namespace reno

using namespace reno;
using namespace reno::heev;

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

namespace {
struct HeevLayout {
  size_t sync, y, p, yp, bnd, scr, s, t, w1, w2, total;
};
HeevLayout heev_layout(int n, int kt) {
  HeevLayout L{};
  const size_t nblk = (size_t)ceil_div(std::max(n - 1, 1), NB);
  size_t off = 0;
  L.sync = off;
  off += align256(sizeof(Sync));
  L.y = off;
  off += align256(2 * (size_t)n * sizeof(double2));
  L.p = off;
  off += align256(2 * 1024 * sizeof(double2));
  L.yp = off;  // partial sums of the lower-triangle reduction (grid path only)
  off += n > NMAX_C8 ? align256((size_t)YP_G * n * sizeof(double2)) : 0;
  L.bnd = off;
  off += align256(4 * sizeof(double));
  L.scr = off;
  off += align256(4 * (size_t)n * kt * sizeof(double));
  L.s = off;
  off += align256(nblk * NB * NB * sizeof(double2));
  L.t = off;
  off += align256(nblk * NB * NB * sizeof(double2));
  L.w1 = off;
  off += align256((size_t)NB * kt * sizeof(double2));
  L.w2 = off;
  off += align256((size_t)NB * kt * sizeof(double2));
  L.total = off;
  return L;
}

GemmOperand op(const void* p, int64_t s_outer, int64_t s_k, int conj) {
  GemmOperand o;
  o.ptr = p;
  o.s_outer = s_outer;
  o.s_k = s_k;
  o.is_complex = 1;
  o.conj = conj;
  return o;
}
}  // namespace

// Cooperative launch of the reduction over the matrices of tab (too large for a cluster):
// one CTA per SM, the SMs shared out in proportion to each matrix's n^2.  When
// the largest matrix has at least LOWER_MIN_N rows the lower-triangle kernel
// runs (each matrix then needs enough CTAs that its rows' (row, chunk)
// partials fit LPARTS, and at most YP_G); otherwise the full-row kernel.
static int launch_hetrd(reno_ctx* ctx, HetrdTable& tab, int nmax, const char* what) {
  static std::atomic<unsigned long long> hetrd_set{0}, lower_set{0};
  int rc = check_cuda(ctx, smem_optin_once(hetrd_kernel, (3 * MAX_N + PARTS) * 16, hetrd_set),
                      (std::string(what) + ": hetrd smem attribute").c_str());
  if (rc == RENO_OK)
    rc = check_cuda(ctx, smem_optin_once(hetrd_lower_kernel, (3 * MAX_N + LPARTS) * 16, lower_set),
                    (std::string(what) + ": hetrd smem attribute").c_str());
  if (rc != RENO_OK) return rc;
  const int G = std::min(sm_count_current_device(), 1024);
  if (tab.count > G) return set_error(ctx, RENO_ERR_INVALID, std::string(what) + ": more matrices than SMs");
  // CTAs a matrix needs under the lower-triangle kernel
  auto gmin_lower = [](int n) {
    const int nch = (int)ceil_div(n - 1, LCH);
    const int rows = std::max(1, LPARTS / std::max(nch, 1));
    return (int)ceil_div(n - 1, rows);
  };
  // RENO_HETRD_LOWER_MIN overrides the size from which the lower-triangle kernel runs
  static const int lower_min = [] {
    const char* e = std::getenv("RENO_HETRD_LOWER_MIN");
    return (e && std::atoi(e) > 0) ? std::atoi(e) : LOWER_MIN_N;
  }();
  bool lower = nmax >= lower_min;
  int need = 0;
  for (int i = 0; i < tab.count; ++i) {
    if (!tab.p[i].YP) lower = false;
    need += gmin_lower(tab.p[i].n);
  }
  if (need > G) lower = false;
  void* kfn = lower ? (void*)hetrd_lower_kernel : (void*)hetrd_kernel;
  const size_t smem = (3 * (size_t)nmax + (lower ? LPARTS : PARTS)) * sizeof(double2);
  int per_sm = 0;
  rc = check_cuda(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, HT, smem),
                  (std::string(what) + ": occupancy").c_str());
  if (rc != RENO_OK) return rc;
  if (per_sm < 1) return set_error(ctx, RENO_ERR_INVALID, std::string(what) + ": hetrd kernel does not fit on an SM");
  double work = 0.0;
  for (int i = 0; i < tab.count; ++i) work += (double)tab.p[i].n * tab.p[i].n;
  int used = 0, reserved = 0;
  if (lower)
    for (int i = 0; i < tab.count; ++i) reserved += gmin_lower(tab.p[i].n);
  for (int i = 0; i < tab.count; ++i) {
    const int left = tab.count - 1 - i;  // at least one CTA for every later matrix
    const int floor_i = lower ? gmin_lower(tab.p[i].n) : 1;
    if (lower) reserved -= floor_i;
    const int later = lower ? reserved : left;
    int nb = i == tab.count - 1 ? G - used
                                : (int)std::lround(G * (double)tab.p[i].n * tab.p[i].n / std::max(work, 1.0));
    nb = std::max(floor_i, std::min(nb, G - used - later));
    if (lower) nb = std::min(nb, YP_G);
    tab.p[i].first = used;
    tab.p[i].nblk = nb;
    used += nb;
  }
  tab.wait_ns = g_wait_ns.load(std::memory_order_relaxed);
  tab.skip_column = g_skip_hetrd_column.exchange(-1);
  void* args[] = {&tab};
  count_launch();
  return check_cuda(ctx, cudaLaunchCooperativeKernel(kfn, dim3(used), dim3(HT), args, smem, ctx->stream),
                    (std::string(what) + ": hetrd launch").c_str());
}

extern "C" int reno_heev_workspace_bytes(int32_t n, int32_t kt, size_t* bytes) {
  if (!bytes || n < 1 || n > MAX_N || kt < 1 || kt > n) return RENO_ERR_INVALID;
  *bytes = heev_layout(n, kt).total;
  return RENO_OK;
}

namespace {

int heev_attrs(reno_ctx* ctx) {
  static std::atomic<unsigned long long> bisect_set{0}, inviter_set{0}, iv_smem_set{0}, larft_set{0}, c8_set{0},
      c16_set{0}, c1_set{0}, wide_set{0};
  const char* what = "reno_heev_top: shared memory attributes";
  cudaError_t rc = smem_optin_once(bisect_kernel, 2 * (MAX_N + SCH) * (int)sizeof(double), bisect_set);
  if (rc == cudaSuccess) rc = smem_optin_once(inviter_kernel, 2 * MAX_N * (int)sizeof(double), inviter_set);
  if (rc == cudaSuccess) rc = smem_optin_once(inviter_smem_kernel, IV_SMEM, iv_smem_set);
  if (rc == cudaSuccess) rc = smem_optin_once(larft_kernel, LARFT_SMEM, larft_set);
  if (rc == cudaSuccess) rc = smem_optin_once(hetrd_cluster_kernel<1>, (int)cluster_smem_bytes(NMAX_C1, 1), c1_set);
  if (rc == cudaSuccess) rc = smem_optin_once(hetrd_cluster_kernel<8>, (int)cluster_smem_bytes(NMAX_C8, 8), c8_set);
  if (rc == cudaSuccess) rc = smem_optin_once(hetrd_cluster_kernel<16>, (int)cluster_smem_bytes(NMAX_C16, 16), c16_set);
  if (rc == cudaSuccess) {
    int dev = 0;
    rc = cudaGetDevice(&dev);
    const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
    if (rc == cudaSuccess && !(bit && (wide_set.load(std::memory_order_acquire) & bit))) {
      rc = cudaFuncSetAttribute(hetrd_cluster_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (rc == cudaSuccess && bit) wide_set.fetch_or(bit, std::memory_order_release);
    }
  }
  return check_cuda(ctx, rc, what);
}

int launch_larft(reno_ctx* ctx, const LarftTable& tab) {
  const int rc = heev_attrs(ctx);
  if (rc != RENO_OK) return rc;
  count_launch();
  larft_kernel<<<tab.blocks, LT, LARFT_SMEM, ctx->stream>>>(tab);
  RENO_LAUNCH_CHECK(ctx, "reno_heev_backtransform: larft");
  return RENO_OK;
}

cudaLaunchConfig_t cluster_config(int cl, int count, int n, cudaStream_t st, cudaLaunchAttribute* at) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)cl;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cl, (unsigned)count);
  cfg.blockDim = dim3(CT);
  cfg.dynamicSmemBytes = cluster_smem_bytes(n, cl);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// 16-CTA clusters of the largest matrix that the current device can hold at
// once (read once per device; 0 where it has no room for even one)
int wide_clusters() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int c = known[dev].load(std::memory_order_acquire);
  if (c == 0) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(16, 1, NMAX_C16, nullptr, &at);
    int num = 0;
    if (cudaOccupancyMaxActiveClusters(&num, hetrd_cluster_kernel<16>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      num = 0;
    }
    c = num + 1;
    known[dev].store(c, std::memory_order_release);
  }
  return c - 1;
}

// tridiagonal reduction of matrices that fit a cluster: one cluster per
// matrix, all of one cluster size in one launch
int heev_reduce_small(reno_ctx* ctx, const EigTable& tab, int cl) {
  if (tab.count == 0) return RENO_OK;
  int nmax = 1;
  for (int i = 0; i < tab.count; ++i) nmax = std::max(nmax, tab.p[i].n);
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = cluster_config(cl, tab.count, nmax, ctx->stream, &at);
  count_launch();
  return check_cuda(ctx,
                    cl == 16  ? cudaLaunchKernelEx(&cfg, hetrd_cluster_kernel<16>, tab)
                    : cl == 8 ? cudaLaunchKernelEx(&cfg, hetrd_cluster_kernel<8>, tab)
                              : cudaLaunchKernelEx(&cfg, hetrd_cluster_kernel<1>, tab),
                    "reno_heev_top: cluster hetrd");
}

// CTAs of the cluster that reduces an n x n matrix (0: the grid does), for a
// call with `tiny` matrices of at most NMAX_C1 rows.  One matrix is done soonest by
// 8 CTAs (120 us at n = 64, 180 on one); more matrices than 8-CTA clusters fit the GPU
// at once go to single CTAs (24 of n = 64: 180 us against 265, 32 of n = 32: 68
// against 179).  Every sum has the same order on any number of CTAs, so the
// choice does not show in the results.
int cluster_of(int n, int tiny) {
  if (n <= NMAX_C1 && tiny > 16) return 1;
  if (n <= NMAX_C8) return 8;
  return n <= NMAX_C16 && wide_clusters() > 0 ? 16 : 0;
}

// eigenvalues n-kt .. n-1 of every T (ascending) and their inverse-iteration
// vectors: one launch per stage for all matrices of the table
int heev_eig(reno_ctx* ctx, const EigTable& tab) {
  if (tab.count == 0) return RENO_OK;
  int nmax = 1, ktmax = 1;
  for (int i = 0; i < tab.count; ++i) {
    nmax = std::max(nmax, tab.p[i].n);
    ktmax = std::max(ktmax, tab.p[i].kt);
  }
  cudaStream_t st = ctx->stream;
  count_launch();
  bounds_kernel<<<dim3(1, tab.count), THREADS, 0, st>>>(tab);
  RENO_LAUNCH_CHECK(ctx, "reno_heev_top: bounds");
  count_launch();
  bisect_kernel<<<dim3((unsigned)ceil_div(ktmax, BW), tab.count), BT, 2 * (size_t)(nmax + SCH) * sizeof(double),
                  st>>>(tab);
  RENO_LAUNCH_CHECK(ctx, "reno_heev_top: bisect");
  // a turn of the shared-memory form is worth four of the other's (0.3 against 1.2 us a row)
  const int V = (int)std::min<size_t>(32, (IV_SMEM / sizeof(double) - 2 * (size_t)nmax) / (5 * (size_t)nmax));
  const int64_t ctas = ceil_div(ktmax, std::max(V, 1)) * (int64_t)tab.count;
  count_launch();
  if (V >= 1 && ctas <= (int64_t)IV_WAVES * sm_count_current_device())
    inviter_smem_kernel<<<dim3((unsigned)ceil_div(ktmax, V), tab.count), 32, inviter_smem_bytes(nmax, V), st>>>(tab, V);
  else
    inviter_kernel<<<dim3((unsigned)ceil_div(ktmax, IV_THREADS), tab.count), IV_THREADS,
                     2 * (size_t)nmax * sizeof(double), st>>>(tab);
  RENO_LAUNCH_CHECK(ctx, "reno_heev_top: inverse iteration");
  return RENO_OK;
}

bool heev_problem_ok(const reno_heev_problem& p) {
  return p.n >= 1 && p.n <= MAX_N && p.kt >= 1 && p.kt <= p.n && p.a && p.d && p.e && p.tau && p.w && p.z;
}

size_t batched_offset(int32_t count, const reno_heev_problem* probs, int upto) {
  size_t off = 0;
  for (int i = 0; i < upto && i < count; ++i) off += align256(heev_layout(probs[i].n, probs[i].kt).total);
  return off;
}

}  // namespace

// The reflector rows of v are written in place of the upper triangle of A,
// so A must be a private copy of G.
extern "C" int reno_heev_top(reno_ctx* ctx, int32_t n, int32_t kt, void* A, double* d, double* e, void* tau,
                             double* w, double* Z, void* ws, size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (n < 1 || n > MAX_N || kt < 1 || kt > n)
    return set_error(ctx, RENO_ERR_INVALID, "reno_heev_top: need 1 <= kt <= n <= 4096");
  if (!A || !d || !e || !tau || !w || !Z || !ws) return set_error(ctx, RENO_ERR_INVALID, "reno_heev_top: null pointer");
  const HeevLayout L = heev_layout(n, kt);
  if (ws_bytes < L.total) return set_error(ctx, RENO_ERR_WORKSPACE, "reno_heev_top: workspace too small");
  char* base = static_cast<char*>(ws);
  Sync* sync = reinterpret_cast<Sync*>(base + L.sync);
  double2* Y = reinterpret_cast<double2*>(base + L.y);
  double2* P = reinterpret_cast<double2*>(base + L.p);
  double* bnd = reinterpret_cast<double*>(base + L.bnd);
  double* scr = reinterpret_cast<double*>(base + L.scr);
  int rc = check_cuda(ctx, cudaMemsetAsync(sync, 0, sizeof(Sync), ctx->stream), "reno_heev_top: memset");
  if (rc == RENO_OK) rc = heev_attrs(ctx);
  if (rc != RENO_OK) return rc;
  EigTable et{};
  et.count = 1;
  et.p[0] = EigProb{static_cast<double2*>(A), static_cast<double2*>(tau), d, e, n, kt, w, Z, bnd, scr};
  if (const int cl = cluster_of(n, 1)) {
    rc = heev_reduce_small(ctx, et, cl);
  } else {
    HetrdTable tab{};
    tab.count = 1;
    tab.p[0] = HetrdProb{static_cast<double2*>(A), n, d, e, static_cast<double2*>(tau), Y, P, sync, 0, 0,
                         reinterpret_cast<double2*>(base + L.yp)};
    rc = launch_hetrd(ctx, tab, n, "reno_heev_top");
  }
  if (rc != RENO_OK) return rc;
  return heev_eig(ctx, et);
}

extern "C" int reno_heev_batched_workspace_bytes(int32_t count, const reno_heev_problem* probs, size_t* bytes) {
  if (!bytes || !probs || count < 1 || count > RENO_HEEV_MAX_BATCH) return RENO_ERR_INVALID;
  for (int i = 0; i < count; ++i)
    if (probs[i].n < 1 || probs[i].n > MAX_N || probs[i].kt < 1 || probs[i].kt > probs[i].n) return RENO_ERR_INVALID;
  *bytes = batched_offset(count, probs, count);
  return RENO_OK;
}

// reno_heev_top for several matrices: the matrices larger than the cluster
// path share one cooperative reduction launch (the grid split among them),
// so the QN blocks of one bond are reduced side by side.
extern "C" int reno_heev_top_batched(reno_ctx* ctx, int32_t count, const reno_heev_problem* probs, int32_t* status,
                                     void* ws, size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (!probs || !status || !ws || count < 1 || count > RENO_HEEV_MAX_BATCH)
    return set_error(ctx, RENO_ERR_INVALID, "reno_heev_top_batched: invalid batch");
  for (int i = 0; i < count; ++i)
    if (!heev_problem_ok(probs[i]))
      return set_error(ctx, RENO_ERR_INVALID, "reno_heev_top_batched: problem " + std::to_string(i) +
                                                  " needs 1 <= kt <= n <= 4096 and non-null pointers");
  if (ws_bytes < batched_offset(count, probs, count))
    return set_error(ctx, RENO_ERR_WORKSPACE, "reno_heev_top_batched: workspace too small");
  int rc = heev_attrs(ctx);
  if (rc != RENO_OK) return rc;
  HetrdTable tab{};
  EigTable single{}, small{}, wide{}, all{};
  int tiny = 0;
  for (int i = 0; i < count; ++i) tiny += probs[i].n <= NMAX_C1;
  int nmax = 0;
  for (int i = 0; i < count; ++i) {
    const reno_heev_problem& p = probs[i];
    char* base = static_cast<char*>(ws) + batched_offset(count, probs, i);
    const HeevLayout L = heev_layout(p.n, p.kt);
    Sync* sync = reinterpret_cast<Sync*>(base + L.sync);
    rc = check_cuda(ctx, cudaMemsetAsync(sync, 0, sizeof(Sync), ctx->stream), "reno_heev_top_batched: memset");
    if (rc != RENO_OK) return rc;
    const EigProb ep{static_cast<double2*>(p.a), static_cast<double2*>(p.tau), p.d, p.e, p.n, p.kt, p.w, p.z,
                     reinterpret_cast<double*>(base + L.bnd), reinterpret_cast<double*>(base + L.scr)};
    all.p[all.count++] = ep;
    if (const int cl = cluster_of(p.n, tiny)) {
      EigTable& t = cl == 1 ? single : cl == 8 ? small : wide;
      t.p[t.count++] = ep;
    } else {
      tab.p[tab.count++] = HetrdProb{static_cast<double2*>(p.a), p.n, p.d, p.e, static_cast<double2*>(p.tau),
                                     reinterpret_cast<double2*>(base + L.y), reinterpret_cast<double2*>(base + L.p),
                                     sync, 0, 0, reinterpret_cast<double2*>(base + L.yp)};
      nmax = std::max(nmax, (int)p.n);
    }
  }
  rc = heev_reduce_small(ctx, single, 1);
  if (rc == RENO_OK) rc = heev_reduce_small(ctx, small, 8);
  if (rc == RENO_OK) rc = heev_reduce_small(ctx, wide, 16);
  if (rc != RENO_OK) return rc;
  if (tab.count) {
    rc = launch_hetrd(ctx, tab, nmax, "reno_heev_top_batched");
    if (rc != RENO_OK) return rc;
  }
  rc = heev_eig(ctx, all);
  if (rc != RENO_OK) return rc;
  for (int i = 0; i < count; ++i) {
    char* base = static_cast<char*>(ws) + batched_offset(count, probs, i);
    const HeevLayout L = heev_layout(probs[i].n, probs[i].kt);
    rc = check_cuda(ctx, cudaMemcpyAsync(status + i, base + L.sync + offsetof(Sync, status), sizeof(int32_t),
                                         cudaMemcpyDeviceToDevice, ctx->stream),
                    "reno_heev_top_batched: status");
    if (rc != RENO_OK) return rc;
  }
  return RENO_OK;
}

// K (n x kt complex128, in: eigenvectors of T, out: Q K) after reno_heev_top
// on the same A, tau and workspace; A's reflector rows are cleaned in place.
extern "C" int reno_heev_backtransform(reno_ctx* ctx, int32_t n, int32_t kt, void* A, const void* tau, void* K,
                                       void* ws, size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (n < 1 || n > MAX_N || kt < 1 || kt > n || !A || !tau || !K || !ws)
    return set_error(ctx, RENO_ERR_INVALID, "reno_heev_backtransform: invalid arguments");
  const HeevLayout L = heev_layout(n, kt);
  if (ws_bytes < L.total) return set_error(ctx, RENO_ERR_WORKSPACE, "reno_heev_backtransform: workspace too small");
  if (n == 1) return RENO_OK;
  char* base = static_cast<char*>(ws);
  double2* Sg = reinterpret_cast<double2*>(base + L.s);
  double2* Tg = reinterpret_cast<double2*>(base + L.t);
  double2* W1 = reinterpret_cast<double2*>(base + L.w1);
  double2* W2 = reinterpret_cast<double2*>(base + L.w2);
  double2* V = static_cast<double2*>(A);
  double2* Kc = static_cast<double2*>(K);
  cudaStream_t st = ctx->stream;
  const int nblk = (int)ceil_div(n - 1, NB);
  const size_t nel = (size_t)n * n;
  count_launch();
  clean_v_kernel<<<(unsigned)ceil_div((int64_t)nel, 256), 256, 0, st>>>(V, n);
  RENO_LAUNCH_CHECK(ctx, "reno_heev_backtransform: clean");
  int rc = check_cuda(ctx, cudaMemsetAsync(Sg, 0, (size_t)nblk * NB * NB * sizeof(double2), st),
                      "reno_heev_backtransform: memset");
  if (rc != RENO_OK) return rc;
  // S_b = V_b^H V_b: the blocks of NB reflectors in one batched GEMM over all
  // n columns (zeros before each row's reflector), a partial last block apart
  const int nfull = (n - 1) / NB;
  if (nfull > 0) {
    GemmParams p;
    p.M = NB;
    p.N = NB;
    p.K = n;
    p.batch = nfull;
    p.A = op(V, n, 1, 1);
    p.A.s_batch = (int64_t)NB * n;
    p.B = op(V, n, 1, 0);
    p.B.s_batch = (int64_t)NB * n;
    p.C = Sg;
    p.sCm = NB;
    p.sCn = 1;
    p.sCb = (int64_t)NB * NB;
    rc = check_cuda(ctx, gemm_fp64(p, st), "reno_heev_backtransform: gram");
    if (rc != RENO_OK) return rc;
  }
  if (nfull < nblk) {
    const int k0 = nfull * NB, kb = n - 1 - k0;
    GemmParams p;
    p.M = kb;
    p.N = kb;
    p.K = n;
    p.A = op(V + (size_t)k0 * n, n, 1, 1);
    p.B = op(V + (size_t)k0 * n, n, 1, 0);
    p.C = Sg + (size_t)nfull * NB * NB;
    p.sCm = NB;
    p.sCn = 1;
    rc = check_cuda(ctx, gemm_fp64(p, st), "reno_heev_backtransform: gram (last block)");
    if (rc != RENO_OK) return rc;
  }
  LarftTable lt;
  lt.add(Sg, static_cast<const double2*>(tau), Tg, n);
  rc = launch_larft(ctx, lt);
  if (rc != RENO_OK) return rc;
  for (int b = nblk - 1; b >= 0; --b) {
    const int k0 = b * NB, kb = std::min(NB, n - 1 - k0);
    const int rows = n - k0 - 1;
    const double2* Vb = V + (size_t)k0 * n + k0 + 1;
    double2* Kb = Kc + (size_t)(k0 + 1) * kt;
    GemmParams p1;  // W1 = V_b^H K
    p1.M = kb;
    p1.N = kt;
    p1.K = rows;
    p1.A = op(Vb, n, 1, 1);
    p1.B = op(Kb, 1, kt, 0);
    p1.C = W1;
    p1.sCm = kt;
    p1.sCn = 1;
    GemmParams p2;  // W2 = (-T_b) W1
    p2.M = kb;
    p2.N = kt;
    p2.K = kb;
    p2.A = op(Tg + (size_t)b * NB * NB, NB, 1, 0);
    p2.B = op(W1, 1, kt, 0);
    p2.C = W2;
    p2.sCm = kt;
    p2.sCn = 1;
    // K[k0+1:] += V_b W2
    GemmParams p3;
    p3.M = rows;
    p3.N = kt;
    p3.K = kb;
    p3.A = op(Vb, 1, n, 0);
    p3.B = op(W2, 1, kt, 0);
    p3.C = Kb;
    p3.sCm = kt;
    p3.sCn = 1;
    p3.accumulate = 1;
    rc = check_cuda(ctx, gemm_fp64(p1, st), "reno_heev_backtransform: V^H K");
    if (rc == RENO_OK) rc = check_cuda(ctx, gemm_fp64(p2, st), "reno_heev_backtransform: T W");
    if (rc == RENO_OK) rc = check_cuda(ctx, gemm_fp64(p3, st), "reno_heev_backtransform: K += V W");
    if (rc != RENO_OK) return rc;
  }
  return RENO_OK;
}

// status word of the last reno_heev_top on a workspace: the int at this
// byte offset of ws (0 = ok, 1 = a grid barrier timed out)
extern "C" int reno_heev_status_offset(size_t* offset) {
  if (!offset) return RENO_ERR_INVALID;
  *offset = offsetof(Sync, status);
  return RENO_OK;
}

// reno_heev_backtransform for every problem of a reno_heev_top_batched call
// (same problems and workspace): K_i <- Q_i K_i.  The GEMMs of all problems
// run as grouped launches: the Grams of the reflector blocks in one launch,
// then, for the blocks of NB reflectors from the last, one launch each for
// V_b^H K, (-T_b) W1 and K += V_b W2 over every problem that has block b.
extern "C" int reno_heev_backtransform_batched(reno_ctx* ctx, int32_t count, const reno_heev_problem* probs,
                                               void* ws, size_t ws_bytes) {
  if (!ctx) return RENO_ERR_INVALID;
  if (!probs || !ws || count < 1 || count > RENO_HEEV_MAX_BATCH)
    return set_error(ctx, RENO_ERR_INVALID, "reno_heev_backtransform_batched: invalid batch");
  if (ws_bytes < batched_offset(count, probs, count))
    return set_error(ctx, RENO_ERR_WORKSPACE, "reno_heev_backtransform_batched: workspace too small");
  cudaStream_t st = ctx->stream;
  struct One {
    int n, kt, nblk;
    double2 *V, *K, *Sg, *Tg, *W1, *W2;
    const double2* tau;
  };
  std::vector<One> P;
  int rc = RENO_OK;
  static_assert(2 * RENO_HEEV_MAX_BATCH <= fp64gemm::MAX_GROUP, "one block step of a batch fits one group");
  auto flush = [&](fp64gemm::GemmGroup& g, const char* what) -> int {
    if (g.count == 0) return RENO_OK;
    const int r = check_cuda(ctx, gemm_fp64_grouped(g, st), what);
    g.count = 0;
    return r;
  };
  auto add = [&](fp64gemm::GemmGroup& g, const GemmParams& q, const char* what) -> int {
    g.p[g.count++] = q;
    return g.count == fp64gemm::MAX_GROUP ? flush(g, what) : RENO_OK;
  };
  for (int i = 0; i < count; ++i) {
    const reno_heev_problem& p = probs[i];
    if (!p.k || !p.a || !p.tau) return set_error(ctx, RENO_ERR_INVALID, "reno_heev_backtransform_batched: null");
    if (p.n < 2) continue;
    char* base = static_cast<char*>(ws) + batched_offset(count, probs, i);
    const HeevLayout L = heev_layout(p.n, p.kt);
    One o{p.n, p.kt, (int)ceil_div(p.n - 1, NB), static_cast<double2*>(p.a),
          static_cast<double2*>(p.k), reinterpret_cast<double2*>(base + L.s), reinterpret_cast<double2*>(base + L.t),
          reinterpret_cast<double2*>(base + L.w1), reinterpret_cast<double2*>(base + L.w2),
          static_cast<const double2*>(p.tau)};
    count_launch();
    clean_v_kernel<<<(unsigned)ceil_div((int64_t)o.n * o.n, 256), 256, 0, st>>>(o.V, o.n);
    RENO_LAUNCH_CHECK(ctx, "reno_heev_backtransform_batched: clean");
    rc = check_cuda(ctx, cudaMemsetAsync(o.Sg, 0, (size_t)o.nblk * NB * NB * sizeof(double2), st),
                    "reno_heev_backtransform_batched: memset");
    if (rc != RENO_OK) return rc;
    P.push_back(o);
  }
  if (P.empty()) return RENO_OK;
  // S_b = V_b^H V_b of every problem (full blocks batched, the partial last block apart)
  fp64gemm::GemmGroup g1, g2, g3;
  for (const One& o : P) {
    const int nfull = (o.n - 1) / NB;
    if (nfull > 0) {
      GemmParams q;
      q.M = NB;
      q.N = NB;
      q.K = o.n;
      q.batch = nfull;
      q.A = op(o.V, o.n, 1, 1);
      q.A.s_batch = (int64_t)NB * o.n;
      q.B = op(o.V, o.n, 1, 0);
      q.B.s_batch = (int64_t)NB * o.n;
      q.C = o.Sg;
      q.sCm = NB;
      q.sCn = 1;
      q.sCb = (int64_t)NB * NB;
      if ((rc = add(g1, q, "reno_heev_backtransform_batched: gram")) != RENO_OK) return rc;
    }
    if (nfull < o.nblk) {
      const int k0 = nfull * NB, kb = o.n - 1 - k0;
      GemmParams q;
      q.M = kb;
      q.N = kb;
      q.K = o.n;
      q.A = op(o.V + (size_t)k0 * o.n, o.n, 1, 1);
      q.B = op(o.V + (size_t)k0 * o.n, o.n, 1, 0);
      q.C = o.Sg + (size_t)nfull * NB * NB;
      q.sCm = NB;
      q.sCn = 1;
      if ((rc = add(g1, q, "reno_heev_backtransform_batched: gram")) != RENO_OK) return rc;
    }
  }
  if ((rc = flush(g1, "reno_heev_backtransform_batched: gram")) != RENO_OK) return rc;
  int bmax = 0;
  LarftTable lt;
  for (const One& o : P) {
    lt.add(o.Sg, o.tau, o.Tg, o.n);
    bmax = std::max(bmax, o.nblk);
  }
  if ((rc = launch_larft(ctx, lt)) != RENO_OK) return rc;
  // blocks of reflectors from the last: every problem with block b advances together
  for (int b = bmax - 1; b >= 0; --b) {
    for (const One& o : P) {
      if (b >= o.nblk) continue;
      const int k0 = b * NB, kb = std::min(NB, o.n - 1 - k0);
      const int rows = o.n - k0 - 1;
      const double2* Vb = o.V + (size_t)k0 * o.n + k0 + 1;
      double2* Kb = o.K + (size_t)(k0 + 1) * o.kt;
      GemmParams q1;  // W1 = V_b^H K
      q1.M = kb;
      q1.N = o.kt;
      q1.K = rows;
      q1.A = op(Vb, o.n, 1, 1);
      q1.B = op(Kb, 1, o.kt, 0);
      q1.C = o.W1;
      q1.sCm = o.kt;
      q1.sCn = 1;
      if ((rc = add(g1, q1, "reno_heev_backtransform_batched: V^H K")) != RENO_OK) return rc;
      GemmParams q2;  // W2 = (-T_b) W1
      q2.M = kb;
      q2.N = o.kt;
      q2.K = kb;
      q2.A = op(o.Tg + (size_t)b * NB * NB, NB, 1, 0);
      q2.B = op(o.W1, 1, o.kt, 0);
      q2.C = o.W2;
      q2.sCm = o.kt;
      q2.sCn = 1;
      if ((rc = add(g2, q2, "reno_heev_backtransform_batched: T W")) != RENO_OK) return rc;
      GemmParams q3;  // K[k0+1:] += V_b W2
      q3.M = rows;
      q3.N = o.kt;
      q3.K = kb;
      q3.A = op(Vb, 1, o.n, 0);
      q3.B = op(o.W2, 1, o.kt, 0);
      q3.C = Kb;
      q3.sCm = o.kt;
      q3.sCn = 1;
      q3.accumulate = 1;
      if ((rc = add(g3, q3, "reno_heev_backtransform_batched: K += V W")) != RENO_OK) return rc;
    }
    if ((rc = flush(g1, "reno_heev_backtransform_batched: V^H K")) != RENO_OK) return rc;
    if ((rc = flush(g2, "reno_heev_backtransform_batched: T W")) != RENO_OK) return rc;
    if ((rc = flush(g3, "reno_heev_backtransform_batched: K += V W")) != RENO_OK) return rc;
  }
  return RENO_OK;
}
