// The MPO stage of a matvec or environment update (hop_expr.py:68-103,
// lib.py:200-237): T2[b][r][n] = sum_q Wt[r][q] T1[b][q][n] with the
// transposed MPO tensor Wt (real, R x Q, R and Q up to a few hundred) and
// complex or real T1.
//
// As a GEMM this stage costs as much as a sixth of a matvec, on operands that
// are almost all zero: a Holstein phonon site has 126 nonzeros of 80 x 80, a
// spin-boson site 54 of 24 x 24 (finite-state operators: identities,
// diagonals, one off-diagonal band).  What bounds it is then one read of T1
// and one write of T2.  Persistent CTAs list the nonzeros once, in shared
// memory, then stream Q x TN tiles of T1 through two stages of cp.async: lane
// = column, a warp per output row, so that reads of the tile are free of bank
// conflicts and stores are whole 256- or 512-byte segments.
//
// A tensor with more than CAP nonzeros or a quarter of its entries (the list's
// dependent adds are then the slower way), and any tile that holds an infinity
// or NaN (whose product with a zero is a NaN that the list would lose), is
// multiplied in full from the same shared-memory tile by m8n8k4 MMAs.
//
// Measured against the GEMM, us (R x Q x N x batch):
//   complex  80 x 80 x 3888 x 251   1079 -> 476 (5.2 TB/s), all nonzero 1070
//            80 x 64 x 256 x 256      66 -> 41,             all nonzero 71
//            50 x 50 x 640 x 64       29 -> 21,             all nonzero 29
//   real     24 x 24 x 2048 x 256     73 -> 37 (5.4 TB/s),  all nonzero 56
#pragma once
#include "gemm_fp64.cuh"

namespace reno {
namespace mpo {

constexpr int THREADS = 256, WARPS = THREADS / 32;
constexpr int CAP = 1024;      // nonzeros kept as a list
constexpr int RMAX = 1024;     // output rows
constexpr int64_t MIN_ELEMS = 1 << 20;  // of T1, see mpo_stage_applies

template <bool C>
struct Num {
  using T = typename std::conditional<C, double2, double>::type;
};

constexpr int pitch(bool cplx, int tn) { return tn + (cplx ? 2 : 4); }
inline size_t smem_bytes(bool cplx, int cpl, int Q) {
  return (size_t)2 * Q * pitch(cplx, 32 * cpl) * (cplx ? 16 : 8) + CAP * (sizeof(double) + sizeof(int)) +
         (RMAX + 2) * sizeof(int);
}

template <bool C, int CPL>
__global__ void __launch_bounds__(THREADS, 2)
    mpo_stage_kernel(const double* __restrict__ Wt, const typename Num<C>::T* __restrict__ T1,
                     typename Num<C>::T* __restrict__ T2, int R, int Q, int N, int64_t ntiles, int tiles_n, int pairs) {
  using T = typename Num<C>::T;
  constexpr int TN = 32 * CPL, P = pitch(C, TN);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tiles = reinterpret_cast<T*>(smem_raw);  // 2 x Q x P
  double* vals = reinterpret_cast<double*>(tiles + (size_t)2 * Q * P);
  int* cols = reinterpret_cast<int*>(vals + CAP);
  int* rowp = cols + CAP;  // R + 1
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sbase = fp64gemm::smem_u32(tiles);

  auto load = [&](int64_t t, int st) {
    const int64_t b = t / tiles_n;
    const int n0 = (int)(t % tiles_n) * TN;
    const T* src = T1 + b * Q * N + n0;
    const uint32_t dst = sbase + (uint32_t)(st * Q * P * sizeof(T));
    if (!C && pairs) {  // N even and T1 16-byte aligned: two real elements per copy
      for (int i = tid; i < Q * (TN / 2); i += THREADS) {
        const int q = i / (TN / 2), c = 2 * (i % (TN / 2));
        const bool ok = n0 + c < N;
        fp64gemm::cp_async_zfill<16>(dst + (uint32_t)((q * P + c) * sizeof(T)), ok ? src + (int64_t)q * N + c : T1, ok);
      }
    } else {
      for (int i = tid; i < Q * TN; i += THREADS) {
        const int q = i / TN, c = i % TN;
        const bool ok = n0 + c < N;
        fp64gemm::cp_async_zfill<sizeof(T)>(dst + (uint32_t)((q * P + c) * sizeof(T)),
                                            ok ? src + (int64_t)q * N + c : T1, ok);
      }
    }
  };
  int64_t t = blockIdx.x;
  if (t < ntiles) load(t, 0);
  fp64gemm::cp_async_commit();

  // ---- the nonzeros of Wt, row by row: counts, offsets, entries
  for (int r = warp; r < R; r += WARPS) {
    int c = 0;
    for (int q = lane; q - lane < Q; q += 32)
      c += __popc(__ballot_sync(0xffffffffu, q < Q && Wt[(size_t)r * Q + q] != 0.0));
    if (lane == 0) rowp[r + 1] = c;
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int r0 = 0; r0 < R; r0 += 32) {
      int x = r0 + lane < R ? rowp[r0 + lane + 1] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (r0 + lane < R) rowp[r0 + lane + 1] = run + x;
      run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) rowp[0] = 0;
  }
  __syncthreads();
  const bool listed = rowp[R] <= CAP && 4 * rowp[R] <= R * Q;
  if (listed)
    for (int r = warp; r < R; r += WARPS) {
      int at = rowp[r];
      for (int q = lane; q - lane < Q; q += 32) {
        const double w = q < Q ? Wt[(size_t)r * Q + q] : 0.0;
        const unsigned m = __ballot_sync(0xffffffffu, w != 0.0);
        if (w != 0.0) {
          const int k = at + __popc(m & ((1u << lane) - 1u));
          vals[k] = w;
          cols[k] = q;
        }
        at += __popc(m);
      }
    }

  for (int st = 0; t < ntiles; t += gridDim.x, st ^= 1) {
    if (t + gridDim.x < ntiles) load(t + gridDim.x, st ^ 1);
    fp64gemm::cp_async_commit();
    fp64gemm::cp_async_wait<1>();
    __syncthreads();
    const T* s = tiles + (size_t)st * Q * P;
    const int64_t b = t / tiles_n;
    const int n0 = (int)(t % tiles_n) * TN;
    T* out = T2 + b * R * N + n0;
    bool finite = true;
    if (listed) {
      double z = 0.0;
      for (int i = tid; i < Q * TN; i += THREADS) {
        const T x = s[(i / TN) * P + i % TN];
        if constexpr (C) z = fma(x.x, 0.0, fma(x.y, 0.0, z));
        else z = fma(x, 0.0, z);
      }
      finite = z == 0.0;
    }
    if (!__syncthreads_or(!(listed && finite))) {
      for (int r = warp; r < R; r += WARPS) {
        T acc[CPL];
#pragma unroll
        for (int u = 0; u < CPL; ++u) acc[u] = T{};
        for (int k = rowp[r]; k < rowp[r + 1]; ++k) {
          const double w = vals[k];
          const T* row = s + cols[k] * P + lane;
#pragma unroll
          for (int u = 0; u < CPL; ++u) {
            const T x = row[32 * u];
            if constexpr (C) acc[u] = make_double2(fma(w, x.x, acc[u].x), fma(w, x.y, acc[u].y));
            else acc[u] = fma(w, x, acc[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < CPL; ++u)
          if (n0 + lane + 32 * u < N) out[(int64_t)r * N + lane + 32 * u] = acc[u];
      }
    } else {
      const int rb = (R + 7) / 8;
      for (int item = warp; item < rb * CPL; item += WARPS) {  // 8 rows x 32 columns
        const int r = 8 * (item % rb) + (lane >> 2), c0 = 32 * (item / rb);
        {
          double re[4][2], im[4][2];
#pragma unroll
          for (int j = 0; j < 4; ++j) re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
          for (int q0 = 0; q0 < Q; q0 += 4) {
            const int q = q0 + (lane & 3);
            const bool in = q < Q;
            const double a = in && r < R ? Wt[(size_t)r * Q + q] : 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const T x = in ? s[q * P + c0 + 8 * j + (lane >> 2)] : T{};
              if constexpr (C) {
                fp64gemm::dmma(re[j][0], re[j][1], a, x.x);
                fp64gemm::dmma(im[j][0], im[j][1], a, x.y);
              } else {
                fp64gemm::dmma(re[j][0], re[j][1], a, x);
              }
            }
          }
          if (r < R)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int c = c0 + 8 * j + 2 * (lane & 3) + e;
                if (n0 + c < N) {
                  if constexpr (C) out[(int64_t)r * N + c] = make_double2(re[j][e], im[j][e]);
                  else out[(int64_t)r * N + c] = re[j][e];
                }
              }
        }
      }
    }
    __syncthreads();  // the stage is refilled by the next round
  }
  fp64gemm::cp_async_wait<0>();
}

// columns per lane: the widest tile whose two stages leave room for two CTAs per SM (0: none)
inline int columns_per_lane(bool cplx, int Q) {
  for (int cpl = cplx ? 2 : 4; cpl >= 1; cpl /= 2)
    if (smem_bytes(cplx, cpl, Q) <= 112 * 1024) return cpl;
  return 0;
}

template <bool C, int CPL>
inline cudaError_t launch(const double* Wt, const void* T1, void* T2, int R, int Q, int N, int batch, cudaStream_t st) {
  using T = typename Num<C>::T;
  static std::atomic<unsigned long long> set{0};
  cudaError_t e = smem_optin_once(mpo_stage_kernel<C, CPL>, 112 * 1024, set);
  if (e != cudaSuccess) return e;
  const int tiles_n = (int)ceil_div(N, 32 * CPL);
  const int64_t ntiles = (int64_t)tiles_n * batch;
  const unsigned grid = (unsigned)std::min<int64_t>(ntiles, 2 * sm_count_current_device());
  const int pairs = !C && N % 2 == 0 && reinterpret_cast<uintptr_t>(T1) % 16 == 0;
  count_launch();
  mpo_stage_kernel<C, CPL><<<grid, THREADS, smem_bytes(C, CPL, Q), st>>>(
      Wt, static_cast<const T*>(T1), static_cast<T*>(T2), R, Q, N, ntiles, tiles_n, pairs);
  return cudaGetLastError();
}

}  // namespace mpo

// Whether p (A = Wt: real, row-major; B = T1[b]: [q][n] with unit n stride;
// C = T2[b]: [r][n], all dense) is an MPO stage that the kernel above takes.
// Below a million elements of T1 both are near a launch's own time (0.2 M
// elements: 7.9 us as a GEMM, 8.5 here; 0.8 M: 14.6 and 12.6, all nonzero
// 14.6); the tile has to fit shared memory.
inline bool mpo_stage_applies(const GemmParams& p) {
  return !p.A.is_complex && !p.A.conj && !p.B.conj && p.A.s_batch == 0 && p.A.s_k == 1 && p.A.s_outer == p.K &&
         p.B.s_outer == 1 && p.B.s_k == p.N && p.B.s_batch == (int64_t)p.K * p.N && p.sCm == p.N && p.sCn == 1 &&
         p.sCb == (int64_t)p.M * p.N && !p.accumulate && !p.A.is_f32 && !p.B.is_f32 && !p.c_f32 && p.M <= mpo::RMAX &&
         (int64_t)p.K * p.N * p.batch >= mpo::MIN_ELEMS && mpo::columns_per_lane(p.B.is_complex, p.K) > 0;
}

inline cudaError_t mpo_stage(const GemmParams& p, cudaStream_t st) {
  const double* W = static_cast<const double*>(p.A.ptr);
  const int cpl = mpo::columns_per_lane(p.B.is_complex, p.K);
  if (p.B.is_complex)
    return cpl == 2 ? mpo::launch<true, 2>(W, p.B.ptr, p.C, p.M, p.K, p.N, p.batch, st)
                    : mpo::launch<true, 1>(W, p.B.ptr, p.C, p.M, p.K, p.N, p.batch, st);
  return cpl == 4   ? mpo::launch<false, 4>(W, p.B.ptr, p.C, p.M, p.K, p.N, p.batch, st)
         : cpl == 2 ? mpo::launch<false, 2>(W, p.B.ptr, p.C, p.M, p.K, p.N, p.batch, st)
                    : mpo::launch<false, 1>(W, p.B.ptr, p.C, p.M, p.K, p.N, p.batch, st);
}

}  // namespace reno
