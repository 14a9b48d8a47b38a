// Strided batched FP64 GEMM on the sm_100a double-precision MMA pipe
// (mma.sync m8n8k4 .f64), complex handled as four real products.
//
//   C[b][m][n] (+)= sum_k opA(A)[b][m][k] * opB(B)[b][k][n]
//
// Every stage of the H_eff matvec and of the environment update is one call
// of this kernel with the strides of the reference's C-order tensors, so no
// operand is ever permuted in HBM (hop_expr.py:57-103, lib.py:200-237).
//
// What bounds it: the FP64 pipe (one m8n8k4 per 16 clocks and sub-partition,
// 36.7 TFLOP/s over the chip; plain DFMA shares the same pipe) for large
// products, and the length of one CTA's own chain for the small ones, whose
// tiles leave most SMs idle.  Hence three tiles and an optional split of K:
//   64 x 64  4 warps of 32 x 32, two stages of 16 K values in shared memory
//            (82 KB complex), so that two CTAs share an SM and one's loads
//            and barriers hide behind the other's MMAs;
//   32 x 32  4 warps of 16 x 16;
//   16 x 16  4 warps that each take every fourth k4 step of the whole tile
//            and sum their accumulators in shared memory: a quarter of the
//            chain of the same tile on one warp;
//   split-K  a cluster of S = 2, 4 or 8 CTAs takes one tile, each an S-th of
//            K; partial tiles are summed in rank order through distributed
//            shared memory (deterministic, no workspace, no second launch).
// gemm_choose() picks by estimated time; its choice depends on the problem
// alone, so a grouped launch rounds each problem as its own launch does.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <cooperative_groups.h>
#include "reno_common.cuh"

namespace reno {

struct GemmOperand {
  const void* ptr = nullptr;
  int64_t s_outer = 0;  // stride of the M (A) or N (B) index, in elements
  int64_t s_k = 0;      // stride of the K index
  int64_t s_batch = 0;
  int is_complex = 0;
  int conj = 0;
  int is_f32 = 0;       // elements are float / float2 (split-precision intermediates only)
};

struct GemmParams {
  int M = 0, N = 0, K = 0, batch = 1;
  GemmOperand A, B;
  void* C = nullptr;
  int64_t sCm = 0, sCn = 0, sCb = 0;
  int accumulate = 0;
  int c_f32 = 0;        // C is float / float2 (split-precision intermediates only)
};

namespace fp64gemm {

constexpr int BK = 16, BKP = BK + 4, THREADS = 128;
enum Tile { T64 = 0, T32 = 1, T16 = 2 };
constexpr int tile_dim(int t) { return t == T64 ? 64 : t == T32 ? 32 : 16; }
// stages of the shared-memory ring; f = real products per element product
// (4 complex x complex, 2 mixed, 1 real).  The small tiles hold too few MMAs
// per chunk to cover an L2 round trip with one chunk in flight: 16 x 16 with
// four stages takes 0.26 us a chunk against 0.35 with two, real 32 x 32 with
// three 228 us against 245 (16384 x 256 x 768).
constexpr int tile_stages(int t, int f) { return t == T64 ? 2 : t == T32 ? (f == 1 ? 3 : 2) : 4; }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void* src, bool valid) {
  const int src_bytes = valid ? BYTES : 0;
  if constexpr (BYTES == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// The copies of one operand's BT x BK tiles by this thread.  The thread ->
// element map follows whichever global index is unit-stride, so that global
// reads coalesce, and the shared-memory tile is laid out the same way:
// [outer][k] with pitch BK + 4, or [k][outer] with pitch BT + 2 (complex) /
// BT + 4 (real); either way the 8 x 4 fragment reads are free of bank
// conflicts, and so are the writes.
template <bool CPLX, int BT>
struct TileLoader {
  using T = typename std::conditional<CPLX, double2, double>::type;
  static constexpr int ELEMS = BT * BK / THREADS;
  static constexpr int OP = BT + (CPLX ? 2 : 4);  // [k][outer] pitch
  static constexpr int TILE = BT * BKP > BK * OP ? BT * BKP : BK * OP;
  const T* src;        // the thread's first element of the current chunk
  const T* safe;       // a readable address for the zero-filled copies
  int64_t step;        // global distance between the thread's elements
  int64_t chunk;       // global distance between chunks
  uint32_t dst, dstep; // shared-memory byte offset of the first element, distance
  int k, kstep;        // first k of the thread, distance in k between its elements
  unsigned omask;      // elements whose outer index is in range
  int so, sk;          // fragment strides in the shared tile (elements)

  __device__ __forceinline__ void init(const GemmOperand& op, const T* base, int outer0, int outer_max, int k0,
                                       int tid) {
    const bool k_fast = op.s_k == 1;
    int o, ostep;
    if (k_fast) {
      k = tid % BK;
      o = tid / BK;
      ostep = THREADS / BK;
      kstep = 0;
      so = BKP;
      sk = 1;
    } else {
      constexpr int KS = THREADS / BT > 0 ? THREADS / BT : 1;
      o = tid % BT;
      k = tid / BT;
      ostep = 0;
      kstep = KS;
      so = 1;
      sk = OP;
    }
    safe = base;
    src = base + (int64_t)(outer0 + o) * op.s_outer + (int64_t)(k0 + k) * op.s_k;
    step = (int64_t)ostep * op.s_outer + (int64_t)kstep * op.s_k;
    chunk = (int64_t)BK * op.s_k;
    dst = (uint32_t)((o * so + k * sk) * sizeof(T));
    dstep = (uint32_t)((ostep * so + kstep * sk) * sizeof(T));
    omask = 0;
#pragma unroll
    for (int i = 0; i < ELEMS; ++i) omask |= (outer0 + o + i * ostep < outer_max) ? (1u << i) : 0u;
  }

  // the next chunk into the shared tile at byte address `tile`; krem = K values left in range
  __device__ __forceinline__ void load(uint32_t tile, int krem) {
    const T* p = src;
    uint32_t d = tile + dst;
#pragma unroll
    for (int i = 0; i < ELEMS; ++i) {
      const bool valid = ((omask >> i) & 1u) && (k + i * kstep < krem);
      cp_async_zfill<sizeof(T)>(d, valid ? p : safe, valid);
      p += step;
      d += dstep;
    }
    src += chunk;
  }
};

template <bool AC, bool BC, int TILE>
constexpr int stage_bytes() {
  return TileLoader<AC, tile_dim(TILE)>::TILE * (AC ? 16 : 8) + TileLoader<BC, tile_dim(TILE)>::TILE * (BC ? 16 : 8);
}
// the stages; afterwards partial tiles (16 x 16: of the four warps) live in the same memory
template <bool AC, bool BC, int TILE>
constexpr int smem_bytes() {
  const int bt = tile_dim(TILE), part = bt * bt * ((AC || BC) ? 16 : 8) * (TILE == T16 ? 4 : 1);
  const int st = tile_stages(TILE, (AC ? 2 : 1) * (BC ? 2 : 1)) * stage_bytes<AC, BC, TILE>();
  return st > part ? st : part;
}

// one output tile (tile column bx, tile row by, batch entry bz) of p; with
// S > 1 this CTA (rank r of its cluster) sums an S-th of K and a share of the
// tile's partials
template <bool AC, bool BC, int TILE>
__device__ __forceinline__ void gemm_tile(const GemmParams& p, int bx, int by, int bz, int S, int rank) {
  constexpr int BT = tile_dim(TILE);
  constexpr int KW = TILE == T16 ? 4 : 1;      // warps sharing the tile's K range
  constexpr int WT = TILE == T16 ? 16 : BT / 2;  // warp tile
  constexpr int F = WT / 8;
  constexpr int ST = tile_stages(TILE, (AC ? 2 : 1) * (BC ? 2 : 1));
  constexpr bool CC = AC || BC;
  using TA = typename std::conditional<AC, double2, double>::type;
  using TB = typename std::conditional<BC, double2, double>::type;
  using TC = typename std::conditional<CC, double2, double>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int A_BYTES = TileLoader<AC, BT>::TILE * sizeof(TA);
  constexpr int ST_BYTES = stage_bytes<AC, BC, TILE>();

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm0 = KW == 1 ? (warp & 1) * WT : 0, wn0 = KW == 1 ? (warp >> 1) * WT : 0;
  const int m0 = by * BT, n0 = bx * BT;
  const int64_t b = bz;
  const int kc = S == 1 ? p.K : (int)(ceil_div(ceil_div(p.K, S), BK) * BK);
  const int k0 = min(p.K, rank * kc), k1 = min(p.K, k0 + kc);
  const int nk = (k1 - k0 + BK - 1) / BK;
  TileLoader<AC, BT> la;
  TileLoader<BC, BT> lb;
  la.init(p.A, reinterpret_cast<const TA*>(p.A.ptr) + b * p.A.s_batch, m0, p.M, k0, tid);
  lb.init(p.B, reinterpret_cast<const TB*>(p.B.ptr) + b * p.B.s_batch, n0, p.N, k0, tid);
  const uint32_t sbase = smem_u32(smem_raw);

  double accr[F][F][2], acci[F][F][2];
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) {
      accr[i][j][0] = accr[i][j][1] = 0.0;
      acci[i][j][0] = acci[i][j][1] = 0.0;
    }
#pragma unroll
  for (int q = 0; q < ST - 1; ++q) {
    if (q < nk) {
      la.load(sbase + q * ST_BYTES, k1 - k0 - q * BK);
      lb.load(sbase + q * ST_BYTES + A_BYTES, k1 - k0 - q * BK);
    }
    cp_async_commit();
  }

  const double sgnA = p.A.conj ? -1.0 : 1.0, sgnB = p.B.conj ? -1.0 : 1.0;
  const int fa = (wm0 + (lane >> 2)) * la.so + (lane & 3) * la.sk;
  const int fb = (wn0 + (lane >> 2)) * lb.so + (lane & 3) * lb.sk;
  int cur = 0;
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<ST - 2>();
    __syncthreads();  // chunk kt has landed; every warp is done with the stage that chunk kt + ST - 1 overwrites
    if (kt + ST - 1 < nk) {
      const uint32_t nb = sbase + (cur == 0 ? ST - 1 : cur - 1) * ST_BYTES;
      const int rem = k1 - k0 - (kt + ST - 1) * BK;
      la.load(nb, rem);
      lb.load(nb + A_BYTES, rem);
    }
    cp_async_commit();
    const TA* a_s = reinterpret_cast<const TA*>(smem_raw + cur * ST_BYTES) + fa;
    const TB* b_s = reinterpret_cast<const TB*>(smem_raw + cur * ST_BYTES + A_BYTES) + fb;
    cur = cur + 1 == ST ? 0 : cur + 1;
#pragma unroll
    for (int kq = 0; kq < BK / 4 / KW; ++kq) {
      const int kk = (KW == 1 ? kq : warp) * 4;
      double ar[F], ai[F], br[F], bi[F];
#pragma unroll
      for (int i = 0; i < F; ++i) {
        const TA va = a_s[i * 8 * la.so + kk * la.sk];
        if constexpr (AC) {
          ar[i] = va.x;
          ai[i] = sgnA * va.y;
        } else {
          ar[i] = va;
          ai[i] = 0.0;
        }
        const TB vb = b_s[i * 8 * lb.so + kk * lb.sk];
        if constexpr (BC) {
          br[i] = vb.x;
          bi[i] = sgnB * vb.y;
        } else {
          br[i] = vb;
          bi[i] = 0.0;
        }
      }
#pragma unroll
      for (int i = 0; i < F; ++i) {
#pragma unroll
        for (int j = 0; j < F; ++j) {
          dmma(accr[i][j][0], accr[i][j][1], ar[i], br[j]);
          if constexpr (AC && BC) dmma(accr[i][j][0], accr[i][j][1], -ai[i], bi[j]);
          if constexpr (BC) dmma(acci[i][j][0], acci[i][j][1], ar[i], bi[j]);
          if constexpr (AC) dmma(acci[i][j][0], acci[i][j][1], ai[i], br[j]);
        }
      }
    }
  }
  cp_async_wait<0>();

  TC* C = reinterpret_cast<TC*>(p.C) + b * p.sCb;
  auto put = [&](int m, int n, TC v) {
    if (m >= p.M || n >= p.N) return;
    TC* c = C + (int64_t)m * p.sCm + (int64_t)n * p.sCn;
    if (p.accumulate) {
      if constexpr (CC) {
        const double2 o = *c;
        v.x += o.x;
        v.y += o.y;
      } else {
        v += *c;
      }
    }
    *c = v;
  };
  if (KW == 1 && S == 1) {
    // fragment (i,j) element e sits at row lane/4, column 2*(lane%4)+e
#pragma unroll
    for (int i = 0; i < F; ++i)
#pragma unroll
      for (int j = 0; j < F; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int m = m0 + wm0 + i * 8 + (lane >> 2), n = n0 + wn0 + j * 8 + (lane & 3) * 2 + e;
          if constexpr (CC) put(m, n, make_double2(accr[i][j][e], acci[i][j][e]));
          else put(m, n, accr[i][j][e]);
        }
    return;
  }
  // partial tiles in shared memory: of the CTA's warps, then of the cluster's CTAs
  TC* part = reinterpret_cast<TC*>(smem_raw);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int at = (KW == 1 ? 0 : warp * BT * BT) + (wm0 + i * 8 + (lane >> 2)) * BT + wn0 + j * 8 +
                       (lane & 3) * 2 + e;
        if constexpr (CC) part[at] = make_double2(accr[i][j][e], acci[i][j][e]);
        else part[at] = accr[i][j][e];
      }
  __syncthreads();
  auto plus = [](TC x, TC y) {
    if constexpr (CC) return make_double2(x.x + y.x, x.y + y.y);
    else return x + y;
  };
  if constexpr (KW > 1) {
    for (int i = tid; i < BT * BT; i += THREADS) {
      TC v = part[i];
#pragma unroll
      for (int w = 1; w < KW; ++w) v = plus(v, part[w * BT * BT + i]);
      if (S == 1) put(m0 + i / BT, n0 + i % BT, v);
      else part[i] = v;
    }
    if (S == 1) return;
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  const int share = BT * BT / S;  // S is a power of two <= 8
  for (int i = rank * share + tid; i < (rank + 1) * share; i += THREADS) {
    TC v = cluster.map_shared_rank(part, 0)[i];
    for (int q = 1; q < S; ++q) v = plus(v, cluster.map_shared_rank(part, q)[i]);
    put(m0 + i / BT, n0 + i % BT, v);
  }
  cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// CTAs of a cluster are neighbours along x: tile = x / S, rank = x % S
template <bool AC, bool BC, int TILE>
__global__ void __launch_bounds__(THREADS, TILE == T64 ? 2 : 4)
    gemm_kernel(const __grid_constant__ GemmParams p, int S, int m_fast) {
  const int x = blockIdx.x / S, y = blockIdx.y;
  gemm_tile<AC, BC, TILE>(p, m_fast ? y : x, m_fast ? x : y, blockIdx.z, S, blockIdx.x % S);
}

// Many independent GEMMs (same operand types) in one launch: tile t belongs
// to problem i, first[i] <= t < first[i + 1], tiles of a problem numbered x
// fastest, then y, then batch.  CAP bounds the problems of a launch: the
// table is a kernel parameter, copied at every launch.
constexpr int MAX_GROUP = 128, SMALL_GROUP = 8;
template <int CAP>
struct GroupTable {
  int count, S;
  int first[CAP + 1];
  GemmParams p[CAP];
};
struct GemmGroup {
  int count = 0;
  GemmParams p[MAX_GROUP];
};

template <bool AC, bool BC, int TILE, int CAP>
__global__ void __launch_bounds__(THREADS, TILE == T64 ? 2 : 4)
    gemm_grouped_kernel(const __grid_constant__ GroupTable<CAP> g) {
  const int t = blockIdx.x / g.S;
  int lo = 0, hi = g.count;  // first[lo] <= t < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (g.first[mid] <= t) lo = mid;
    else hi = mid;
  }
  const GemmParams& p = g.p[lo];
  const int lt = t - g.first[lo];
  constexpr int BT = tile_dim(TILE);
  const int nx = (int)ceil_div(p.N, BT), ny = (int)ceil_div(p.M, BT);
  gemm_tile<AC, BC, TILE>(p, lt % nx, (lt / nx) % ny, lt / (nx * ny), g.S, blockIdx.x % g.S);
}

// Tile and K split of a problem: the least estimated time (microseconds).  A
// CTA's chain is its chunks, each as long as its MMAs (4 clocks apiece over
// the SM's four sub-partitions) plus the latency that its ring cannot hide;
// an SM works through its share of the CTAs at the FP64 pipe's rate times a
// measured factor, plus each CTA's start and epilogue (with a split: two
// cluster barriers and the partial sums).  T64 CTAs run in pairs, so an odd
// one costs a pair's time.  The constants are fitted to timings of 33 shapes
// from 32 x 32 x 128 to 2048^3; the choice was within 14 % of the best of the
// twelve (tile, split) pairs on each.
struct Choice {
  int tile, S;
};
inline Choice gemm_choose(const GemmParams& p) {
  const int f = (p.A.is_complex ? 2 : 1) * (p.B.is_complex ? 2 : 1);
  constexpr double kSms = 148.0, kClk = 1.0 / 1965.0;  // us per clock
  constexpr double lat[3] = {0.22, 0.18, 0.12}, fixed1[3] = {1.0, 0.3, 0.2}, fixedS[3] = {2.5, 1.0, 0.7};
  const double fac[3] = {f == 1 ? 1.3 : 1.12, f == 1 ? 1.33 : 1.17, f == 1 ? 1.65 : f == 2 ? 1.4 : 1.22};
  Choice best{T64, 1};
  double tbest = 1e300;
  for (int tile = T64; tile <= T16; ++tile) {
    const int bt = tile_dim(tile);
    const double tiles = (double)ceil_div(p.M, bt) * ceil_div(p.N, bt) * p.batch;
    for (int S = 1; S <= 8; S *= 2) {
      if (S > 1 && p.K / S < 2 * BK) break;
      const double chunks = (double)ceil_div(ceil_div(p.K, S), BK);
      const double mma = (BK / 4) * (bt / 8) * (bt / 8) * f * 4.0 * kClk;
      double per_sm = std::ceil(tiles * S / kSms);
      const double cta = S > 1 ? fixedS[tile] : fixed1[tile];
      const double chain = chunks * (mma + lat[tile]);
      if (tile == T64 && per_sm > 1.0) per_sm = 2.0 * std::ceil(per_sm / 2.0);
      const double t = std::max(chain, per_sm * chunks * mma * fac[tile]) + per_sm * cta + (S > 1 ? 1.0 : 0.0);
      if (t < tbest) {
        tbest = t;
        best = Choice{tile, S};
      }
    }
  }
  return best;
}

template <typename Kernel, typename... Args>
inline cudaError_t launch_clustered(Kernel* kernel, dim3 grid, size_t sm, int S, cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)S;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = S > 1 ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <bool AC, bool BC, int TILE>
inline cudaError_t launch_one(const GemmParams& p, int S, cudaStream_t st) {
  constexpr int BT = tile_dim(TILE);
  const size_t sm = smem_bytes<AC, BC, TILE>();
  static std::atomic<unsigned long long> smem_set{0};
  cudaError_t e = smem_optin_once(gemm_kernel<AC, BC, TILE>, (int)sm, smem_set);
  if (e != cudaSuccess) return e;
  const int64_t nx = ceil_div(p.N, BT), ny = ceil_div(p.M, BT);
  // walk the tiles of the smaller operand fastest, so that the larger one streams from HBM once;
  // the grid's y holds 65535 tiles (1.05 M rows of 16), so that a taller product has them along x
  const int m_fast = nx <= 65535 && (p.M < p.N || ny > 65535) ? 1 : 0;
  const dim3 grid((unsigned)((m_fast ? ny : nx) * S), (unsigned)(m_fast ? nx : ny), (unsigned)p.batch);
  return launch_clustered(gemm_kernel<AC, BC, TILE>, grid, sm, S, st, p, S, m_fast);
}

template <bool AC, bool BC, int TILE, int CAP>
inline cudaError_t launch_table(const GemmGroup& g, const int* idx, int count, int S, cudaStream_t st) {
  constexpr int BT = tile_dim(TILE);
  const size_t sm = smem_bytes<AC, BC, TILE>();
  static std::atomic<unsigned long long> smem_set{0};
  cudaError_t e = smem_optin_once(gemm_grouped_kernel<AC, BC, TILE, CAP>, (int)sm, smem_set);
  if (e != cudaSuccess) return e;
  GroupTable<CAP> t;
  t.count = count;
  t.S = S;
  t.first[0] = 0;
  for (int i = 0; i < count; ++i) {
    t.p[i] = g.p[idx[i]];
    const int64_t tiles = ceil_div(t.p[i].N, BT) * ceil_div(t.p[i].M, BT) * t.p[i].batch;
    if ((t.first[i] + tiles) * S > 0x7fffffff) return cudaErrorInvalidValue;
    t.first[i + 1] = t.first[i] + (int)tiles;
  }
  return launch_clustered(gemm_grouped_kernel<AC, BC, TILE, CAP>, dim3((unsigned)(t.first[count] * S)), sm, S, st, t);
}

template <bool AC, bool BC>
inline cudaError_t launch_t(const GemmParams& p, cudaStream_t st) {
  const Choice c = gemm_choose(p);
  if (c.tile == T64) return launch_one<AC, BC, T64>(p, c.S, st);
  if (c.tile == T32) return launch_one<AC, BC, T32>(p, c.S, st);
  return launch_one<AC, BC, T16>(p, c.S, st);
}

// One launch per (tile, split) that the group's problems choose.
template <bool AC, bool BC>
inline cudaError_t launch_grouped_t(const GemmGroup& g, cudaStream_t st) {
  Choice ch[MAX_GROUP];
  bool done[MAX_GROUP];
  for (int i = 0; i < g.count; ++i) {
    done[i] = g.p[i].M <= 0 || g.p[i].N <= 0 || g.p[i].batch <= 0;
    if (!done[i]) ch[i] = gemm_choose(g.p[i]);
  }
  for (int i = 0; i < g.count; ++i) {
    if (done[i]) continue;
    int idx[MAX_GROUP], n = 0;
    for (int j = i; j < g.count; ++j)
      if (!done[j] && ch[j].tile == ch[i].tile && ch[j].S == ch[i].S) {
        idx[n++] = j;
        done[j] = true;
      }
    cudaError_t e;
    const int S = ch[i].S;
    if (n <= SMALL_GROUP) {
      e = ch[i].tile == T64   ? launch_table<AC, BC, T64, SMALL_GROUP>(g, idx, n, S, st)
          : ch[i].tile == T32 ? launch_table<AC, BC, T32, SMALL_GROUP>(g, idx, n, S, st)
                              : launch_table<AC, BC, T16, SMALL_GROUP>(g, idx, n, S, st);
    } else {
      e = ch[i].tile == T64   ? launch_table<AC, BC, T64, MAX_GROUP>(g, idx, n, S, st)
          : ch[i].tile == T32 ? launch_table<AC, BC, T32, MAX_GROUP>(g, idx, n, S, st)
                              : launch_table<AC, BC, T16, MAX_GROUP>(g, idx, n, S, st);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace fp64gemm

// A group of FP64 GEMMs whose operands all have the same types; every
// problem's result is bitwise that of its own gemm_fp64.
inline cudaError_t gemm_fp64_grouped(const fp64gemm::GemmGroup& g, cudaStream_t st) {
  if (g.count < 1 || g.count > fp64gemm::MAX_GROUP) return cudaErrorInvalidValue;
  const bool ac = g.p[0].A.is_complex, bc = g.p[0].B.is_complex;
  for (int i = 0; i < g.count; ++i) {
    const GemmParams& p = g.p[i];
    if (p.A.is_f32 || p.B.is_f32 || p.c_f32 || (bool)p.A.is_complex != ac || (bool)p.B.is_complex != bc)
      return cudaErrorInvalidValue;
  }
  if (ac && bc) return fp64gemm::launch_grouped_t<true, true>(g, st);
  if (ac) return fp64gemm::launch_grouped_t<true, false>(g, st);
  if (bc) return fp64gemm::launch_grouped_t<false, true>(g, st);
  return fp64gemm::launch_grouped_t<false, false>(g, st);
}

// Launch the FP64 GEMM; returns a CUDA error code.
inline cudaError_t gemm_fp64(const GemmParams& p, cudaStream_t st) {
  if (p.M <= 0 || p.N <= 0 || p.batch <= 0) return cudaSuccess;
  // FP32 operands / outputs exist only between split-precision stages
  if (p.A.is_f32 || p.B.is_f32 || p.c_f32) return cudaErrorInvalidValue;
  const bool ac = p.A.is_complex, bc = p.B.is_complex;
  if (ac && bc) return fp64gemm::launch_t<true, true>(p, st);
  if (ac) return fp64gemm::launch_t<true, false>(p, st);
  if (bc) return fp64gemm::launch_t<false, true>(p, st);
  return fp64gemm::launch_t<false, false>(p, st);
}

}  // namespace reno
