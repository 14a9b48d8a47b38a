// Split-precision complex GEMM on the 5th-generation tensor cores (sm_100a).
//
// C (real or complex) = opA(A) opB(B) with A, B real or complex with any
// strides, computed as
//     A ~ A_hi + A_lo,  B ~ B_hi + B_lo    (BF16 or TF32 pairs)
//     C ~ A_hi B_hi + A_hi B_lo + A_lo B_hi   (FP32 accumulation in TMEM)
// Complex operands use the real embedding: the smaller operand is "doubled"
// into [[Re, -Im], [Im, Re]] rows, the other is K-concatenated as [Re | Im],
// so each complex GEMM is ONE real GEMM whose rows (or columns) interleave the
// real and imaginary parts of the result.
//
// Pipeline (persistent: one CTA per SM walks 128 x 256 output tiles; 10 warps):
//   warp 0     TMA producer: 4 tiles per stage (A_hi, A_lo, B_hi, B_lo),
//              64-byte swizzled K-major boxes, mbarrier complete_tx.  Four
//              48 KB stages: with two of 96 KB only one is in flight while the
//              other computes, too little to cover the L2's latency (M = 256
//              two-site matvec 1604 -> 1576 us, its last stage 360 -> 322; the
//              first loads 3.8 GB through L2 in 413 us)
//   warp 1     TMEM allocator + single-thread tcgen05.mma issuer: 3 products
//              per stage, tcgen05.commit frees the stage
//   warps 2-9  epilogue (two warps per TMEM lane quarter, half the columns
//              each): tcgen05.ld 32x32b from TMEM, strided writes of the
//              (interleaved complex) output as FP64, or as FP32 when the
//              output only feeds the next split stage (the accumulator is
//              FP32, so nothing is lost) -- the operands A, B are FP64 or
//              such FP32 intermediates
// Every mbarrier wait is bounded; on timeout the kernel records the site in
// a device error word, skips the remaining work and still frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cstring>
#include "split_gemm.cuh"

namespace reno {
namespace split {

constexpr int EPI_WARPS = 8;  // 16 do not gain: the stores are bound by the load/store unit, not by latency
constexpr int BM = 128, BN = 256, STAGES = 4, THREADS = 32 * (2 + EPI_WARPS);  // warp 0 TMA, warp 1 MMA, then epilogue
constexpr int EPI_COLS = BN * 4 / EPI_WARPS;  // columns of a tile per epilogue warp
constexpr int KROW_BYTES = 64;  // one SW64 row of K per stage
constexpr int A_TILE = BM * KROW_BYTES;   // 8 KB
constexpr int B_TILE = BN * KROW_BYTES;   // 16 KB
constexpr int STAGE_BYTES = 2 * A_TILE + 2 * B_TILE;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
constexpr uint32_t TMEM_COLS = 256;  // one accumulator buffer (two are allocated)

// device error word: 0 = ok; otherwise 1000 + site of the first timed-out wait
__device__ int g_split_error = 0;

enum OutMode { OUT_REAL = 0, OUT_COLS_CPLX = 1, OUT_ROWS_CPLX = 2, OUT_PACK = 3 };

struct Epi {
  void* C;
  int64_t sCm, sCn, sCb;  // output strides in output elements
  int M, N;               // logical output dims
  int mode;
  int accumulate;
  int rows_p, cols_p;     // rows / cols of the real product C' actually present
  int c_f32;              // C holds float (complex: float2) instead of double
  // OUT_PACK: the tile is written as the next split stage's packed operand.
  // Output element (m, n, ri) of the real product (ri: re/im component, from
  // the row interleave when A was doubled, inter = 1, or the column interleave
  // when B was doubled, inter = 2) goes to hi/lo element
  //   bz*s_b + (m / Dm)*s_m1 + (m % Dm)*s_m0 + (n / Dn)*s_n1 + (n % Dn)*s_n0 + ri*s_ri
  void* phi;
  void* plo;
  int64_t s_b, s_m1, s_m0, s_n1, s_n0, s_ri;
  int Dm, Dn, inter;
};

template <typename T>
__device__ __forceinline__ void st_real(void* C, int64_t i, float v, int acc) {
  T* p = reinterpret_cast<T*>(C) + i;
  *p = (acc ? *p : T(0)) + (T)v;
}

template <typename T2>
__device__ __forceinline__ void st_cplx(void* C, int64_t i, float re, float im, int acc) {
  T2* p = reinterpret_cast<T2*>(C) + i;
  T2 o = acc ? *p : T2{0, 0};
  o.x += re;
  o.y += im;
  *p = o;
}

// x = hi + lo in the split format: bits of hi and lo (BF16 in the low 16 bits, or TF32)
template <int ESZ>
__device__ __forceinline__ void split_bits(float x, uint32_t& hb, uint32_t& lb) {
  if constexpr (ESZ == 2) {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
    hb = __bfloat16_as_ushort(h);
    lb = __bfloat16_as_ushort(l);
  } else {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(x));
    const float rem = x - __uint_as_float(hb);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lb) : "f"(rem));
  }
}

template <int ESZ>
__device__ __forceinline__ void split_store_bits(void* hi, void* lo, int64_t idx, uint32_t hb, uint32_t lb) {
  if constexpr (ESZ == 2) {
    reinterpret_cast<unsigned short*>(hi)[idx] = (unsigned short)hb;
    reinterpret_cast<unsigned short*>(lo)[idx] = (unsigned short)lb;
  } else {
    reinterpret_cast<uint32_t*>(hi)[idx] = hb;
    reinterpret_cast<uint32_t*>(lo)[idx] = lb;
  }
}

// one 32-byte store (p is 32-byte aligned)
__device__ __forceinline__ void st_global_v8(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

__device__ __forceinline__ void st_global_v4(void* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// 16 output values v[t*STRIDE + OFF] (t = 0..15) of one (m, ri) for columns
// n0 .. n0+15 into the packed planes: 32-byte stores (whole sectors; 16-byte
// ones took up to a fifth of a stage longer) when the run is contiguous and its
// address allows it, 16-byte ones where it lies on half a sector (an odd row pitch, or a
// workspace that is itself aligned to 16 bytes, all that the tensor maps ask for),
// scalar stores otherwise.  Lanes hold different rows, so a store
// instruction costs a cycle of the load/store unit per lane whatever its width.
template <int ESZ, int STRIDE, int OFF>
__device__ __forceinline__ void pack_run(const float* v, const Epi& e, int64_t mbase, int n0, int ri) {
  if (n0 >= e.N) return;
  const int nq = n0 / e.Dn;
  int nr = n0 - nq * e.Dn;
  const int64_t idx0 = mbase + (int64_t)ri * e.s_ri + (int64_t)nq * e.s_n1 + (int64_t)nr * e.s_n0;
  unsigned char* planes[2] = {reinterpret_cast<unsigned char*>(e.phi) + idx0 * ESZ,
                              reinterpret_cast<unsigned char*>(e.plo) + idx0 * ESZ};
  const uintptr_t off = (reinterpret_cast<uintptr_t>(planes[0]) | reinterpret_cast<uintptr_t>(planes[1])) % 32;
  if (e.s_n0 == 1 && n0 + 16 <= e.N && nr + 16 <= e.Dn && off % 16 == 0) {
    uint32_t hb[16], lb[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) split_bits<ESZ>(v[t * STRIDE + OFF], hb[t], lb[t]);
    uint32_t w[4 * ESZ];  // 16 elements of one plane, 32 bits at a time
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
      const uint32_t* src = pl == 0 ? hb : lb;
#pragma unroll
      for (int q = 0; q < 4 * ESZ; ++q) w[q] = ESZ == 2 ? src[2 * q] | (src[2 * q + 1] << 16) : src[q];
      if (off == 0) {
#pragma unroll
        for (int q = 0; q < ESZ / 2; ++q) st_global_v8(planes[pl] + 32 * q, w + 8 * q);
      } else {
#pragma unroll
        for (int q = 0; q < ESZ; ++q)
          reinterpret_cast<uint4*>(planes[pl])[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      }
    }
  } else {
    // the index moves along with n: with a division per element this branch took 220 cycles a value, and
    // the third stage of an M = 192 two-site matvec 649 us (206 now)
    const int64_t wrap = e.s_n1 - (int64_t)e.Dn * e.s_n0;
    int64_t idx = idx0;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      if (n0 + t < e.N) {
        uint32_t hb, lb;
        split_bits<ESZ>(v[t * STRIDE + OFF], hb, lb);
        split_store_bits<ESZ>(e.phi, e.plo, idx, hb, lb);
        idx += e.s_n0;
        if (++nr == e.Dn) {
          nr = 0;
          idx += wrap;
        }
      }
    }
  }
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// bounded wait (wait_ns of wall clock): returns false and raises the abort flag on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int site,
                                          uint64_t wait_ns) {
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > wait_ns) break;
    }
  }
  *abort_flag = 1;
  atomicCAS(&g_split_error, 0, 1000 + site);
  return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// K-major, 64-byte swizzle shared-memory matrix descriptor (SBO = 8 rows x 64 B)
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;            // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512u >> 4) << 32;   // stride byte offset
  d |= (uint64_t)1u << 46;            // descriptor version for sm_100
  d |= (uint64_t)4u << 61;            // SWIZZLE_64B
  return d;
}

template <int ESZ>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  if constexpr (ESZ == 2) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc));
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc));
  }
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

#define TMEM_LD32(taddr, r)                                                                                         \
  asm volatile(                                                                                                     \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18," \
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"                                                \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),            \
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),      \
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),    \
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])     \
      : "r"(taddr))

// Epilogue of columns [c_begin, c_end) of one output tile: TMEM -> registers
// (32 columns at a time) -> the output in the Epi mode.  Warp w reads TMEM
// lane quarter q = w % 4, i.e. tile rows q*32 .. q*32+31; two warps share a
// quarter, each taking half of the BN columns.
// Output of 32 accumulated columns c0 .. c0+31 of tile row q*32 + lane in the
// Epi mode.
template <int ESZ>
__device__ __forceinline__ void epilogue_store(const Epi& epi, const float* v, int q, int lane, int m_tile, int n_tile,
                                               int bz, int c0) {
  const int row = q * 32 + lane;  // tile row of this thread
  const int rp = m_tile * BM + row;
  {
    const int cp = n_tile * BN + c0;  // product column of v[0]
    if (epi.mode == OUT_PACK) {
      const int m = epi.inter == 1 ? (rp >> 1) : rp;
      if (m < epi.M) {
        const int64_t mbase =
            (int64_t)bz * epi.s_b + (int64_t)(m / epi.Dm) * epi.s_m1 + (int64_t)(m % epi.Dm) * epi.s_m0;
        if (epi.inter == 2) {
          pack_run<ESZ, 2, 0>(v, epi, mbase, cp / 2, 0);
          pack_run<ESZ, 2, 1>(v, epi, mbase, cp / 2, 1);
        } else {
          const int ri = epi.inter == 1 ? (rp & 1) : 0;
          pack_run<ESZ, 1, 0>(v, epi, mbase, cp, ri);
          pack_run<ESZ, 1, 16>(v, epi, mbase, cp + 16, ri);
        }
      }
    } else if (epi.mode == OUT_REAL) {
      if (rp < epi.M) {
        const int64_t base = (int64_t)bz * epi.sCb + (int64_t)rp * epi.sCm;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int n = cp + j;
          if (n < epi.N) {
            if (epi.c_f32)
              st_real<float>(epi.C, base + (int64_t)n * epi.sCn, v[j], epi.accumulate);
            else
              st_real<double>(epi.C, base + (int64_t)n * epi.sCn, v[j], epi.accumulate);
          }
        }
      }
    } else if (epi.mode == OUT_COLS_CPLX) {
      if (rp < epi.M) {
        const int64_t base = (int64_t)bz * epi.sCb + (int64_t)rp * epi.sCm;
        const int64_t first = base + cp / 2;
        if (epi.sCn == 1 && !epi.c_f32 && !epi.accumulate && cp / 2 + 16 <= epi.N &&
            (reinterpret_cast<uintptr_t>(epi.C) + 16 * (uint64_t)first) % 32 == 0) {
          // two complex numbers, one whole 32-byte sector, per store
          double2* p = reinterpret_cast<double2*>(epi.C) + first;
#pragma unroll
          for (int j = 0; j < 8; ++j) st_global_v4(p + 2 * j, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          return;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int n = cp / 2 + j;
          if (n < epi.N) {
            if (epi.c_f32)
              st_cplx<float2>(epi.C, base + (int64_t)n * epi.sCn, v[2 * j], v[2 * j + 1], epi.accumulate);
            else
              st_cplx<double2>(epi.C, base + (int64_t)n * epi.sCn, v[2 * j], v[2 * j + 1], epi.accumulate);
          }
        }
      }
    } else {
      // rows interleave re/im: lanes (2i, 2i+1) hold (re, im) of complex row rp/2
      const bool even = (lane & 1) == 0;
      float mine[16], got[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float send = even ? v[16 + j] : v[j];
        got[j] = __shfl_xor_sync(0xffffffffu, send, 1);
        mine[j] = even ? v[j] : v[16 + j];
      }
      const int m = rp >> 1;
      if (m < epi.M) {
        const int64_t base = (int64_t)bz * epi.sCb + (int64_t)m * epi.sCm;
        const int nb = cp + (even ? 0 : 16);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int n = nb + j;
          if (n < epi.N) {
            const float re = even ? mine[j] : got[j], im = even ? got[j] : mine[j];
            if (epi.c_f32)
              st_cplx<float2>(epi.C, base + (int64_t)n * epi.sCn, re, im, epi.accumulate);
            else
              st_cplx<double2>(epi.C, base + (int64_t)n * epi.sCn, re, im, epi.accumulate);
          }
        }
      }
    }
  }
}

template <int ESZ>
__device__ __forceinline__ void epilogue_tile(const Epi& epi, uint32_t tacc, int q, int lane, int m_tile, int n_tile,
                                              int bz, int c_begin, int c_end) {
  c_end = min(c_end, epi.cols_p - n_tile * BN);  // columns past the operand's last row hold nothing
  for (int c0 = c_begin; c0 < c_end; c0 += 32) {
    uint32_t r[32];
    const uint32_t taddr = tacc + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
    TMEM_LD32(taddr, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;");
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
    epilogue_store<ESZ>(epi, v, q, lane, m_tile, n_tile, bz, c0);
  }
}

// tile t of the (bz, slow, fast) raster: M tiles fastest when m_fast
__device__ __forceinline__ void tile_coords(int t, int mt, int nt, int m_fast, int& m_tile, int& n_tile, int& bz) {
  const int per = mt * nt;
  bz = t / per;
  const int r = t - bz * per;
  if (m_fast) {
    m_tile = r % mt;
    n_tile = r / mt;
  } else {
    n_tile = r % nt;
    m_tile = r / nt;
  }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait that ignores the abort flag: used only to drain the CTA's own
// copies and MMAs in flight before it frees TMEM and exits
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity, uint64_t wait_ns) {
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0;; ++it) {
    if (mbar_try(bar, parity)) return;
    if ((it & 255u) == 255u && global_ns() - t0 > wait_ns) {
      atomicCAS(&g_split_error, 0, 1009);
      return;
    }
  }
}

// Persistent kernel: one CTA per SM walks output tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ... in the raster above.  TMEM holds two BN-column
// FP32 accumulators; the MMA thread fills buffer (i & 1) for the CTA's i-th
// tile while the epilogue warps drain the other, so each tile's epilogue
// overlaps the next tile's TMA + MMA mainloop.  The smem stage ring runs on
// across tiles.  Barriers: full / empty (TMA <-> MMA, per stage), tmem_full
// (MMA -> epilogue, per buffer, tcgen05.commit), tmem_empty (epilogue -> MMA,
// per buffer, one arrive per epilogue warp, 8 warps), drain (the MMA thread's last
// commit, waited for before TMEM is freed).
//
// PROMOTE (opt-in, reno_set_split_accumulation_chunk): the tensor cores'
// FP32 accumulation truncates, so its error is a bias that grows with the
// number of terms.  In this form a tile's K range is cut into chunks of kc K
// tiles; each chunk accumulates in one TMEM buffer (the two buffers
// alternate chunk by chunk, so the MMA fills one while the epilogue reads the
// other), and the epilogue warps add every chunk's partial sums into FP32
// registers with round-to-nearest additions before the tile's output.
template <int ESZ, bool PROMOTE>
__global__ void __launch_bounds__(THREADS, 1)
    split_gemm_kernel(const __grid_constant__ CUtensorMap tmAh, const __grid_constant__ CUtensorMap tmAl,
                      const __grid_constant__ CUtensorMap tmBh, const __grid_constant__ CUtensorMap tmBl, Epi epi,
                      int num_k_tiles, int k_elems, int a_batched, int b_batched, int m_fast, int mt, int nt,
                      int ntiles, uint64_t wait_ns, int skip_stage, int kc) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;  // [2]
  uint64_t* tmem_empty = tmem_full + 2;  // [2]
  uint64_t* drain = tmem_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], EPI_WARPS);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer
    uint32_t g = 0;  // k tiles issued by this CTA
    bool ok = true;
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
      int m_tile, n_tile, bz;
      tile_coords(t, mt, nt, m_fast, m_tile, n_tile, bz);
      const int za = a_batched ? bz : 0, zb = b_batched ? bz : 0;
      for (int kt = 0; kt < num_k_tiles; ++kt) {
        const int s = g % STAGES;
        const uint32_t ph = (g / STAGES) & 1;
        if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, 1, wait_ns)) {
          ok = false;
          break;
        }
        if (blockIdx.x == 0 && (int)g == skip_stage) {  // test hook: stage g of CTA 0 stays unloaded
          ++g;
          continue;
        }
        unsigned char* st = smem + s * STAGE_BYTES;
        mbar_expect_tx(&full[s], STAGE_BYTES);
        const int kx = kt * (KROW_BYTES / ESZ);
        tma_load_3d(st, &tmAh, &full[s], kx, m_tile * BM, za);
        tma_load_3d(st + A_TILE, &tmAl, &full[s], kx, m_tile * BM, za);
        tma_load_3d(st + 2 * A_TILE, &tmBh, &full[s], kx, n_tile * BN, zb);
        tma_load_3d(st + 2 * A_TILE + B_TILE, &tmBl, &full[s], kx, n_tile * BN, zb);
        ++g;
      }
    }
    // land every copy this CTA issued before it can exit (immediate for the
    // ones the MMA thread already consumed)
    for (uint32_t j = (g > (uint32_t)STAGES ? g - STAGES : 0u); j < g; ++j)
      mbar_drain(&full[j % STAGES], (j / STAGES) & 1, wait_ns);
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    constexpr uint32_t fmt = ESZ == 2 ? 1u : 2u;  // BF16 : TF32
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);
    uint32_t g = 0;
    bool ok = true;
    int i = 0;  // accumulation units: tiles, or (tile, chunk) pairs under PROMOTE
    const int chunk = PROMOTE ? kc : num_k_tiles;
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
     for (int k0 = 0; k0 < num_k_tiles && ok; k0 += chunk, ++i) {
      const int b = i & 1;
      const uint32_t use = (uint32_t)(i >> 1);
      if (!mbar_wait(&tmem_empty[b], (use & 1) ^ 1, abort_flag, 4, wait_ns)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t tacc = tmem + (uint32_t)(b * TMEM_COLS);
      const int k1 = min(num_k_tiles, k0 + chunk);
      for (int kt = k0; kt < k1; ++kt) {
        const int s = g % STAGES;
        const uint32_t ph = (g / STAGES) & 1;
        if (!mbar_wait(&full[s], ph, abort_flag, 2, wait_ns)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t base = smem_u32(smem + s * STAGE_BYTES);
        const uint64_t dah = sdesc(base), dal = sdesc(base + A_TILE);
        const uint64_t dbh = sdesc(base + 2 * A_TILE), dbl = sdesc(base + 2 * A_TILE + B_TILE);
        // K beyond k_elems is TMA zero fill: skip the sub-steps that only see it
        constexpr int STEPS = KROW_BYTES / 32, SUB = 32 / ESZ;  // 32-byte instruction steps, elements of one
        const int rem = k_elems - kt * (KROW_BYTES / ESZ);
        const int nsub = rem >= STEPS * SUB ? STEPS : (rem + SUB - 1) / SUB;
#pragma unroll
        for (int kk = 0; kk < STEPS; ++kk) {
          if (kk < nsub) {
            const uint64_t adv = (uint64_t)((kk * 32) >> 4);  // 32 bytes of K per instruction
            const uint32_t first = (kt == k0 && kk == 0) ? 0u : 1u;
            umma<ESZ>(tacc, dah + adv, dbh + adv, idesc, first);
            umma<ESZ>(tacc, dah + adv, dbl + adv, idesc, 1u);
            umma<ESZ>(tacc, dal + adv, dbh + adv, idesc, 1u);
          }
        }
        umma_commit(&empty[s]);
        ++g;
      }
      if (ok) umma_commit(&tmem_full[b]);
    }
    // every MMA this thread issued completes before TMEM is freed
    umma_commit(drain);
    mbar_drain(drain, 0, wait_ns);
  } else if (warp >= 2) {
    // ---------------- epilogue
    const int q = warp % 4;                      // TMEM lane quarter this warp may access
    const int c_begin = ((warp - 2) / 4) * EPI_COLS;  // four warps (one per quarter) share a column range
    int i = 0;
    if constexpr (PROMOTE) {
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        float acc[EPI_COLS];  // this thread's row, columns c_begin .. c_begin + EPI_COLS - 1
        for (int k0 = 0; k0 < num_k_tiles; k0 += kc, ++i) {
          const int b = i & 1;
          const uint32_t use = (uint32_t)(i >> 1);
          if (!mbar_wait(&tmem_full[b], use & 1, abort_flag, 3, wait_ns) || *abort_flag) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t tacc = tmem + (uint32_t)(b * TMEM_COLS) + ((uint32_t)(q * 32) << 16) + (uint32_t)c_begin;
#pragma unroll
          for (int p = 0; p < EPI_COLS / 32; ++p) {
            uint32_t r[32];
            TMEM_LD32(tacc + (uint32_t)(32 * p), r);
            asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
            for (int j = 0; j < 32; ++j)
              acc[32 * p + j] = k0 == 0 ? __uint_as_float(r[j]) : __fadd_rn(acc[32 * p + j], __uint_as_float(r[j]));
          }
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncwarp();
          if (lane == 0) mbar_arrive(&tmem_empty[b]);
        }
        if (!ok) break;
        int m_tile, n_tile, bz;
        tile_coords(t, mt, nt, m_fast, m_tile, n_tile, bz);
#pragma unroll
        for (int p = 0; p < EPI_COLS / 32; ++p) epilogue_store<ESZ>(epi, acc + 32 * p, q, lane, m_tile, n_tile, bz, c_begin + 32 * p);
      }
    } else {
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
      const int b = i & 1;
      const uint32_t use = (uint32_t)(i >> 1);
      if (!mbar_wait(&tmem_full[b], use & 1, abort_flag, 3, wait_ns)) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      if (*abort_flag) break;
      int m_tile, n_tile, bz;
      tile_coords(t, mt, nt, m_fast, m_tile, n_tile, bz);
      epilogue_tile<ESZ>(epi, tmem + (uint32_t)(b * TMEM_COLS), q, lane, m_tile, n_tile, bz, c_begin,
                         c_begin + EPI_COLS);
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[b]);
    }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TMEM_COLS));
  }
}

// ------------------------------------------------------------------ packing
// Operand packing modes (rows R, reduction length K of the logical operand):
enum PackMode {
  P_REAL = 0,       // out[r][k]       = x[r,k]                       K' = K
  P_CAT = 1,        // out[r][k | K+k] = (re, im) of x[r,k]           K' = 2K
  P_DBL_CPLX = 2,   // out[2r] = [re, -im], out[2r+1] = [im, re]      K' = 2K, 2R rows
  P_DBL_SPLIT = 3   // out[2r][k] = re, out[2r+1][k] = im             K' = K,  2R rows
};

// Rows are packed in groups: row r = g + i * rstep, i = 0 .. ceil((R - g) / rstep) - 1,
// sits at (g % D0) * s_g0 + (g / D0) * s_g1 + i * s_i.  A plain row stride is one
// group; an operand whose rows run over several of the source's indices is
// cut into groups along the index that is contiguous in the source.
struct PackArgs {
  const void* src;
  int src_complex, conj, src_f32;
  int64_t s_k, s_b;  // element strides of K and batch
  int D0, rstep;
  int64_t s_g0, s_g1, s_i;
  int R, K;
  int rtiles, ktiles;
  void* hi;
  void* lo;
  int64_t pitch;        // row pitch of the packed buffer (elements, 16-byte multiple)
  int64_t rows_out;     // rows per batch in the packed buffer
};

template <int ESZ>
__device__ __forceinline__ void split_store(void* hi, void* lo, int64_t idx, double x) {
  if constexpr (ESZ == 2) {
    const __nv_bfloat16 h = __double2bfloat16(x);
    const __nv_bfloat16 l = __double2bfloat16(x - (double)__bfloat162float(h));
    reinterpret_cast<__nv_bfloat16*>(hi)[idx] = h;
    reinterpret_cast<__nv_bfloat16*>(lo)[idx] = l;
  } else {
    const float f = (float)x;
    uint32_t hb, lb;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(f));
    const float h = __uint_as_float(hb);
    const float rem = (float)(x - (double)h);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lb) : "f"(rem));
    reinterpret_cast<float*>(hi)[idx] = h;
    reinterpret_cast<float*>(lo)[idx] = __uint_as_float(lb);
  }
}

// |x| is 0 or in a range in which x and x - BF16(x) (0, or at most 53 binary
// orders below x) are both normal FP32 numbers or 0
__device__ __forceinline__ bool float_range(double x) {
  const uint32_t mag = (uint32_t)__double2hiint(x) & 0x7fffffffu;
  return mag - (960u << 20) < ((1150u - 960u) << 20) || (mag | (uint32_t)__double2loint(x)) == 0;
}

// x as FP32 rounded to odd (truncated, last bit set when that was inexact): a
// later rounding to BF16 then gives what rounding x itself would.  For x in
// FP32's normal range or 0, in integer operations: conversions from FP64 and
// back kept the whole pack from running at the memory's rate.
__device__ __forceinline__ float float_to_odd(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mag = __funnelshift_l(lo, max(hi & 0x7fffffffu, 896u << 20) - (896u << 20), 3);
  return __uint_as_float((hi & 0x80000000u) | mag | min(lo & 0x1fffffffu, 1u));
}

// elements idx and idx + 1 (n = 2; one when n = 1) of a packed row: one store
// per plane when the pair is aligned.  FAST: both values are in float_range.
template <int ESZ, bool FAST>
__device__ __forceinline__ void split_store_pair(void* hi, void* lo, int64_t idx, double x0, double x1, int n) {
  if (n == 2 && (idx & 1) == 0) {
    if constexpr (FAST) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(float_to_odd(x0), float_to_odd(x1));
      reinterpret_cast<__nv_bfloat162*>(hi)[idx >> 1] = h;
      reinterpret_cast<__nv_bfloat162*>(lo)[idx >> 1] = __floats2bfloat162_rn(
          float_to_odd(x0 - (double)__low2float(h)), float_to_odd(x1 - (double)__high2float(h)));
      return;
    }
    if constexpr (ESZ == 4) {
      float h[2], l[2];
      split_store<ESZ>(h, l, 0, x0);
      split_store<ESZ>(h, l, 1, x1);
      reinterpret_cast<float2*>(hi)[idx >> 1] = make_float2(h[0], h[1]);
      reinterpret_cast<float2*>(lo)[idx >> 1] = make_float2(l[0], l[1]);
      return;
    }
  }
  split_store<ESZ>(hi, lo, idx, x0);
  if (n == 2) split_store<ESZ>(hi, lo, idx + 1, x1);
}

constexpr int PACK_R = 32, PACK_K = 64;

// rows i0 + ty, i0 + ty + 8, ... of a staged tile -> the packed planes
template <int ESZ, int MODE, bool FAST>
__device__ __forceinline__ void pack_rows(const PackArgs& a, const double2 (*tile)[PACK_K + 1], int64_t base, int rows,
                                          int64_t r, int k) {
  const int n = min(a.K - k, 2), tx = threadIdx.x;
  if (n <= 0) return;
  constexpr bool DBL = MODE == P_DBL_CPLX || MODE == P_DBL_SPLIT;
  int64_t at = base + (DBL ? 2 * r : r) * a.pitch + k;
  const int64_t step = (DBL ? 16 : 8) * (int64_t)a.rstep * a.pitch;
  for (int i = threadIdx.y; i < rows; i += 8, at += step) {
    const double2 p = tile[i][2 * tx], q = tile[i][2 * tx + 1];
    split_store_pair<ESZ, FAST>(a.hi, a.lo, at, p.x, q.x, n);
    if constexpr (MODE == P_CAT) {
      split_store_pair<ESZ, FAST>(a.hi, a.lo, at + a.K, p.y, q.y, n);
    } else if constexpr (MODE == P_DBL_CPLX) {
      split_store_pair<ESZ, FAST>(a.hi, a.lo, at + a.K, -p.y, -q.y, n);
      split_store_pair<ESZ, FAST>(a.hi, a.lo, at + a.pitch, p.y, q.y, n);
      split_store_pair<ESZ, FAST>(a.hi, a.lo, at + a.pitch + a.K, p.x, q.x, n);
    } else if constexpr (MODE == P_DBL_SPLIT) {
      split_store_pair<ESZ, FAST>(a.hi, a.lo, at + a.pitch, p.y, q.y, n);
    }
  }
}

template <typename T>
__device__ __forceinline__ double2 pack_value(T x, double) { return make_double2((double)x, 0.0); }
__device__ __forceinline__ double2 pack_value(double2 x, double s) { return make_double2(x.x, s * x.y); }
__device__ __forceinline__ double2 pack_value(float2 x, double s) { return make_double2(x.x, s * x.y); }

// the 32 x 64 source tile into shared memory, eight loads of each thread in
// flight at once; returns whether all of the thread's values are in float_range
template <typename T>
__device__ __forceinline__ bool pack_load(const PackArgs& a, double2 (*tile)[PACK_K + 1], int64_t src0, int rows,
                                          int cols, bool k_fast) {
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  // value j sits (j >> 1) big and (j & 1) small steps from the thread's first
  const int i0 = k_fast ? ty : tx, c0 = k_fast ? tx : ty;
  const int di = k_fast ? 8 : 0, dc = k_fast ? 0 : 16, ec = k_fast ? 32 : 8;
  const int64_t big = di * a.s_i + dc * a.s_k, small = ec * a.s_k;
  const T* src = reinterpret_cast<const T*>(a.src) + src0 + (int64_t)i0 * a.s_i + (int64_t)c0 * a.s_k;
  T v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = T{};
    if (i0 + (j >> 1) * di < rows && c0 + (j >> 1) * dc + (j & 1) * ec < cols) v[j] = src[(j >> 1) * big + (j & 1) * small];
  }
  const double sgn = a.conj ? -1.0 : 1.0;
  double2* t = &tile[i0][c0];
  const int tbig = di * (PACK_K + 1) + dc;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const double2 x = pack_value(v[j], sgn);
    ok = ok && float_range(x.x) && float_range(x.y);
    t[(j >> 1) * tbig + (j & 1) * ec] = x;
  }
  return ok;
}

// One 32 x 64 (rows x K) source tile per block, staged through shared memory so
// that both the strided reads (FP64, or FP32 intermediates) and the
// K-contiguous packed writes coalesce.  Packed rows hold K' elements at a
// 16-byte pitch; the tensor maps end at K', so the TMA loads zero-fill the
// rest of the last K tile and no padding is ever written.  Each
// thread has its eight loads in flight at once, and a warp writes 128 bytes of
// a BF16 row.  Bound by instruction issue (2.8 a cycle; 52% of the memory's
// rate): the psi operand of the M = 256 two-site matvec, 16.8 M complex
// numbers, 403 MB moved, takes 87 us, 63 at the copy rate.  With rows read
// across the source's contiguous index and every pair rounded by FP64
// conversions it took 127 us.
template <int ESZ, int MODE>
__global__ void __launch_bounds__(256, 5) pack_kernel(PackArgs a) {
  __shared__ double2 tile[PACK_R][PACK_K + 1];
  const int b = blockIdx.z;
  // row tiles fastest: neighbouring blocks read on along the source's contiguous index
  int x = blockIdx.x;
  const int i0 = (x % a.rtiles) * PACK_R;
  x /= a.rtiles;
  const int g = x % a.rstep;
  const int k0 = (x / a.rstep) * PACK_K;
  const int rows = min(PACK_R, (a.R - g + a.rstep - 1) / a.rstep - i0);  // of this group, in this tile
  const int64_t src0 = (int64_t)b * a.s_b + (int64_t)(g % a.D0) * a.s_g0 + (int64_t)(g / a.D0) * a.s_g1 +
                       (int64_t)i0 * a.s_i + (int64_t)k0 * a.s_k;
  const bool k_fast = (a.s_k == 1) || (a.s_i != 1);
  const int cols = a.K - k0;
  bool ok;
  if (a.src_complex)
    ok = a.src_f32 ? pack_load<float2>(a, tile, src0, rows, cols, k_fast)
                   : pack_load<double2>(a, tile, src0, rows, cols, k_fast);
  else
    ok = a.src_f32 ? pack_load<float>(a, tile, src0, rows, cols, k_fast)
                   : pack_load<double>(a, tile, src0, rows, cols, k_fast);
  const int64_t base = (int64_t)b * a.rows_out * a.pitch;
  const int64_t r = (int64_t)g + (int64_t)(i0 + threadIdx.y) * a.rstep;
  const int k = k0 + 2 * threadIdx.x;
  if constexpr (ESZ == 2) {
    if (__syncthreads_and(ok)) {
      pack_rows<ESZ, MODE, true>(a, tile, base, rows, r, k);
      return;
    }
  } else {
    __syncthreads();
  }
  pack_rows<ESZ, MODE, false>(a, tile, base, rows, r, k);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's tensor-map encoder, fetched through the runtime so that the
// library does not link libcuda (it loads on machines without a driver)
static EncodeTiledFn encoder() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 3-D map (K', rows, batch) over a packed buffer of row pitch `pitch`; loads
// past K' read zeros
static bool make_map(CUtensorMap* tm, void* base, int esz, int64_t kext, int64_t pitch, int64_t rows, int64_t nb,
                     int box_rows) {
  EncodeTiledFn enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)kext, (cuuint64_t)rows, (cuuint64_t)nb};
  cuuint64_t strides[2] = {(cuuint64_t)(pitch * esz), (cuuint64_t)(pitch * esz * rows)};
  cuuint32_t box[3] = {(cuuint32_t)(KROW_BYTES / esz), (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

struct Plan {
  int esz, kstep;        // element size, elements per K row of a stage
  int modeA, modeB, out;
  int64_t KA;            // logical K' (after re/im concatenation)
  int64_t pitch;         // packed row pitch: K' rounded up to 16 bytes
  int64_t rowsA, rowsB;  // packed rows per batch
  int64_t nbA, nbB;      // packed batches
  size_t offAh, offAl, offBh, offBl, total;
};

static size_t al(size_t x) { return (x + 1023) & ~size_t(1023); }

static Plan make_plan(const GemmParams& p, int prec) {
  Plan q{};
  q.esz = prec == RENO_PREC_BF16X3 ? 2 : 4;
  q.kstep = KROW_BYTES / q.esz;
  const bool ac = p.A.is_complex, bc = p.B.is_complex;
  int64_t kf = 1;
  if (ac && bc) {
    // double the operand with fewer rows: its rows are re-used across the whole other side
    const bool dblA = (int64_t)p.M * (p.A.s_batch ? p.batch : 1) <= (int64_t)p.N * (p.B.s_batch ? p.batch : 1);
    if (dblA) {
      q.modeA = P_DBL_CPLX;
      q.modeB = P_CAT;
      q.out = OUT_ROWS_CPLX;
    } else {
      q.modeA = P_CAT;
      q.modeB = P_DBL_CPLX;
      q.out = OUT_COLS_CPLX;
    }
    kf = 2;
  } else if (bc) {
    q.modeA = P_REAL;
    q.modeB = P_DBL_SPLIT;
    q.out = OUT_COLS_CPLX;
  } else if (ac) {
    q.modeA = P_DBL_SPLIT;
    q.modeB = P_REAL;
    q.out = OUT_ROWS_CPLX;
  } else {
    q.modeA = P_REAL;
    q.modeB = P_REAL;
    q.out = OUT_REAL;
  }
  q.KA = kf * p.K;
  const int64_t align = 16 / q.esz;  // TMA row strides are 16-byte multiples
  q.pitch = ((q.KA + align - 1) / align) * align;
  q.rowsA = (q.modeA == P_DBL_CPLX || q.modeA == P_DBL_SPLIT) ? 2 * (int64_t)p.M : p.M;
  q.rowsB = (q.modeB == P_DBL_CPLX || q.modeB == P_DBL_SPLIT) ? 2 * (int64_t)p.N : p.N;
  q.nbA = p.A.s_batch ? p.batch : 1;
  q.nbB = p.B.s_batch ? p.batch : 1;
  const size_t sa = (size_t)q.rowsA * q.pitch * q.nbA * q.esz;
  const size_t sb = (size_t)q.rowsB * q.pitch * q.nbB * q.esz;
  q.offAh = 0;
  q.offAl = al(sa);
  q.offBh = q.offAl + al(sa);
  q.offBl = q.offBh + al(sb);
  q.total = q.offBl + al(sb);
  return q;
}

template <int ESZ>
static cudaError_t run_pack(const GemmOperand& op, int R, int K, int nb, int mode, const SplitRows& rs, void* hi,
                            void* lo, int64_t pitch, int64_t rows_out, cudaStream_t st) {
  PackArgs a;
  a.src = op.ptr;
  a.src_complex = op.is_complex;
  a.conj = op.conj;
  a.src_f32 = op.is_f32;
  a.s_k = op.s_k;
  a.s_b = op.s_batch;
  // row r = (r2 * D1 + r1) * D0 + r0; tiles run along the slowest index that has more than one value
  a.D0 = std::max(rs.D0, 1);
  const bool levels = rs.D0 > 0, two = levels && (int64_t)rs.D0 * std::max(rs.D1, 1) >= R;
  a.rstep = !levels ? 1 : two ? std::min(rs.D0, std::max(R, 1)) : rs.D0 * std::max(rs.D1, 1);
  a.s_g0 = levels ? op.s_outer : 0;
  a.s_g1 = levels && !two ? rs.s_r1 : 0;
  a.s_i = !levels ? op.s_outer : two ? rs.s_r1 : rs.s_r2;
  a.rtiles = (int)ceil_div(ceil_div(R, a.rstep), PACK_R);
  a.ktiles = (int)ceil_div(K, PACK_K);
  a.R = R;
  a.K = K;
  a.hi = hi;
  a.lo = lo;
  a.pitch = pitch;
  a.rows_out = rows_out;
  const int64_t blocks = (int64_t)a.ktiles * a.rtiles * a.rstep;
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  dim3 grid((unsigned)blocks, 1, (unsigned)nb);
  count_launch();
  switch (mode) {
    case P_REAL: pack_kernel<ESZ, P_REAL><<<grid, dim3(32, 8), 0, st>>>(a); break;
    case P_CAT: pack_kernel<ESZ, P_CAT><<<grid, dim3(32, 8), 0, st>>>(a); break;
    case P_DBL_CPLX: pack_kernel<ESZ, P_DBL_CPLX><<<grid, dim3(32, 8), 0, st>>>(a); break;
    default: pack_kernel<ESZ, P_DBL_SPLIT><<<grid, dim3(32, 8), 0, st>>>(a); break;
  }
  return cudaGetLastError();
}

static int inter_of(int modeA, int modeB) {
  if (modeA == P_DBL_CPLX || modeA == P_DBL_SPLIT) return 1;
  if (modeB == P_DBL_CPLX || modeB == P_DBL_SPLIT) return 2;
  return 0;
}

// C' = A' B'^T over packed operands; the epilogue writes FP64/FP32 C (c != null)
// or the next stage's packed operand (po != null)
template <int ESZ>
static cudaError_t launch_split(const SplitPacked& A, const SplitPacked& B, int M, int N, int batch,
                                const GemmParams* c, const SplitPackOut* po, cudaStream_t st) {
  CUtensorMap tAh, tAl, tBh, tBl;
  if (A.kext != B.kext) return cudaErrorInvalidValue;
  if (!make_map(&tAh, A.hi, ESZ, A.kext, A.pitch, A.rows, A.nb, BM) ||
      !make_map(&tAl, A.lo, ESZ, A.kext, A.pitch, A.rows, A.nb, BM) ||
      !make_map(&tBh, B.hi, ESZ, B.kext, B.pitch, B.rows, B.nb, BN) ||
      !make_map(&tBl, B.lo, ESZ, B.kext, B.pitch, B.rows, B.nb, BN))
    return cudaErrorInvalidValue;
  const int inter = inter_of(A.mode, B.mode);
  Epi epi{};
  epi.M = M;
  epi.N = N;
  epi.rows_p = (int)A.rows;
  epi.cols_p = (int)B.rows;
  if (po) {
    epi.mode = OUT_PACK;
    epi.phi = po->hi;
    epi.plo = po->lo;
    epi.s_b = po->s_b;
    epi.s_m1 = po->s_m1;
    epi.s_m0 = po->s_m0;
    epi.s_n1 = po->s_n1;
    epi.s_n0 = po->s_n0;
    epi.s_ri = po->s_ri;
    epi.Dm = po->Dm > 0 ? po->Dm : 1 << 30;
    epi.Dn = po->Dn > 0 ? po->Dn : 1 << 30;
    epi.inter = inter;
  } else {
    epi.mode = inter == 1 ? OUT_ROWS_CPLX : inter == 2 ? OUT_COLS_CPLX : OUT_REAL;
    epi.C = c->C;
    epi.sCm = c->sCm;
    epi.sCn = c->sCn;
    epi.sCb = c->sCb;
    epi.accumulate = c->accumulate;
    epi.c_f32 = c->c_f32;
  }
  const int64_t kstep = KROW_BYTES / ESZ;
  const int chunk_k = g_split_chunk_k.load(std::memory_order_relaxed);
  const int kc = chunk_k > 0 ? (int)std::max<int64_t>(1, chunk_k / (2 * kstep)) * 2 : 0;  // whole 128-byte rows
  static std::atomic<unsigned long long> smem_set{0}, smem_set_p{0};
  {
    cudaError_t e = kc > 0 ? smem_optin_once(split_gemm_kernel<ESZ, true>, SMEM_BYTES, smem_set_p)
                           : smem_optin_once(split_gemm_kernel<ESZ, false>, SMEM_BYTES, smem_set);
    if (e != cudaSuccess) return e;
  }
  const int64_t mt = ceil_div(A.rows, BM), nt = ceil_div(B.rows, BN);
  // walk the smaller operand's tiles fastest (packed rows per batch decide)
  const int m_fast = (A.rows <= B.rows && mt > 1) ? 1 : 0;
  const int64_t ntiles = mt * nt * (int64_t)batch;
  if (ntiles > 0x7fffffff) return cudaErrorInvalidValue;
  const int sms = sm_count_current_device();
  const int grid = (int)std::min<int64_t>(ntiles, sms);  // one persistent CTA per SM
  count_launch();
  const uint64_t wait_ns = g_wait_ns.load(std::memory_order_relaxed);
  const int skip = g_skip_split_stage.exchange(-1);
  const int nkt = (int)ceil_div(A.kext, kstep);
  if (kc > 0)
    split_gemm_kernel<ESZ, true><<<grid, THREADS, SMEM_BYTES, st>>>(
        tAh, tAl, tBh, tBl, epi, nkt, (int)A.kext, A.nb > 1 ? 1 : 0, B.nb > 1 ? 1 : 0, m_fast, (int)mt, (int)nt,
        (int)ntiles, wait_ns, skip, kc);
  else
    split_gemm_kernel<ESZ, false><<<grid, THREADS, SMEM_BYTES, st>>>(
        tAh, tAl, tBh, tBl, epi, nkt, (int)A.kext, A.nb > 1 ? 1 : 0, B.nb > 1 ? 1 : 0, m_fast, (int)mt, (int)nt,
        (int)ntiles, wait_ns, skip, 0);
  return cudaGetLastError();
}

template <int ESZ>
static cudaError_t run_split(const GemmParams& p, const Plan& q, char* ws, cudaStream_t st) {
  SplitPacked A{ws + q.offAh, ws + q.offAl, q.pitch, q.rowsA, q.nbA, q.KA, q.modeA};
  SplitPacked B{ws + q.offBh, ws + q.offBl, q.pitch, q.rowsB, q.nbB, q.KA, q.modeB};
  cudaError_t e = run_pack<ESZ>(p.A, p.M, p.K, (int)q.nbA, q.modeA, SplitRows{}, A.hi, A.lo, q.pitch, q.rowsA, st);
  if (e == cudaSuccess) e = run_pack<ESZ>(p.B, p.N, p.K, (int)q.nbB, q.modeB, SplitRows{}, B.hi, B.lo, q.pitch, q.rowsB, st);
  if (e != cudaSuccess) return e;
  return launch_split<ESZ>(A, B, p.M, p.N, p.batch, &p, nullptr, st);
}

}  // namespace split

size_t split_gemm_required_bytes(const GemmParams& p, int prec) {
  if (prec == RENO_PREC_FP64 || p.M <= 0 || p.N <= 0 || p.batch <= 0) return 0;
  return split::make_plan(p, prec).total;
}

size_t split_gemm_workspace_bytes(int64_t a_elems, int64_t b_elems) {
  // conservative: complex operands doubled and K-concatenated, hi+lo, 4-byte elements
  return (size_t)(8 * 4 * 2) * (size_t)(a_elems + b_elems) + (size_t)(64 << 20);
}

cudaError_t split_gemm(const GemmParams& p, int prec, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (p.M <= 0 || p.N <= 0 || p.batch <= 0) return cudaSuccess;
  if (p.K <= 0) return (p.A.is_f32 || p.B.is_f32 || p.c_f32) ? cudaErrorInvalidValue : gemm_fp64(p, st);
  const split::Plan q = split::make_plan(p, prec);
  if (q.total > ws_bytes || !ws) return cudaErrorInvalidValue;
  if (q.esz == 2) return split::run_split<2>(p, q, static_cast<char*>(ws), st);
  return split::run_split<4>(p, q, static_cast<char*>(ws), st);
}

int split_esz(int prec) { return prec == RENO_PREC_BF16X3 ? 2 : 4; }

int64_t split_pitch(int64_t kext, int prec) {
  const int64_t align = 16 / split_esz(prec);
  return ((kext + align - 1) / align) * align;
}

size_t split_packed_bytes(int64_t rows, int64_t kext, int64_t nb, int prec) {
  return 2 * split::al((size_t)rows * split_pitch(kext, prec) * nb * split_esz(prec));
}

SplitPacked split_packed_at(void* base, int64_t rows, int64_t kext, int64_t nb, int mode, int prec) {
  const size_t plane = split::al((size_t)rows * split_pitch(kext, prec) * nb * split_esz(prec));
  return SplitPacked{base, static_cast<char*>(base) + plane, split_pitch(kext, prec), rows, nb, kext, mode};
}

cudaError_t split_pack(const GemmOperand& op, int R, int K, int nb, const SplitRows& rs, const SplitPacked& dst,
                       int prec, cudaStream_t st) {
  if (R <= 0 || K <= 0 || nb <= 0) return cudaSuccess;
  if (split_esz(prec) == 2)
    return split::run_pack<2>(op, R, K, nb, dst.mode, rs, dst.hi, dst.lo, dst.pitch, dst.rows, st);
  return split::run_pack<4>(op, R, K, nb, dst.mode, rs, dst.hi, dst.lo, dst.pitch, dst.rows, st);
}

cudaError_t split_run(const SplitPacked& A, const SplitPacked& B, int M, int N, int batch, const GemmParams* c,
                      const SplitPackOut* po, int prec, cudaStream_t st) {
  if (M <= 0 || N <= 0 || batch <= 0) return cudaSuccess;
  if ((c == nullptr) == (po == nullptr)) return cudaErrorInvalidValue;
  if (split_esz(prec) == 2) return split::launch_split<2>(A, B, M, N, batch, c, po, st);
  return split::launch_split<4>(A, B, M, N, batch, c, po, st);
}

int split_gemm_take_error() {
  int h = 0;
  cudaMemcpyFromSymbol(&h, split::g_split_error, sizeof(int));
  if (h) {
    int z = 0;
    cudaMemcpyToSymbol(split::g_split_error, &z, sizeof(int));
  }
  return h;
}

}  // namespace reno
