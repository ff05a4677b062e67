// Float64 GEMM on the tensor cores (tcgen05) by residue arithmetic.
//
// The dense products of the float64 path -- sampling a dense interface block
// (matAssembly/HBS/HBSnew.py:211-227), the Schur complements, pivot-block
// inverses and block products of the red-black and Thomas eliminations
// (direct_solve/omsdirectsolve.py:89-94, 238-277, 316-324) -- are bound by
// GB300's float64 pipe (2 FMA per clock and SM, ~1.05 TFLOP/s measured).
// Here such a product runs as 16 bfloat16 products on the tensor cores whose
// results are exact, after the method published as "Ozaki scheme II"
// (K. Ozaki, Y. Uchino, T. Imamura, 2025): scale each row of op(A) and each
// column of op(B) to t-bit integers, multiply modulo pairwise coprime
// moduli, and rebuild the integer product by the Chinese remainder theorem.
//
//   1. crt_convert_kernel: row r of op(A) (column of op(B)) with largest
//      exponent field F becomes the integers a' = rint(a 2^(t - F + 1022)),
//      |a'| <= 2^t, and their balanced residues modulo p_0 .. p_15, |r| <=
//      128: exact in bfloat16.  B's residues carry the factor (P/p)^-1 mod p
//      of the reconstruction.
//      A seventeenth plane holds the magnitudes |a| / a in bfloat16.
//   2. crt_gemm_kernel: per modulus a bfloat16 GEMM with float32 accumulation
//      in TMEM.  The sum of 1024 products of two residues is at most 2^24,
//      so every accumulator holds the exact integer; deeper products are
//      drained every 960 terms.  The epilogue reduces each sum modulo p and
//      stores it as one byte.
//   3. crt_combine_kernel: X = sum_l y_l P/p_l - k P as a 128-bit integer
//      (byte dot products, __dp4a), rounded once to float64, scaled by the
//      row and column powers of two, then alpha and beta.
//
// With t = (123 - log2 K) / 2 (56 at K = 1024) the only errors are the
// rounding of the inputs at 2^-(t+1) of their row's (column's) largest entry
// and the final rounding; a float64 FMA chain rounds once per term.  So the
// error of an output is at most K 2^-t a b, a the largest entry of its row of
// op(A), b of its column of op(B), where that of an FMA chain is K 2^-53 times
// its own sum s of |a_ik| |b_kj|.  Where the scales of op(A) and op(B) oppose
// along k, s is far below a b (rows diag(d) R against diag(1/d) C).  One more
// bfloat16 product, of the magnitudes |a_ik| / a and |b_kj| / b, gives s / (a b)
// (the terms rounded down by at most 2^-6), and step 3 forms an output by a
// float64 dot product instead
//   * where it is below 2^(51-t) everywhere in the output's row or everywhere
//     in its column: no output there would be as accurate as an FMA chain's to
//     within a factor of four, and
//   * where it is below 2^-44 for the output itself.
// Elsewhere the error is below 4 K 2^-53 times the largest s of the row and of
// the column, both scaled by the columns' b and the rows' a: a normwise bound
// that no scaling of rows, columns or k can spoil.  (An output whose own s is
// small beside the others of both its row and its column has fewer right digits
// than an FMA chain's, down to a few at 2^-44.)
// Rows or columns that hold an infinity or a NaN take the dot products too,
// with the float64 kernel's result.
//
// Work per element of A and B: 16 residues at ~9 integer / float32 slots and
// the magnitude; per element of C: 17 x 2K bfloat16 flops, 17 bytes and ~220
// slots of step 3.  Four 1024^3 products: 78 us of conversion, 123 of products
// (1.2 PFLOP/s on the tensor cores) and 43 of reconstruction (80, 116 and 40
// without the magnitudes), against 7.2 ms on the float64 pipe; with operands of
// which every output is a dot product 8.0 ms.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <numeric>

#include "crt.cuh"
#include "hbs.cuh"

namespace slu {
namespace {

using namespace crt;

// ---------------------------------------------------------------- conversion
struct CrtOperand {
  const double* x;
  int ld;
  long long s0, s1;
  int rows;              // rows of op(A), columns of op(B)
  int kcontig;           // consecutive k adjacent in memory
  __nv_bfloat16* out;    // residues [modulus][batch][row][Kp], magnitudes behind them
  int* ex;               // exponent field per [batch][row]; 2047 = not finite
  int* wide;             // zeroed here: see CrtGemm
};

// |v| / 2^(F - 1022) as a bfloat16, rounded down, in the upper half of a word
// (F: the row's largest exponent field); what is below 2^-60 as 2^-60, zero as
// zero.  sub = (max(F, 187) - 126) << 20: in rows all below 2^-836 (their
// subnormals have no exponent to subtract from) everything counts as small, and
// the row takes float64 dot products.
__device__ __forceinline__ uint32_t magnitude(uint2 v, int sub) {
  const uint32_t h = v.y & 0x7fffffffu;
  return (h | v.x) ? (uint32_t)max((int)h - sub, 67 << 20) << 3 : 0u;
}

// A CTA converts ROWS rows, 2048 / ROWS consecutive k at a time (32, 16 or 8
// rows, so that operands 64 or 128 deep keep every thread busy), through
// shared memory, which also turns k-strided operands around.  Eight k per
// thread and modulus: 16-byte stores.  One chunk: the exponents come from the
// staged values; more: one pass over the rows before.  ~190 instructions per
// element; 4 M elements (two 1024 x 1024 pairs): 42 us; 128 x (64 + 261) rows
// of 64: 29 us (88 with 8 rows per CTA, which leaves most threads idle).
template <int ROWS>
__global__ void __launch_bounds__(256, 2)
crt_convert_kernel(CrtOperand a, CrtOperand b, int strips_a, int K, int Kp, int t, int batch0,
                   int batch) {
  constexpr int KC = 2048 / ROWS, G = KC / 8;   // k per chunk; threads per row
  constexpr int P = KC + KC / 8 + 1;            // a pad every 8 values, rows one bank apart
  __shared__ uint2 tile[ROWS * P];
  __shared__ int s_ex[ROWS];
  const bool second = (int)blockIdx.x >= strips_a;
  const CrtOperand& o = second ? b : a;
  const int r0 = (second ? blockIdx.x - strips_a : blockIdx.x) * ROWS;
  const int bt = blockIdx.y, b0 = bt % batch0, b1 = bt / batch0;
  const uint2* x = reinterpret_cast<const uint2*>(o.x + b0 * o.s0 + b1 * o.s1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nr = min(ROWS, o.rows - r0);
  const bool single = Kp <= KC;
  if (!single) {
    // exponent field of every row (ROWS = 8 here: one warp per row)
    if (tid < ROWS) s_ex[tid] = 0;
    __syncthreads();
    if (o.kcontig) {
      for (int r = warp; r < nr; r += 8) {
        const uint2* row = x + (long long)(r0 + r) * o.ld;
        int f = 0;
        for (int k = lane; k < K; k += 32) f = max(f, (int)(row[k].y & 0x7fffffffu));
        f = __reduce_max_sync(0xffffffffu, f);
        if (lane == 0) s_ex[r] = f >> 20;
      }
    } else {
      const int r = tid % ROWS;
      if (r < nr) {
        const uint2* col = x + r0 + r;
        int f = 0;
        for (int k = tid / ROWS; k < K; k += 256 / ROWS)
          f = max(f, (int)(col[(long long)k * o.ld].y & 0x7fffffffu));
        atomicMax(&s_ex[r], f >> 20);
      }
    }
  }
  const int row = tid / G, kq = tid % G;
  const bool live = row < nr;
  const long long plane = (long long)batch * o.rows * Kp;
  __nv_bfloat16* dst = o.out + ((long long)bt * o.rows + r0 + row) * Kp + 8 * kq;
  for (int kc = 0; kc < Kp; kc += KC) {
    const int kn = min(KC, K - kc);   // may be <= 0 in the padding
    __syncthreads();
    // eight values per thread, all loads before the first store
    uint2 v[8];
    if (o.kcontig) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid + 256 * i) / KC, k = (tid + 256 * i) % KC;
        v[i] = (r < nr && k < kn) ? x[(long long)(r0 + r) * o.ld + kc + k] : make_uint2(0, 0);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid + 256 * i) / KC, k = (tid + 256 * i) % KC;
        tile[r * P + k + (k >> 3)] = v[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = tid % ROWS, k = (tid + 256 * i) / ROWS;
        v[i] = (r < nr && k < kn) ? x[(long long)(kc + k) * o.ld + r0 + r] : make_uint2(0, 0);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = tid % ROWS, k = (tid + 256 * i) / ROWS;
        tile[r * P + k + (k >> 3)] = v[i];
      }
    }
    __syncthreads();
    const uint2* src = tile + row * P + 9 * kq;
    int ex;
    if (single) {
      ex = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) ex = max(ex, (int)((src[u].y >> 20) & 0x7ff));
#pragma unroll
      for (int s = G / 2; s > 0; s >>= 1) ex = max(ex, __shfl_xor_sync(0xffffffffu, ex, s));
    } else {
      ex = s_ex[row];
    }
    if (kc == 0 && kq == 0 && live) {
      o.ex[(long long)bt * o.rows + r0 + row] = ex;
      o.wide[(long long)bt * o.rows + r0 + row] = 0;
    }
    if (!live || kc + 8 * kq >= Kp) continue;
    {
      // (not finite: dot products; the others' rows and columns are not to count on it)
      const int sub = ex == 0x7ff ? 0x7fffffff : (max(ex, 187) - 126) << 20;
      uint32_t w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        w[u] = __byte_perm(magnitude(src[2 * u], sub), magnitude(src[2 * u + 1], sub), 0x7632);
      *reinterpret_cast<uint4*>(dst + NM * plane + kc) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      scaled(src[u].y, src[u].x, max(ex, 1), t, ex != 0x7ff, lo[u], hi[u]);
#pragma unroll
    for (int l = 0; l < NM; ++l) {
      const uint32_t c0 = second ? c_tab.cb[0][l] : c_tab.ca[0][l];
      const uint32_t c1 = second ? c_tab.cb[1][l] : c_tab.ca[1][l];
      const int bias = 0x4B400000 + (second ? c_tab.bb[l] : c_tab.ba[l]);
      const float p = c_tab.pf[l], ip = c_tab.inv[l];
      uint32_t w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        w[u] = pack_bf16(residue(lo[2 * u], hi[2 * u], c0, c1, bias, p, ip),
                         residue(lo[2 * u + 1], hi[2 * u + 1], c0, c1, bias, p, ip));
      *reinterpret_cast<uint4*>(dst + l * plane + kc) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// ---------------------------------------------------------------- tcgen05 GEMM
constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (kEpiWarps + 2);   // warps 0-7 epilogue, 8 TMA, 9 MMA
constexpr int kMaxStages = 8;
constexpr int kRing = 208 * 1024;
constexpr long long kWaitLimit = 1LL << 22;
constexpr int kTmemCols = 512;                   // two accumulators of up to 256 columns
constexpr int kChunkOne = 16, kChunkMany = 15;   // k-tiles per exact float32 sum

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait for the phase with the given parity; gives up early once
// another role has.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
  const uint32_t addr = smem_u32(bar);
  for (long long i = 0; i < kWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (fail && *fail) return false;
  }
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// K-major, 128B swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// Exponent field of the smallest magnitude sum (beside the operands' largest
// entries) that an output may have.
constexpr uint32_t kSumFloor = 127 - 44;

struct CrtGemm {
  int M, N, batch;
  int tm, tn;            // tiles
  int BN;                // tile columns, a multiple of 16, at most 256
  int KT, chunks, per;   // k-tiles; chunks of `per` k-tiles
  int stages;
  long long items;       // (NM + 1) * batch * tm * tn
  int8_t* R;             // residues [modulus][batch][M][pitch], then the
                         // exponent field of every magnitude sum (0: zero,
                         // every product has a zero factor)
  float theta;           // 2^(51 - t)
  int *wa, *wb;          // rows and columns with a sum of theta or more
  int pitch;
  volatile unsigned* err;
};

// Persistent: each CTA runs every gridDim-th (modulus, batch, tile) item.
//   warp 8: TMA into a ring of (A 128 x 64, B BN x 64) slabs
//   warp 9: tcgen05.mma, the items' chunks alternating between the two TMEM
//           accumulators
//   warps 0-7: drain the other accumulator meanwhile (lanes 32 (w % 4) ..,
//           columns of half w / 4): reduce modulo p, pack, 16-byte stores
// Tiles of 128 x up to 256 columns: a smaller one doubles the operand
// traffic per flop, and 256 is the widest the instruction takes.
__global__ void __maxnreg__(168)
crt_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CrtGemm g) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
  __shared__ __align__(8) uint64_t ready_bar[2];
  __shared__ __align__(8) uint64_t drained_bar[2];
  __shared__ __align__(8) uint64_t quiet_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_fail;
  __shared__ volatile long long s_issued;
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.stages, BN = g.BN;
  const uint32_t stage_bytes = A_BYTES + BN * BK * 2;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&ready_bar[a], 1);
      mbar_init(&drained_bar[a], 32 * kEpiWarps);
    }
    mbar_init(&quiet_bar, 1);
    s_fail = 0;
    s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int tiles = g.tm * g.tn;

  if (warp == kEpiWarps) {
    if (lane == 0) {
      long long it = 0;
      bool ok = true;
      for (long long id = blockIdx.x; id < g.items && ok; id += gridDim.x) {
        const long long mb = id / tiles;              // modulus * batch + batch index
        const int tile = (int)(id - mb * tiles);
        const int m0 = (tile / g.tn) * BM, n0 = (tile % g.tn) * BN;
        const int ya = (int)(mb * g.M) + m0, yb = (int)(mb * g.N) + n0;
        for (int kt = 0; kt < g.KT; ++kt, ++it) {
          const int s = (int)(it % S);
          if (it >= S && !mbar_wait(&empty_bar[s], (uint32_t)((it / S) + 1) & 1, &s_fail)) {
            s_fail = 1;
            ok = false;
            break;
          }
          unsigned char* a = smem + s * stage_bytes;
          mbar_expect_tx(&full_bar[s], stage_bytes);
          tma_load_2d(a, &tmA, kt * BK, ya, &full_bar[s]);
          tma_load_2d(a + A_BYTES, &tmB, kt * BK, yb, &full_bar[s]);
          s_issued = it + 1;
        }
      }
    }
  } else if (warp == kEpiWarps + 1) {
    if (lane == 0) {
      // kind::f16: D f32, A/B bf16, both K-major, M = 128, N = BN
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
      long long it = 0;
      uint32_t n = 0;   // chunks issued
      bool ok = true;
      for (long long id = blockIdx.x; id < g.items && ok; id += gridDim.x) {
        int kt = 0;
        for (int c = 0; c < g.chunks && ok; ++c, ++n) {
          const uint32_t a = n & 1;
          if (n >= 2 && !mbar_wait(&drained_bar[a], ((n >> 1) - 1) & 1, &s_fail)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t dacc = tmem + a * 256;
          const int kend = min(kt + g.per, g.KT);
          for (int j = 0; kt < kend; ++j, ++kt, ++it) {
            const int s = (int)(it % S);
            if (!mbar_wait(&full_bar[s], (uint32_t)(it / S) & 1, &s_fail)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(smem + s * stage_bytes), sb = sa + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              mma_bf16(dacc, smem_desc(sa + kk * 32), smem_desc(sb + kk * 32), idesc,
                       (j | kk) != 0);
            mma_commit(&empty_bar[s]);
          }
          if (ok) mma_commit(&ready_bar[a]);
        }
      }
      if (!ok) s_fail = 1;
      // every MMA issued has finished before TMEM and the ring are given up
      mma_commit(&quiet_bar);
      mbar_wait(&quiet_bar, 0, nullptr);
    }
  } else {
    const int q = warp & 3, half = warp >> 2;
    const int groups = BN / 16, g0 = half ? (groups + 1) / 2 : 0, g1 = half ? groups : (groups + 1) / 2;
    const uint32_t lanes = (uint32_t)(q * 32) << 16;
    uint32_t n = 0;
    bool ok = true;
    for (long long id = blockIdx.x; id < g.items && ok; id += gridDim.x) {
      const long long mb = id / tiles;
      const int tile = (int)(id - mb * tiles), l = (int)(mb / g.batch);
      const int row = (tile / g.tn) * BM + q * 32 + lane, n0 = (tile % g.tn) * BN;
      const bool mags = l == NM;
      const float p = mags ? 0.f : c_tab.pf[l], ip = mags ? 0.f : c_tab.inv[l];
      const long long bt = mb - (long long)l * g.batch;
      int8_t* out = g.R + (mb * g.M + row) * g.pitch + n0;
      for (int c = 0; c < g.chunks; ++c, ++n) {
        const uint32_t a = n & 1;
        ok = mbar_wait(&ready_bar[a], (n >> 1) & 1, &s_fail);
        if (!__all_sync(0xffffffffu, ok)) {   // warp-uniform: the loads below are collective
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int j = g0; j < g1; ++j) {
          uint32_t v[16];
          tmem_ld16(tmem + lanes + a * 256 + 16 * j, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (mags) {
            if (n0 + 16 * j >= g.pitch) continue;   // uniform
            uint32_t w[4], wide = 0;
#pragma unroll
            for (int e = 0; e < 16; ++e)
              wide |= (__uint_as_float(v[e]) >= g.theta ? 1u : 0u) << e;
#pragma unroll
            for (int e = 0; e < 16; e += 4)
              w[e >> 2] = __byte_perm(__byte_perm(v[e] << 1, v[e + 1] << 1, 0x73),
                                      __byte_perm(v[e + 2] << 1, v[e + 3] << 1, 0x73), 0x5410);
            const int nc = min(16, g.N - n0 - 16 * j);
            wide &= row < g.M && nc > 0 ? 0xffffu >> (16 - nc) : 0u;
            const uint32_t cols = __reduce_or_sync(0xffffffffu, wide);
            if (cols >> lane & 1) g.wb[bt * g.N + n0 + 16 * j + lane] = 1;
            if (row < g.M) {
              if (wide) g.wa[bt * g.M + row] = 1;
              uint4* dst = reinterpret_cast<uint4*>(out + 16 * j);
              if (c > 0) {   // the largest of the chunks
                const uint4 o = *dst;
                w[0] = __vmaxu4(w[0], o.x);
                w[1] = __vmaxu4(w[1], o.y);
                w[2] = __vmaxu4(w[2], o.z);
                w[3] = __vmaxu4(w[3], o.w);
              }
              *dst = make_uint4(w[0], w[1], w[2], w[3]);
            }
          } else if (row < g.M && n0 + 16 * j < g.pitch) {
            uint4* dst = reinterpret_cast<uint4*>(out + 16 * j);
            uint32_t old[4] = {0, 0, 0, 0};
            if (c > 0) {
              const uint4 o = *dst;
              old[0] = o.x; old[1] = o.y; old[2] = o.z; old[3] = o.w;
            }
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float x = __uint_as_float(v[e]);
              if (c > 0) x += (float)(int8_t)(old[e >> 2] >> (8 * (e & 3)));
              const uint32_t y = reduced(x, p, ip) & 0xffu;
              w[e >> 2] = (e & 3) ? w[e >> 2] | (y << (8 * (e & 3))) : y;
            }
            *dst = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&drained_bar[a]);
      }
    }
    if (!ok) {
      s_fail = 1;
      if (lane == 0 && g.err) *g.err = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) {
    // the copies already issued land before the CTA exits
    if (g.err) *g.err = 1;
    const long long issued = s_issued;
    for (long long j = issued > S ? issued - S : 0; j < issued; ++j)
      mbar_wait(&full_bar[j % S], (uint32_t)(j / S) & 1, nullptr);
  }
  __syncthreads();
  if (warp == kEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
}

// ---------------------------------------------------------------- reconstruction
struct CrtCombine {
  int M, N, K, batch0, batch;
  const int8_t* R;
  int pitch;
  const int *ea, *eb;
  const int *wa, *wb;     // see CrtGemm
  int t;
  double alpha, beta;
  int kind;   // alpha, beta: 0 = 1, 0; 1 = -1, 0; 2 = 1, 1; 3 = -1, 1; 4 = any (a float64 compare
              // costs as much as 30 integer instructions)
  double* C;
  int ldc;
  long long sC0, sC1;
  // operands, for rows and columns that are not finite
  const double *A, *B;
  long long ak, ai, sA0, sA1, bk, bj, sB0, sB1;   // strides along k, i, j
};

__device__ __forceinline__ void put(const CrtCombine& g, double* c, double v) {
  if (g.kind == 4) {
    v *= g.alpha;
    if (g.beta != 0.0) v = fma(g.beta, *c, v);
  } else {
    if (g.kind & 1) v = __hiloint2double((int)(hi32(v) ^ 0x80000000u), __double2loint(v));
    if (g.kind & 2) v = *c + v;
  }
  *c = v;
}

// One thread per four consecutive elements of a row of C: four bytes of every
// residue plane, transposed in registers so a __dp4a sums four moduli.  Eight
// threads take a segment of 32 outputs (a sector of every plane), a CTA every
// gridDim-th segment.  The outputs that take a dot product go to a list and are
// spread over the CTA, eight lanes each.  They come as whole rows, columns or
// corners, and a CTA forms 1024 of them in 300 us (depth 1024, float64 pipe): so
// the grid has no factor in common with the segments of a row, and they fall
// to all CTAs alike.
__global__ void __launch_bounds__(256)
crt_combine_kernel(const __grid_constant__ CrtCombine g) {
  __shared__ unsigned short list[1024];   // 32 segment + column
  __shared__ int listed;
  const int tid = threadIdx.x, tn = (g.N + 31) / 32;
  const long long segs = (long long)g.batch * g.M * tn, T = gridDim.x;
  const long long plane = (long long)g.batch * g.M * g.pitch;
  if (tid == 0) listed = 0;
  for (long long s0 = blockIdx.x; s0 < segs; s0 += 32 * T) {
    const long long sg = s0 + (tid >> 3) * T;
    const long long br = sg / tn;   // batch * M + row
    const int j0 = 32 * (int)(sg - br * tn) + 4 * (tid & 7);
    uint32_t bad = 0;
    if (sg < segs && j0 < g.N) {
      const int bt = (int)(br / g.M), i = (int)(br - (long long)bt * g.M);
      const int b0 = bt % g.batch0, b1 = bt / g.batch0;
      const int8_t* src = g.R + br * g.pitch + j0;
      uint32_t r[NM];
#pragma unroll
      for (int l = 0; l < NM; ++l) r[l] = *reinterpret_cast<const uint32_t*>(src + l * plane);
      const uint32_t sums = *reinterpret_cast<const uint32_t*>(src + NM * plane);
      // r[4 a + e] <- byte e of planes 4 a .. 4 a + 3
#pragma unroll
      for (int a = 0; a < NM; a += 4) {
        const uint32_t x0 = __byte_perm(r[a], r[a + 1], 0x5140), x1 = __byte_perm(r[a], r[a + 1], 0x7362);
        const uint32_t y0 = __byte_perm(r[a + 2], r[a + 3], 0x5140), y1 = __byte_perm(r[a + 2], r[a + 3], 0x7362);
        r[a] = __byte_perm(x0, y0, 0x5410);
        r[a + 1] = __byte_perm(x0, y0, 0x7632);
        r[a + 2] = __byte_perm(x1, y1, 0x5410);
        r[a + 3] = __byte_perm(x1, y1, 0x7632);
      }
      const int fa = g.ea[br];
      const bool wide = g.wa[br] != 0;
      double* c = g.C + b0 * g.sC0 + b1 * g.sC1 + (long long)i * g.ldc + j0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (j0 + e >= g.N) break;
        const long long jb = (long long)bt * g.N + j0 + e;
        const int fb = g.eb[jb];
        const uint32_t s = sums >> (8 * e) & 0xff;
        if (fa == 0x7ff || fb == 0x7ff || (s && (s < kSumFloor || !(wide && g.wb[jb])))) {
          bad |= 1u << e;
        } else {
          put(g, c + e, combine(r[e], r[4 + e], r[8 + e], r[12 + e],
                                max(fa, 1) + max(fb, 1) - 2 * (1022 + g.t)));
        }
      }
    }
    if (!__syncthreads_or(bad)) continue;
    if (bad) {
      int at = atomicAdd(&listed, __popc(bad));
      for (; bad; bad &= bad - 1) list[at++] = (unsigned short)(4 * tid + __ffs(bad) - 1);
    }
    __syncthreads();
    const int n = listed;
    for (int x0 = 0; x0 < n; x0 += 32) {
      const int x = x0 + (tid >> 3), el = list[min(x, n - 1)];
      const long long sl = s0 + (el >> 5) * T, br = sl / tn;
      const int j = 32 * (int)(sl - br * tn) + (el & 31), bt = (int)(br / g.M);
      const int i = (int)(br - (long long)bt * g.M), b0 = bt % g.batch0, b1 = bt / g.batch0;
      const double* ap = g.A + b0 * g.sA0 + b1 * g.sA1 + i * g.ai;
      const double* bp = g.B + b0 * g.sB0 + b1 * g.sB1 + j * g.bj;
      double v = 0.0;
#pragma unroll 8
      for (int k = tid & 7; k < g.K; k += 8) v = fma(ap[k * g.ak], bp[k * g.bk], v);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (x < n && (tid & 7) == 0)
        put(g, g.C + b0 * g.sC0 + b1 * g.sC1 + (long long)i * g.ldc + j, v);
    }
    __syncthreads();
    if (tid == 0) listed = 0;
  }
}

// ---------------------------------------------------------------- host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  if (!fn) throw Error(SLU_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  return fn;
}

CUtensorMap residue_map(const void* base, long long rows, int Kp, int box_rows) {
  CUtensorMap m;
  cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Kp * 2};
  cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                           strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(SLU_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return m;
}

size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Workspace of one launch set (residues and magnitudes of A and B, result
// residues and sums, exponents and largest sums).
size_t crt_bytes(int M, int N, int K, long long nb) {
  const size_t Kp = up(K, BK), pitch = up(N, 16);
  return up((size_t)2 * (NM + 1) * nb * M * Kp, 1024) + up((size_t)2 * (NM + 1) * nb * N * Kp, 1024) +
         up((size_t)(NM + 1) * nb * M * pitch, 1024) + up((size_t)8 * nb * (M + N), 1024) + 4096;
}

// Larger products than the handle's scratch limit allows run in pieces (deeper
// ones in slices of kDepthMax, accumulated in C).
constexpr size_t kWsMax = Handle::kScratchMax;
constexpr int kDepthMax = 8192;

struct Operand {
  const double* x;
  int ld;
  bool trans;
  long long s0, s1;
};

void crt_piece(Handle& h, int M, int N, int K, double alpha, const Operand& A, const Operand& B,
               double beta, double* C, int ldc, long long sC0, long long sC1, int batch0,
               int batch) {
  cudaStream_t st = h.stream;
  const int Kp = (int)up(K, BK), pitch = (int)up(N, 16), t = bits_for(K);
  Scratch scratch(h.gemm_ws, st);
  Workspace& ws = scratch.w;
  ws.reserve(crt_bytes(M, N, K, batch), st);
  constexpr size_t NP = NM + 1;   // planes: residues and magnitudes
  auto* ra = ws.take<__nv_bfloat16>(NP * batch * M * Kp);
  auto* rb = ws.take<__nv_bfloat16>(NP * batch * N * Kp);
  auto* R = ws.take<int8_t>(NP * batch * M * pitch);
  int* ea = ws.take<int>((size_t)batch * M);
  int* eb = ws.take<int>((size_t)batch * N);
  int* wa = ws.take<int>((size_t)batch * M);
  int* wb = ws.take<int>((size_t)batch * N);
  const CrtOperand oa{A.x, A.ld, A.s0, A.s1, M, !A.trans, ra, ea, wa};
  const CrtOperand ob{B.x, B.ld, B.s0, B.s1, N, B.trans, rb, eb, wb};
  auto convert = [&](auto kern, int rows) {
    const int sa = (M + rows - 1) / rows, sb = (N + rows - 1) / rows;
    kern<<<dim3(sa + sb, batch), 256, 0, st>>>(oa, ob, sa, K, Kp, t, batch0, batch);
    check_launch("crt_convert_kernel");
  };
  if (Kp <= 64) convert(crt_convert_kernel<32>, 32);
  else if (Kp <= 128) convert(crt_convert_kernel<16>, 16);
  else convert(crt_convert_kernel<8>, 8);
  CrtGemm g{};
  g.M = M;
  g.N = N;
  g.batch = batch;
  g.tm = (M + BM - 1) / BM;
  // widest tiles that still give every SM an item, evenly over the columns
  g.tn = (N + 255) / 256;
  while ((long long)NP * batch * g.tm * g.tn < num_sms() && (N + g.tn - 1) / g.tn > 64) ++g.tn;
  g.BN = (int)up((N + g.tn - 1) / g.tn, 16);
  g.tn = (N + g.BN - 1) / g.BN;
  g.KT = Kp / BK;
  g.chunks = g.KT <= kChunkOne ? 1 : (g.KT + kChunkMany - 1) / kChunkMany;
  g.per = (g.KT + g.chunks - 1) / g.chunks;
  g.stages = std::min(kMaxStages, kRing / (A_BYTES + g.BN * BK * 2));
  g.items = (long long)NP * batch * g.tm * g.tn;
  g.R = R;
  g.theta = std::ldexp(1.0f, 51 - t);
  g.wa = wa;
  g.wb = wb;
  g.pitch = pitch;
  g.err = h.err_word();
  const CUtensorMap ma = residue_map(ra, (long long)NP * batch * M, Kp, BM);
  const CUtensorMap mb = residue_map(rb, (long long)NP * batch * N, Kp, g.BN);
  const size_t sm = (size_t)g.stages * (A_BYTES + g.BN * BK * 2) + 1024;
  ensure_smem(reinterpret_cast<const void*>(crt_gemm_kernel), sm);
  crt_gemm_kernel<<<(unsigned)std::min<long long>(g.items, num_sms()), kThreads, sm, st>>>(ma, mb,
                                                                                           g);
  check_launch("crt_gemm_kernel");
  CrtCombine c{};
  c.M = M;
  c.N = N;
  c.K = K;
  c.batch0 = batch0;
  c.batch = batch;
  c.R = R;
  c.pitch = pitch;
  c.ea = ea;
  c.eb = eb;
  c.wa = wa;
  c.wb = wb;
  c.t = t;
  c.alpha = alpha;
  c.beta = beta;
  c.kind = (alpha != 1.0 && alpha != -1.0) || (beta != 0.0 && beta != 1.0)
               ? 4
               : (alpha == -1.0 ? 1 : 0) + (beta == 1.0 ? 2 : 0);
  c.C = C;
  c.ldc = ldc;
  c.sC0 = sC0;
  c.sC1 = sC1;
  c.A = A.x;
  c.ak = A.trans ? A.ld : 1;
  c.ai = A.trans ? 1 : A.ld;
  c.sA0 = A.s0;
  c.sA1 = A.s1;
  c.B = B.x;
  c.bk = B.trans ? 1 : B.ld;
  c.bj = B.trans ? B.ld : 1;
  c.sB0 = B.s0;
  c.sB1 = B.s1;
  const int tn = (N + 31) / 32;
  long long ctas = std::min(((long long)batch * M * tn + 31) / 32, 32LL * num_sms());
  while (std::gcd(ctas, (long long)tn) != 1) ++ctas;
  crt_combine_kernel<<<(unsigned)ctas, 256, 0, st>>>(c);
  check_launch("crt_combine_kernel");
}

}  // namespace

void gemm_f64_tensor(Handle& h, bool ta, bool tb, int M, int N, int K, double alpha,
                     const double* A, int lda, long long sA0, long long sA1, const double* B,
                     int ldb, long long sB0, long long sB1, double beta, double* C, int ldc,
                     long long sC0, long long sC1, int batch0, int batch1) {
  if (M <= 0 || N <= 0 || batch0 <= 0 || batch1 <= 0) return;
  if (K > kDepthMax) {
    for (int k0 = 0; k0 < K; k0 += kDepthMax)
      gemm_f64_tensor(h, ta, tb, M, N, std::min(kDepthMax, K - k0), alpha,
                      A + (ta ? (long long)k0 * lda : (long long)k0), lda, sA0, sA1,
                      B + (tb ? (long long)k0 : (long long)k0 * ldb), ldb, sB0, sB1,
                      k0 ? 1.0 : beta, C, ldc, sC0, sC1, batch0, batch1);
    return;
  }
  // pieces of at most kWsMax workspace: rows and columns halved (each half a
  // multiple of a tile) until one matrix fits, then as many matrices as fit
  int Mp = M, Np = N;
  while (crt_bytes(Mp, Np, K, 1) > kWsMax && (Mp > 1024 || Np > 1024)) {
    if (Mp >= Np) Mp = (int)up((Mp + 1) / 2, 256);
    else Np = (int)up((Np + 1) / 2, 256);
  }
  long long fit = std::max<long long>(1, kWsMax / crt_bytes(Mp, Np, K, 1));
  fit = std::min<long long>(fit, 65535);
  // residue rows are indexed by 32-bit TMA coordinates
  fit = std::max<long long>(1, std::min(fit, (1LL << 30) / (NM + 1) / std::max(Mp, Np)));
  // pieces of about one size: whole rows of the batch, else parts of them
  auto even = [](long long n, long long most) {
    const long long pieces = (n + most - 1) / most;
    return (n + pieces - 1) / pieces;
  };
  const int n0 = (int)even(batch0, std::min<long long>(fit, batch0));
  const int n1 = n0 < batch0 ? 1 : (int)even(batch1, std::min<long long>(fit / n0, batch1));
  for (int i0 = 0; i0 < M; i0 += Mp)
    for (int j0 = 0; j0 < N; j0 += Np) {
      const int m = std::min(Mp, M - i0), n = std::min(Np, N - j0);
      const double* a = A + (ta ? (long long)i0 : (long long)i0 * lda);
      const double* b = B + (tb ? (long long)j0 * ldb : (long long)j0);
      double* c = C + (long long)i0 * ldc + j0;
      for (int q1 = 0; q1 < batch1; q1 += n1)
        for (int q0 = 0; q0 < batch0; q0 += n0) {
          const int c0 = std::min(n0, batch0 - q0), c1 = std::min(n1, batch1 - q1);
          crt_piece(h, m, n, K, alpha, {a + q0 * sA0 + q1 * sA1, lda, ta, sA0, sA1},
                    {b + q0 * sB0 + q1 * sB1, ldb, tb, sB0, sB1}, beta, c + q0 * sC0 + q1 * sC1, ldc,
                    sC0, sC1, c0, c0 * c1);
        }
    }
}

// Residue products pay where the float64 pipe is the bound: enough flops to
// cover three launches, and enough of them per element of C and of the
// operands to cover the conversions.  Products of 32 rows, 261 columns and
// depth 64: 8 of them 14 us in float64, 16 (1.7e7 flops) 22, 32 135 -> 33, 64
// 200 -> 49; 48 x 200 x 64, 32 of them 55 -> 29.
bool gemm_tensor_pays(int M, int N, int K, long long nb) {
  return M >= 32 && N >= 32 && K >= 64 && 2.0 * M * N * K * nb >= 2.0e7;
}

void gemm_f64(Handle& h, bool ta, bool tb, int M, int N, int K, double alpha, const double* A,
              int lda, long long sA0, long long sA1, const double* B, int ldb, long long sB0,
              long long sB1, double beta, double* C, int ldc, long long sC0, long long sC1,
              int batch0, int batch1) {
  if (batch0 > 0 && batch1 > 0 && gemm_tensor_pays(M, N, K, (long long)batch0 * batch1))
    gemm_f64_tensor(h, ta, tb, M, N, K, alpha, A, lda, sA0, sA1, B, ldb, sB0, sB1, beta, C, ldc,
                    sC0, sC1, batch0, batch1);
  else
    gemm_batched<double>(h.stream, ta, tb, M, N, K, alpha, A, lda, sA0, sA1, B, ldb, sB0, sB1,
                         beta, C, ldc, sC0, sC1, batch0, batch1);
}

}  // namespace slu
