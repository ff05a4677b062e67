// The tree steps of HBS solves and applies with many right-hand sides as exact
// residue products on the tensor cores, float64 in and out.
//
// The steps are those of the float64 step kernels (sweep.cuh, sweep_host.cuh;
// ULVsparse.solve, matAssembly/HBS/ULVsparse.py:296-353, and HBSMAT.matmat /
// rmatmat, matAssembly/HBS/HBSnew.py:308-350): out_b = S_b z_b per block.
// Those are bound by the float64 pipe, at 71-87% of it, so only another unit
// makes them faster.  Here a step is 16 bfloat16 products modulo the primes of
// crt.cuh, each exact in float32 (at most 128 terms of at most 2^14), and one
// reconstruction per output, rounded once: the error is that of rounding S and
// z to t = 58 or 59 bits of their row's and column's largest entry.  Where the
// columns of a block of S differ by more than 2^kSpread, they are scaled to one
// size by powers of two (kx, made with the images) and the entries of z that they
// meet by the inverse.  So each column of z meets, at its largest entry, an entry
// of S within 2^-kSpread of its row's largest: the error in a column of outputs,
// its rows scaled by those of S, is at most w 2^(kSpread - t), below w 2^-53,
// times the largest sum of |S| |z| there, where a float64 FMA chain's is w 2^-53
// of the output's own.  Outputs below 2^-44 of the row's and column's largest
// entries are formed by float64 dot products, so every output keeps 2^-14 of its
// own size.  (The steps of an operator whose couplings have singular values down
// to 1e-12 have many outputs at 2^-33: with the line at 2^-32 their dot products,
// 20-40K clocks each, took a solve of 1024 columns from 680 to 832 us; at 2^-22
// random cancellation alone, two or three outputs a step, added half to a solve of
// 261 columns.)
//
// One persistent kernel per step.  A tile is a block, up to 128 operator rows
// and 32, 16 or 8 columns (tiling_of: 16 moduli of 32 columns fill TMEM):
//   * S's residues are made once per factorisation (crt_op_kernel, on the first
//     call that uses them) as core-matrix images.  Warps 0-3 bring them into
//     shared memory by bulk copies, warp j moduli j, j + 4, ..: all sixteen
//     stay resident while a CTA's consecutive tiles share them where they fit
//     (64 x 64 blocks), else they stream through a ring of slots;
//   * the same four warps issue the MMAs, one lane each: one thread took 80-90
//     clocks per MMA, and 250-300 where one waits for the one before it in the
//     same accumulator; four warps with an accumulator each overlap them;
//   * 16 warps gather z (through up to three ranges and a permutation, the
//     next tile's values already in flight), find the column exponents, write
//     the residues a group of four or eight moduli at a time, and after the
//     last MMA read the 16 sums of each output, reduce, reconstruct and store.
//     Up to 64 rows go as MMAs of M = 64, whose rows lie in 16 lanes of every
//     quarter of TMEM: all four scheduler partitions reconstruct (with M = 128
//     two of them had nothing to do: 12K clocks a tile, now 4K).
// Everything but the MMAs is integer and float32 work, which bounds a tile:
// ~170 clocks per 32 elements of z and ~320 per 32 outputs on the integer
// pipe's half rate, against 64 w clocks of the float64 pipe per 32 outputs.  A
// tile of 64 x 64 x 32 takes 17K clocks where that work is 8K (the phases of a
// tile follow one another), the float64 pipe 66K.
// Measured (us, float64 steps -> these): 8192 rows with leaves of 64 and rank
// 32, 261 columns: solve 2100 -> 423, transposed 2017 -> 434, apply 1317 ->
// 381; 4096 rows, 64 columns: 252 -> 117, 275 -> 122, 180 -> 110 (the balanced
// columns and the look at small outputs 1-3% of it).  The relative
// error against 64 bits over those shapes: solves 1.2e-15 (float64 steps
// 1.2e-15), applies 1.1e-15 (1.1e-15): that of the operators, not of the steps.
// Columns or operator rows that are not finite take float64 dot products.
// Every mbarrier wait is bounded; on a timeout the kernel sets the caller's
// error word, lets its copies land, frees its TMEM and returns.
#include <algorithm>

#include "crt.cuh"
#include "hbs.cuh"
#include "sweep_host.cuh"

namespace slu {
namespace {

using namespace crt;

constexpr int kRows = 128;         // operator rows per tile (MMA M)
constexpr int kMaxW = 128;         // widest step
constexpr int kMma = 4;            // warps that copy operator images and issue MMAs
constexpr int kWarps = 16;         // compute warps, after them
constexpr int kThreads = 32 * (kMma + kWarps);
constexpr size_t kSmemMax = 224 * 1024;
constexpr long long kWaitLimit = 1LL << 22;

struct CrtStep {
  sweep::Step<double> s;     // geometry and vectors; s.S for what is not finite
  const __nv_bfloat16* img;  // [Nb][ntile][NM][RT x wP]
  const int* ex;             // exponent field of every row: [Nb][ntile * RT]
  const short* kx;           // powers of two off S's columns [Nb][wP], or nullptr
  int RT, wP, ntile, t;      // rows and tiles of the images
  int split, RS;             // a tile's rows: RS of RT / split
  int slots, groups;         // image slots, z group buffers
  volatile unsigned* err;    // device or mapped host memory
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
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
// Contiguous global -> shared copy completing on an mbarrier.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// K-major, no swizzle: core matrices of 8 rows x 16 bytes, adjacent in K 128
// bytes apart, 8-row groups sbo bytes apart
__device__ __forceinline__ uint64_t desc_noswz(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)(128 >> 4) << 16 |
         (uint64_t)((sbo >> 4) & 0x3FFFu) << 32 | (uint64_t)1 << 46;
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
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}

constexpr int kSpread = 4;             // powers of two
constexpr short kZeroColumn = -8192;   // kx of a column of zeros
constexpr int kZeroRow = -8192;        // ex of a row of zeros

// v 2^e; infinity (for a float64 dot product) where that or v is not a normal
// number, zero where v or the column of S is zero.
__device__ __forceinline__ uint2 times_pow2(uint2 v, int e) {
  const int fe = (int)(v.y >> 20 & 0x7ff), f = fe + e;
  if (fe != 0 && fe != 0x7ff && f >= 1 && f <= 2046) return make_uint2(v.x, v.y + ((uint32_t)e << 20));
  const bool zero = ((v.y & 0x7fffffffu) | v.x) == 0 || (fe != 0x7ff && e == kZeroColumn);
  return make_uint2(0, zero ? 0u : 0x7ff00000u);
}

// Row k of block b's z vector (all columns): the step's input ranges in order.
__device__ __forceinline__ const double* z_row(const sweep::Step<double>& s, int b, int k) {
  int q = 0, kk = k;
  while (q + 1 < s.nin && kk >= s.in_rows[q]) kk -= s.in_rows[q++];
  long long row = (long long)b * s.in_blk[q] + kk;
  if (q == 0 && s.in_perm) row = __ldg(s.in_perm + row);
  return s.in_p[q] + row * s.in_ld[q];
}
__device__ __noinline__ double dot_f64(const sweep::Step<double>& s, int b, int row, int col) {
  const double* S = s.S + (long long)b * s.sS + (long long)row * s.w;
  double v = 0.0;
  for (int k = 0; k < s.w; ++k) v = fma(S[k], z_row(s, b, k)[col], v);
  return v;
}

// Tile t of a step: block b, row tile rt, column tile ct (ct fastest: the
// tiles that read the same operator images run together).
struct Tile {
  int b, rt, ct;
};
__device__ __forceinline__ Tile tile_of(int t, int nrt, int nct) {
  Tile T;
  const int br = t / nct;
  T.ct = t - br * nct;
  T.b = br / nrt;
  T.rt = br - T.b * nrt;
  return T;
}

// Moduli per hand-over of z residues from the conversion to the MMAs: eight
// where two z buffers and eight images fit in shared memory (up to 64 rows and
// fewer than 32 columns or 64 of the operator's: 444 -> 432 us against four).
__host__ __device__ constexpr int handover(int nc, bool half, bool narrow) {
  return half && (nc < 32 || narrow) ? 8 : 4;
}

// NC: columns per tile (MMA N).  KPT: consecutive k per thread (512 threads,
// NC columns).  HALF: at most 64 rows, as MMAs of M = 64 (16 rows in each
// quarter of TMEM).
template <int NC, int KPT, bool HALF>
__global__ void __launch_bounds__(kThreads, 1) crt_step_kernel(const CrtStep o) {
  // moduli per hand-over of z residues (KPT NC: 128 up to 64 columns of the operator)
  constexpr int MH = handover(NC, HALF, KPT * NC == 128);
  constexpr int NHO = NM / MH;
  constexpr int PH = MH / kMma;          // of one MMA warp
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t afull[NM], aempty[NM];
  __shared__ __align__(8) uint64_t zfull[4], zempty[4], tfull, tempty, quiet[kMma];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_fail, d_fail;
  __shared__ int cmax[kWarps][NC];
  __shared__ int cex[2][NC];

  const sweep::Step<double>& s = o.s;
  const int wP = o.wP, nrt = o.ntile * o.split;
  const int nct = (s.c + NC - 1) / NC;
  const int ntiles = s.nb * nrt * nct;
  // a contiguous range of tiles: consecutive ones share operator images
  const int t0 = (int)((long long)blockIdx.x * ntiles / gridDim.x);
  const int nt = (int)((long long)(blockIdx.x + 1) * ntiles / gridDim.x) - t0;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* zB = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  const uint32_t zbytes = (uint32_t)NC * wP * 2;   // z residues of one modulus
  const int NG = o.groups;                         // z group buffers (MH moduli each)
  unsigned char* ring = zB + MH * NG * zbytes;
  const uint32_t abytes = (uint32_t)o.RS * wP * 2;   // operator image of one modulus
  const int S = o.slots;
  const bool resident = S == NM;
  auto key = [&](int i) {
    const Tile T = tile_of(t0 + i, nrt, nct);
    return T.b * nrt + T.rt;
  };
  // first of a tile's images; modulus l's is l RT wP elements on
  auto image = [&](int i) {
    const int kx = key(i), bt = kx / o.split;
    return o.img + (size_t)bt * NM * o.RT * wP + (size_t)(kx - bt * o.split) * o.RS * wP;
  };

  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&afull[i], 1);
      mbar_init(&aempty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&zfull[i], 1);
      mbar_init(&zempty[i], kMma);
    }
    mbar_init(&tfull, kMma);
    mbar_init(&tempty, kWarps);
    for (int i = 0; i < kMma; ++i) mbar_init(&quiet[i], 1);
    s_fail = 0;
    d_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(NM * NC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp < kMma) {
    // ---------------- warp j of four, one lane: images (constant, so no wait
    // for the previous launch) and MMAs of moduli j, j + 4, j + 8, j + 12, in
    // image slots j, j + 4, ..
    if (lane == 0) {
      const int j = warp, Sj = S / kMma, total = 4 * nt;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NC >> 3) << 17) |
                             ((uint32_t)((HALF ? 64 : 128) >> 4) << 24);
      const uint32_t sbo = (uint32_t)wP * 16;
      const uint64_t za = desc_noswz(smem_u32(zB), sbo), aa = desc_noswz(smem_u32(ring), sbo);
      const uint32_t zs = zbytes >> 4, as = abytes >> 4;   // descriptor steps
      // image m of this warp (tile m / 4, modulus j + 4 (m % 4)) into slot sl
      int ci = 0, cl = 0, cs = j, copies = 0;
      const size_t istride = (size_t)o.RT * wP;
      const __nv_bfloat16* src = image(0) + j * istride;
      auto copy = [&]() {
        bulk_copy(ring + cs * abytes, src + 4 * cl * istride, abytes, &afull[cs]);
        ++copies;
        if ((cs += kMma) >= S) cs = j;
        if (++cl == 4) {
          cl = 0;
          if (++ci < nt) src = image(ci) + j * istride;
        }
      };
      bool ok = true;
      uint32_t aph = resident ? 1 : 0, eph = 0, zph = 0;   // phase parities
      int slot = j, eslot = j, gb = 0;
      if (!resident)
        for (int m = 0; m < min(Sj, total); ++m) copy();
      for (int i = 0; i < nt && ok; ++i) {
        if (resident && (i == 0 || key(i) != key(i - 1))) {
          // all MMAs of the previous tile have read their images
          if (i > 0 && !mbar_wait(&tfull, (uint32_t)(i - 1) & 1, &s_fail)) {
            ok = false;
            break;
          }
          ci = i;
          src = image(i) + j * istride;
          for (int m = 0; m < 4; ++m) copy();
          aph ^= 1;
        }
        // the epilogue has read the previous tile's accumulators
        if (i > 0 && !mbar_wait(&tempty, (uint32_t)(i - 1) & 1, &s_fail)) ok = false;
#pragma unroll 1
        for (int h = 0; h < NHO && ok; ++h) {
          // this warp's moduli of the hand-over, in turn: MMAs into one
          // accumulator wait for one another (~250 clocks)
          int sl[PH];
          uint64_t ad[PH];
          ok = mbar_wait(&zfull[gb], zph, &s_fail);
#pragma unroll
          for (int m = 0; m < PH; ++m) {
            sl[m] = slot;
            ad[m] = aa + (uint64_t)(slot * as);
            ok = ok && mbar_wait(&afull[slot], aph, &s_fail);
            if ((slot += kMma) >= S) {
              slot = j;
              if (!resident) aph ^= 1;
            }
          }
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t bd = za + (uint64_t)((MH * gb + j) * zs);
          const uint32_t td = tmem + (uint32_t)((MH * h + j) * NC);
#pragma unroll 4
          for (int k = 0; k < wP / 16; ++k)
#pragma unroll
            for (int m = 0; m < PH; ++m)
              mma_bf16(td + (uint32_t)(kMma * m * NC), ad[m] + 16 * k,
                       bd + (uint64_t)(kMma * m * zs) + 16 * k, idesc, k != 0);
          mma_commit(&zempty[gb]);
          if (++gb == NG) {
            gb = 0;
            zph ^= 1;
          }
          if (!resident) {
            for (int m = 0; m < PH; ++m) mma_commit(&aempty[sl[m]]);
            // the slots of the MMAs before these (of these, if there are no
            // others) take the next images
            if (NHO * i + h > 0 || Sj == PH)
              for (int m = 0; m < PH && copies < total && ok; ++m) {
                ok = mbar_wait(&aempty[eslot], eph, &s_fail);
                if (!ok) break;
                copy();
                if ((eslot += kMma) >= S) {
                  eslot = j;
                  eph ^= 1;
                }
              }
          }
        }
        if (ok) mma_commit(&tfull);
      }
      if (!ok) {
        s_fail = 1;
        if (o.err) *o.err = 1;
      }
      // every MMA issued has finished and every copy landed before TMEM and
      // shared memory are given up
      mma_commit(&quiet[j]);
      mbar_wait(&quiet[j], 0, nullptr);
      for (int m = max(0, copies - Sj); m < copies; ++m)
        mbar_wait(&afull[j + kMma * (m % Sj)], (uint32_t)(m / Sj) & 1, nullptr);
    }
    __syncwarp();
  } else {
    const int cw = warp - kMma, col = lane % NC;
    const int k0 = (cw * (32 / NC) + lane / NC) * KPT;
    uint2 z[KPT];
    uint32_t kx[(KPT + 1) / 2];   // two a word
    auto fetch = [&](int i) {
      const Tile T = tile_of(t0 + i, nrt, nct);
      const int c = T.ct * NC + col;
      if (o.kx) {
        const short* kp = o.kx + (long long)T.b * wP + (k0 < wP ? k0 : 0);
        if constexpr (KPT == 1) {
          kx[0] = (uint16_t)__ldg(kp);
        } else {
#pragma unroll
          for (int u = 0; u < KPT / 2; ++u) kx[u] = __ldg(reinterpret_cast<const uint32_t*>(kp) + u);
        }
      }
#pragma unroll
      for (int u = 0; u < KPT; ++u) {
        z[u] = make_uint2(0, 0);
        if (k0 + u < s.w && c < s.c)
          z[u] = *reinterpret_cast<const uint2*>(z_row(s, T.b, k0 + u) + c);
      }
    };
    sweep::grid_dependency_wait();
    if (nt > 0) fetch(0);
    constexpr int CG = NC / 4;           // columns per warp of a TMEM quarter
    const int q = cw & 3, g = cw >> 2;   // quarter (= warp % 4), columns CG g ..
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + CG * g;
    for (int i = 0; i < nt; ++i) {
      const Tile T = tile_of(t0 + i, nrt, nct);
      if (o.kx) {
#pragma unroll
        for (int u = 0; u < KPT; ++u)
          z[u] = times_pow2(z[u], (int)(short)(kx[u >> 1] >> (16 * (u & 1))));
      }
      // column exponents
      int mx = 0;
#pragma unroll
      for (int u = 0; u < KPT; ++u) mx = max(mx, (int)(z[u].y & 0x7fffffffu));
#pragma unroll
      for (int x = NC; x < 32; x *= 2) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      cmax[cw][col] = mx;
      if (cw == 0 && lane == 0 && s_fail) d_fail = 1;
      asm volatile("bar.sync 1, %0;" ::"r"(32 * kWarps) : "memory");
      if (d_fail) break;   // the same for every compute warp
      int F = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) F = max(F, cmax[w][col]);
      F >>= 20;
      if (cw == 0) cex[i & 1][col] = F;
      // residues, MH moduli per hand-over (a warp without k only arrives)
      uint32_t lo[KPT], hi[KPT];
#pragma unroll
      for (int u = 0; u < KPT; ++u)
        scaled(z[u].y, z[u].x, max(F, 1), o.t, F != 0x7ff, lo[u], hi[u]);
      unsigned char* zdst =
          zB + (col >> 3) * (wP * 16) + (k0 >> 3) * 128 + (col & 7) * 16 + (k0 & 7) * 2;
#pragma unroll 1
      for (int h = 0; h < NHO; ++h) {
        const int G = NHO * i + h, gb = G % NG;
        // the group buffer's previous MMAs have read it
        const bool free = G < NG || mbar_wait(&zempty[gb], (uint32_t)(G / NG - 1) & 1, &s_fail);
        unsigned char* dst = zdst + MH * gb * (int)zbytes;
        if (k0 < wP && free) {
#pragma unroll
          for (int q = 0; q < MH; ++q) {
            const int l = MH * h + q;
            const uint32_t c0 = c_tab.ca[0][l], c1 = c_tab.ca[1][l];
            const int bias = 0x4B400000 + c_tab.ba[l];
            const float p = c_tab.pf[l], ip = c_tab.inv[l];
            float y[KPT];
#pragma unroll
            for (int u = 0; u < KPT; ++u) y[u] = residue(lo[u], hi[u], c0, c1, bias, p, ip);
            unsigned char* d = dst + q * zbytes;
            if constexpr (KPT == 8)
              *reinterpret_cast<uint4*>(d) = make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]),
                                                        pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
            else if constexpr (KPT == 4)
              *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
            else if constexpr (KPT == 2)
              *reinterpret_cast<uint32_t*>(d) = pack_bf16(y[0], y[1]);
            else
              *reinterpret_cast<__nv_bfloat16*>(d) = __float2bfloat16_rn(y[0]);
          }
        }
        // all warps together: left alone, the scheduler finishes one warp's
        // groups before the next warp's first, and the MMAs wait for the last
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"r"(32 * kWarps) : "memory");
        if (cw == 0 && lane == 0) mbar_arrive(&zfull[gb]);
      }
      if (i + 1 < nt) fetch(i + 1);
      else sweep::launch_dependents();
      // this thread's output row, and columns c0 + es, + 2, .. (HALF) or c0, + 1, ..
      const int rt = T.rt / o.split, sub = T.rt - rt * o.split;
      const int r0 = rt * o.RT + sub * o.RS, r = HALF ? 16 * q + (lane & 15) : 32 * q + lane;
      const int nr = min(sub + 1 < o.split ? o.RS : o.RT - sub * o.RS, s.rows - r0);
      const int es = HALF ? lane >> 4 : 0;
      const int c0 = T.ct * NC + CG * g, nc = min(CG, s.c - c0);
      const bool mine = (HALF ? 16 : 32) * q < nr && nc > 0;   // uniform over the warp
      double* out = nullptr;
      int fa = 0;
      if (r < nr) {
        const int row = r0 + r;
        if (row < s.split) {
          const long long p = (long long)T.b * s.out_blk[0] + row;
          out = s.out_p[0] + (s.out_perm ? __ldg(s.out_perm + p) : p) * s.out_ld[0] + c0;
        } else {
          out = s.out_p[1] + ((long long)T.b * s.out_blk[1] + (row - s.split)) * s.out_ld[1] + c0;
        }
        fa = __ldg(o.ex + (size_t)(T.b * o.ntile + rt) * o.RT + sub * o.RS + r);
      }
      const bool ok = mbar_wait(&tfull, (uint32_t)i & 1, &s_fail);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          s_fail = 1;
          if (o.err) *o.err = 1;
        }
        continue;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      constexpr int EP = HALF ? CG / 2 : CG;   // outputs per thread
      constexpr int EU = EP < 2 ? EP : 2;
      uint32_t R[EP][4];
      if (mine) {
#pragma unroll
        for (int l4 = 0; l4 < 4; ++l4) {
          uint32_t v[4][CG];
#pragma unroll
          for (int l = 0; l < 4; ++l) tmem_ld(taddr + (uint32_t)((4 * l4 + l) * NC), v[l]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < EP; ++e) {
            uint32_t y[4];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
              uint32_t x;
              if constexpr (HALF) {
                // rows in lanes 0..15: the other half takes the odd columns
                const uint32_t odd = __shfl_sync(0xffffffffu, v[l][2 * e + 1], lane & 15);
                x = lane < 16 ? v[l][2 * e] : odd;
              } else {
                x = v[l][e];
              }
              y[l] = reduced(__uint_as_float(x), c_tab.pf[4 * l4 + l], c_tab.inv[4 * l4 + l]);
            }
            R[e][l4] = __byte_perm(__byte_perm(y[0], y[1], 0x40), __byte_perm(y[2], y[3], 0x40),
                                   0x5410);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty);
      if (mine && r < nr) {
        // two outputs per pass, the registers moved up after it: unrolled eight
        // times the reconstruction outgrows the instruction cache
#pragma unroll 1
        for (int e0 = 0; e0 < EP; e0 += EU) {
#pragma unroll
          for (int u = 0; u < EU; ++u) {
            const int e = HALF ? 2 * (e0 + u) + es : e0 + u;
            if (e < nc) {
              const int fb = cex[i & 1][CG * g + e], f = fa + max(fb, 1);
              double v = combine(R[u][0], R[u][1], R[u][2], R[u][3], f - 2 * (1022 + o.t));
              // not finite, or below 2^-44 of the largest entries
              if (fa == 0x7ff || fb == 0x7ff || (int)(hi32(v) >> 20 & 0x7ff) < f - 1065)
                v = dot_f64(s, T.b, r0 + r, c0 + e);
              out[e] = v;
            }
          }
#pragma unroll
          for (int j = 0; j + EU < EP; ++j)
#pragma unroll
            for (int a = 0; a < 4; ++a) R[j][a] = R[j + EU][a];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NM * NC)
                 : "memory");
}

// The operators of one direction, for one launch.
constexpr int kMaxOps = 56;
struct ImageOp {
  const double* S;
  __nv_bfloat16* img;
  int* ex;
  short* kx;
  int first;   // rows (padded) of the operators before it
  int firstb;  // blocks of the operators before it
  int rows, w, RT, wP, ntile, t;
};
struct ImageOps {
  int count, total, blocks;
  int* scaled;   // [count], zeroed: operators that have a kx other than 0
  ImageOp op[kMaxOps];
};

// exponent field of a number, 1 for a subnormal one
__device__ __forceinline__ int field(uint2 v) { return max((int)(v.y >> 20 & 0x7ff), 1); }
__device__ __forceinline__ bool is_zero(uint2 v) { return ((v.y & 0x7fffffffu) | v.x) == 0; }

// kx of every column of every block, from its largest finite entry; one CTA per
// block.
__global__ void __launch_bounds__(kMaxW) crt_column_kernel(const __grid_constant__ ImageOps a) {
  __shared__ int lo, hi;
  const int gb = blockIdx.x, k = threadIdx.x;
  int i = 0;
  while (i + 1 < a.count && gb >= a.op[i + 1].firstb) ++i;
  const ImageOp& o = a.op[i];
  const int b = gb - o.firstb;
  if (k == 0) {
    lo = 0x7fff;
    hi = 0;
  }
  __syncthreads();
  int e = 0;   // 0: a column of zeros
  if (k < o.w) {
    const uint2* S = reinterpret_cast<const uint2*>(o.S + (long long)b * o.rows * o.w + k);
#pragma unroll 8
    for (int r = 0; r < o.rows; ++r) {
      const uint2 v = S[(long long)r * o.w];
      const int f = field(v);
      if (f < 0x7ff && !is_zero(v)) e = max(e, f);
    }
    if (e) {
      atomicMin(&lo, e);
      atomicMax(&hi, e);
    }
  }
  __syncthreads();
  const short kx = k >= o.w ? 0 : (e == 0 ? kZeroColumn : (hi - lo > kSpread ? (short)(e - 1023) : 0));
  if (k < o.wP) o.kx[(long long)b * o.wP + k] = kx;
  if (kx) a.scaled[i] = 1;
}

// Residue images: one warp per (operator, block, tile row), lane = eight
// consecutive k; rows beyond the operator's are zero.
__global__ void __launch_bounds__(256) crt_op_kernel(const __grid_constant__ ImageOps a) {
  const int gr = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (gr >= a.total) return;
  int i = 0;
  while (i + 1 < a.count && gr >= a.op[i + 1].first) ++i;
  const ImageOp& o = a.op[i];
  const int gw = gr - o.first, RT = o.RT, wP = o.wP, w = o.w;
  const int bt = gw / RT, rr = gw - bt * RT, b = bt / o.ntile, r = (bt - b * o.ntile) * RT + rr;
  const uint2* row = reinterpret_cast<const uint2*>(o.S + ((long long)b * o.rows + r) * w);
  uint2 v[8];
  int ex[8], mx = kZeroRow;
  bool finite = true;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int k = 8 * lane + u;
    v[u] = (r < o.rows && k < w) ? row[k] : make_uint2(0, 0);
    finite = finite && field(v[u]) < 0x7ff;
    ex[u] = is_zero(v[u]) ? kZeroRow : field(v[u]) - o.kx[(long long)b * wP + k];
    mx = max(mx, ex[u]);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  finite = __all_sync(0xffffffffu, finite);
  if (lane == 0) o.ex[gw] = finite ? mx : 0x7ff;
  if (8 * lane >= wP) return;
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
    scaled_by(v[u].y, v[u].x, mx - ex[u], o.t, finite && ex[u] > kZeroRow, lo[u], hi[u]);
  __nv_bfloat16* dst = o.img + (size_t)bt * NM * RT * wP + (size_t)(rr >> 3) * (wP * 8) +
                       lane * 64 + (rr & 7) * 8;
#pragma unroll
  for (int l = 0; l < NM; ++l) {
    const uint32_t c0 = c_tab.cb[0][l], c1 = c_tab.cb[1][l];
    const int bias = 0x4B400000 + c_tab.bb[l];
    const float p = c_tab.pf[l], ip = c_tab.inv[l];
    uint32_t x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      x[u] = pack_bf16(residue(lo[2 * u], hi[2 * u], c0, c1, bias, p, ip),
                       residue(lo[2 * u + 1], hi[2 * u + 1], c0, c1, bias, p, ip));
    *reinterpret_cast<uint4*>(dst + (size_t)l * RT * wP) = make_uint4(x[0], x[1], x[2], x[3]);
  }
}

// Row tiles of an operator's images: `ntile` of RT rows (a multiple of eight).
void row_tiles(int rows, int& ntile, int& RT) {
  ntile = (rows + kRows - 1) / kRows;
  RT = ((rows + ntile - 1) / ntile + 7) / 8 * 8;
}

// One operator's part of a direction's images.
struct Part {
  CrtOp* op;
  const DevBuf* S;
};

// Makes the images of `parts` in `buf`; false where they don't fit in the
// memory they may take.
bool make_images(cudaStream_t st, const std::vector<Part>& parts, size_t limit, DevBuf& buf) {
  if ((int)parts.size() > kMaxOps) return false;
  ImageOps a{};
  size_t bytes = (4 * parts.size() + 1023) / 1024 * 1024;   // `scaled`
  long long total = 0, blocks = 0;
  std::vector<size_t> at;
  for (const Part& p : parts) {
    CrtOp& o = *p.op;
    row_tiles(o.rows, o.ntile, o.RT);
    o.wP = (o.w + 15) / 16 * 16;
    const size_t tr = (size_t)o.Nb * o.ntile * o.RT;
    // a split tile's copy takes eight rows more than there are where RT / 8 is odd
    at.push_back(bytes);
    bytes += (2 * (NM * tr + 8) * o.wP + 1023) / 1024 * 1024;
    at.push_back(bytes);
    bytes += (4 * tr + 1023) / 1024 * 1024;
    at.push_back(bytes);
    bytes += (2 * (size_t)o.Nb * o.wP + 1023) / 1024 * 1024;
    total += (long long)tr;
    blocks += o.Nb;
  }
  if (bytes > limit || total >= (1LL << 31)) return false;
  try {
    buf.alloc(bytes, st);
  } catch (const Error&) {
    cudaGetLastError();   // no memory for them: the float64 steps need none
    return false;
  }
  a.scaled = buf.as<int>();
  SLU_CHECK_CUDA(cudaMemsetAsync(a.scaled, 0, 4 * parts.size(), st));
  for (size_t i = 0; i < parts.size(); ++i) {
    CrtOp& o = *parts[i].op;
    ImageOp& d = a.op[a.count++];
    d.S = parts[i].S->as<double>();
    d.img = reinterpret_cast<__nv_bfloat16*>(buf.as<char>() + at[3 * i]);
    d.ex = reinterpret_cast<int*>(buf.as<char>() + at[3 * i + 1]);
    d.kx = reinterpret_cast<short*>(buf.as<char>() + at[3 * i + 2]);
    d.first = a.total;
    d.firstb = a.blocks;
    d.rows = o.rows;
    d.w = o.w;
    d.RT = o.RT;
    d.wP = o.wP;
    d.ntile = o.ntile;
    d.t = bits_for(o.w);
    a.total += o.Nb * o.ntile * o.RT;
    a.blocks += o.Nb;
    o.img = d.img;
    o.ex = d.ex;
    o.kx = d.kx;
  }
  crt_column_kernel<<<(unsigned)blocks, kMaxW, 0, st>>>(a);
  check_launch("crt_column_kernel");
  crt_op_kernel<<<(unsigned)((a.total + 7) / 8), 256, 0, st>>>(a);
  check_launch("crt_op_kernel");
  // operators that need no scaling (their steps skip it)
  std::vector<int> need(parts.size());
  SLU_CHECK_CUDA(cudaMemcpyAsync(need.data(), a.scaled, 4 * parts.size(), cudaMemcpyDeviceToHost, st));
  stream_wait(st);   // other streams may use the images from here on, too
  for (size_t i = 0; i < parts.size(); ++i)
    if (!need[i]) parts[i].op->kx = nullptr;
  return true;
}

// A step's tiles: nc columns, RT / split rows.  Narrower and lower ones while
// one wave of CTAs takes them all, since a tile's time is nearly that of its
// conversions and reconstructions (64 x 64 operators: 8.5 us with 32 columns,
// 6 with 16, 4.5 with 8).
struct Tiling {
  int nc = 32, split = 1, RS = 0;
  long long tiles = 0;
};
Tiling tiling_of(long long nb, int rows, int c) {
  const long long sms = num_sms();
  int ntile, RT;
  row_tiles(rows, ntile, RT);
  Tiling g;
  auto tiles = [&](int nc, int split) { return nb * ntile * split * ((c + nc - 1) / nc); };
  if (tiles(16, 1) <= sms) g.nc = 16;
  if (RT > 64 && tiles(g.nc, 2) <= sms) g.split = 2;
  g.RS = g.split == 1 ? RT : (RT + 15) / 16 * 8;
  if (g.RS <= 64 && g.nc == 16 && tiles(8, g.split) <= sms) g.nc = 8;
  g.tiles = tiles(g.nc, g.split);
  return g;
}

void launch(cudaStream_t st, const sweep::Step<double>& s, const CrtOp& op, volatile unsigned* err,
            const char* what) {
  SLU_REQUIRE(op.img && s.S && s.rows == op.rows && s.w == op.w && s.nb == op.Nb,
              "residue step: operator does not match its step");
  CrtStep o{};
  o.s = s;
  o.img = op.img;
  o.ex = op.ex;
  o.kx = op.kx;
  o.RT = op.RT;
  o.wP = op.wP;
  o.ntile = op.ntile;
  o.t = bits_for(op.w);
  o.err = err;
  const Tiling g = tiling_of(s.nb, op.rows, s.c);
  const int nc = g.nc;
  o.split = g.split;
  o.RS = g.RS;
  const bool half = o.RS <= 64;
  const size_t z = (size_t)NM * nc * op.wP * 2, a = (size_t)o.RS * op.wP * 2;
  // the MMA reads 64 or 128 rows from an image of RS
  const size_t tail = (size_t)((half ? 64 : kRows) - o.RS) * op.wP * 2;
  // z group buffers: all where the images then still fit as a whole, else half
  // (at least two); the rest of shared memory holds operator images
  const bool narrow = op.wP <= 64;
  const int mh = handover(nc, half, narrow), all = NM / mh;
  o.groups = z + NM * a + tail + 1024 <= kSmemMax ? all : 2;
  const size_t zb = z / all * o.groups;
  o.slots = (int)std::min<size_t>(NM, (kSmemMax - 1024 - zb - tail) / a) / mh * mh;
  SLU_REQUIRE(o.slots >= mh, "residue step too wide");
  sweep::LaunchPlan p;
  p.ctas = std::min<long long>(g.tiles, num_sms());
  p.threads = kThreads;
  p.smem = 1024 + zb + tail + o.slots * a;
  auto kern = nc == 32 ? (half ? (narrow ? crt_step_kernel<32, 4, true> : crt_step_kernel<32, 8, true>)
                               : (narrow ? crt_step_kernel<32, 4, false>
                                         : crt_step_kernel<32, 8, false>))
            : nc == 16 ? (half ? (narrow ? crt_step_kernel<16, 2, true> : crt_step_kernel<16, 4, true>)
                               : (narrow ? crt_step_kernel<16, 2, false>
                                         : crt_step_kernel<16, 4, false>))
                       : (narrow ? crt_step_kernel<8, 1, true> : crt_step_kernel<8, 2, true>);
  ensure_smem(reinterpret_cast<const void*>(kern), p.smem);
  sweep::launch_pdl(kern, p, st, what, o);
}

// f(nb, rows, w) for every step of a direction.
template <typename F>
void each_step(const Hbs& H, bool solve, bool trans, F f) {
  for (int t = 0; t < H.L; ++t) {
    const Level& l = H.lv[t];
    const bool root = t == H.L - 1;
    const int nb = root ? 1 : l.Nb;
    if (solve) {
      const int rows = t == 0 ? l.n : 2 * l.n, w = root ? l.n : l.nu + 2 * l.k;
      if (!root) f(nb, l.n, l.n);
      f(nb, trans ? w : rows, trans ? rows : w);
    } else {
      if (!root) f(nb, l.k, l.n);
      f(nb, l.n, root ? l.n : l.n + l.k);
    }
  }
}

// Makes the residue images of a direction unless they are there.
bool ready(Handle& h, Hbs& H, bool solve, bool trans) {
  const int dir = (solve ? 0 : 2) + (trans ? 1 : 0);
  std::atomic<bool>& have = H.has_crt[dir];
  if (have) return true;
  if (H.no_crt[dir]) return false;
  cudaStream_t st = h.stream;
  // the first use waits for the images: not inside a stream capture
  if (capturing(st)) return false;
  std::lock_guard<std::mutex> lock(H.lazy_mu);
  if (have) return true;
  if (H.no_crt[dir]) return false;
  const bool compose = !solve && !H.has_apply[trans ? 1 : 0];
  if (compose) hbs_make_apply(h, H, trans, false);
  std::vector<Part> parts;
  auto add = [&](CrtOp& o, const DevBuf& S, int nb, int rows, int w) {
    o.Nb = nb;
    o.rows = rows;
    o.w = w;
    parts.push_back({&o, &S});
  };
  for (int t = 0; t < H.L; ++t) {
    Level& l = H.lv[t];
    const bool root = t == H.L - 1;
    const int nb = root ? 1 : l.Nb;
    if (solve) {
      const int rows = t == 0 ? l.n : 2 * l.n, w = root ? l.n : l.nu + 2 * l.k;
      if (!root) add(trans ? l.crQ : l.crQt, trans ? l.Q : l.Qt, nb, l.n, l.n);
      if (trans) add(l.crSwT, l.SwT, nb, w, rows);
      else add(l.crSw, l.Sw, nb, rows, w);
    } else {
      if (!root) add(trans ? l.crUpT : l.crUp, trans ? l.AupT : l.Aup, nb, l.k, l.n);
      add(trans ? l.crDnT : l.crDn, trans ? l.AdnT : l.Adn, nb, l.n, root ? l.n : l.n + l.k);
    }
  }
  const bool made = make_images(st, parts, H.crt_limit, H.crt_buf[dir]);
  if (!made) {
    H.no_crt[dir] = true;
    if (!compose) return false;
    stream_wait(st);   // the composed operators
  }
  if (compose) H.has_apply[trans ? 1 : 0] = true;
  have = made;
  return made;
}

}  // namespace

// By shape and c alone.  The float64 steps take 2 us each and their
// multiplications at the pipe's rate, 0.87 TFLOP/s of what a step asks for;
// the residue steps 3.5 us each and a tile's time per wave of tiles (above).
// They have to win by 40 us, about what the images cost on the first call:
// solves of 4096 rows (leaves of 64, rank 32) with 48 columns take 198 -> 116
// us, 64: 249 -> 117, 300: 1292 -> 293; of 1024 rows with 64
// columns 79 -> 72 (left to float64), 128: 128 -> 79; with leaves of 16 the
// float64 steps stay ahead (4096 rows, 300 columns: 297 against 607).
// Up to 32 columns a call's bits are those of the float64 steps, which groups and
// single calls share.  One level may be solved in place, which wants whole columns
// per CTA.
bool crt_steps_pay(const Hbs& H, bool solve, bool trans, int c) {
  if (c <= 32 || H.L < 2) return false;
  bool fit = true;
  double f64 = 0.0, crt = 0.0;   // us
  each_step(H, solve, trans, [&](int nb, int rows, int w) {
    fit = fit && nb >= 1 && rows >= 1 && w >= 1 && w <= kMaxW;
    if (!fit) return;
    const Tiling g = tiling_of(nb, rows, c);
    fit = g.tiles * NM < (1LL << 31);
    const double tile = g.nc == 8 ? 4.5 : (g.nc == 16 ? 6.0 : 8.5) * (g.RS <= 64 ? 1.0 : 1.3);
    const long long sms = num_sms();
    f64 += 2.0 + 2.0 * nb * rows * (double)w * c / 0.87e6;
    crt += 3.5 + tile * (double)((g.tiles + sms - 1) / sms);
  });
  return fit && f64 >= crt + 40.0;
}

bool crt_steps_run(const Hbs& H, bool solve, bool trans, int c) {
  return !H.no_crt[(solve ? 0 : 2) + (trans ? 1 : 0)] && crt_steps_pay(H, solve, trans, c);
}

bool crt_prepare(Handle& h, Hbs& H, bool solve, bool trans, int c) {
  return crt_steps_pay(H, solve, trans, c) && ready(h, H, solve, trans);
}

// B (N x c, caller ordering) <- A^{-1} X or A^{-T} X; scratch: five buffers of
// `stride` elements (as ulv_solve_fused); X == B solves in place.
void crt_solve(cudaStream_t st, const Hbs& H, bool trans, const double* X, int ldx, double* B,
               int ldb, int c, double* scratch, size_t stride, volatile unsigned* err) {
  SLU_REQUIRE(H.has_crt[trans ? 1 : 0], "residue solve not prepared");
  const int L = H.L;
  const std::vector<long long>& NN = H.NN;
  double* ru = scratch;
  if (!trans) {
    const int64_t* perm = H.perm.as<int64_t>();
    double* P[4] = {scratch + stride, scratch + 2 * stride, scratch + 3 * stride,
                    scratch + 4 * stride};
    if (L == 1) {
      sweep::Step<double> s = sweep::root_step<double>(H, X, ldx, B, ldb, nullptr, nullptr, c);
      s.in_p[0] = X;
      s.in_ld[0] = ldx;
      launch(st, s, H.lv[0].crSw, err, "crt_root_step");
      return;
    }
    const double* src = X;
    int lds = ldx;
    for (int t = 0; t + 1 < L; ++t) {
      launch(st,
             sweep::forward_step<double>(H, t, src, lds, t == 0 ? perm : nullptr, ru + NN[t] * c,
                                         P[t & 1], c),
             H.lv[t].crQt, err, "crt_fwd_step");
      src = P[t & 1];
      lds = c;
    }
    launch(st, sweep::root_step<double>(H, src, lds, B, ldb, P[2], P[3], c), H.lv[L - 1].crSw, err,
           "crt_root_step");
    int in = 2;
    for (int t = L - 2; t >= 0; --t) {
      const int out = in == 2 ? 0 : 2;
      launch(st,
             sweep::backward_step<double>(H, t, ru + NN[t] * c, P[in + 1], P[in], P[out],
                                          P[out + 1], B, ldb, c),
             H.lv[t].crSw, err, "crt_bwd_step");
      in = out;
    }
    return;
  }
  const int64_t* ip = H.iperm.as<int64_t>();
  double* P[2] = {scratch + stride, scratch + 3 * stride};
  if (L == 1) {
    launch(st, sweep::rootT_step<double>(H, X, ldx, ip, B, ldb, ip, c), H.lv[0].crSwT, err,
           "crt_rootT_step");
    return;
  }
  for (int t = 0; t + 1 < L; ++t)
    launch(st,
           sweep::backwardT_step<double>(H, t, t == 0 ? X : P[(t - 1) & 1], t == 0 ? ldx : c,
                                         t == 0 ? ip : nullptr, ru + NN[t] * c, P[t & 1], c),
           H.lv[t].crSwT, err, "crt_bwdT_step");
  int cur = (L - 1) & 1;
  launch(st, sweep::rootT_step<double>(H, P[(L - 2) & 1], c, nullptr, P[cur], c, nullptr, c),
         H.lv[L - 1].crSwT, err, "crt_rootT_step");
  for (int t = L - 2; t >= 0; --t) {
    const bool leaf = t == 0;
    launch(st,
           sweep::forwardT_step<double>(H, t, ru + NN[t] * c, P[cur], leaf ? B : P[cur ^ 1],
                                        leaf ? ldb : c, leaf ? ip : nullptr, c),
           H.lv[t].crQ, err, "crt_fwdT_step");
    cur ^= 1;
  }
}

// Y = A X or A^T X; scratch of hbs_apply_scratch_elems elements.
void crt_apply(cudaStream_t st, const Hbs& H, bool trans, const double* X, int ldx, double* Y,
               int ldy, int c, double* scratch, volatile unsigned* err) {
  SLU_REQUIRE(H.has_crt[trans ? 3 : 2], "residue apply not prepared");
  const int L = H.L;
  const int64_t* perm = H.perm.as<int64_t>();
  std::vector<double*> VV(L, nullptr);
  size_t off = 0;
  for (int t = 0; t + 1 < L; ++t) {
    VV[t + 1] = scratch + off;
    off += ((size_t)H.lv[t].Nb * H.lv[t].k * c + 63) & ~size_t(63);
  }
  double* u[2] = {scratch + off, scratch + off + (((size_t)H.N * c + 63) & ~size_t(63))};
  auto dn = [&](const Level& l) { return (trans ? l.AdnT : l.Adn).as<double>(); };
  const Level& r = H.lv[L - 1];
  if (L == 1) {
    launch(st, sweep::down_step<double>(r, dn(r), true, X, ldx, perm, nullptr, Y, ldy, perm, c),
           trans ? r.crDnT : r.crDn, err, "crt_apply_root");
    return;
  }
  for (int t = 0; t + 1 < L; ++t) {
    const Level& l = H.lv[t];
    launch(st,
           sweep::up_step<double>(l, (trans ? l.AupT : l.Aup).as<double>(), t == 0 ? X : VV[t],
                                  t == 0 ? ldx : c, t == 0 ? perm : nullptr, VV[t + 1], c),
           trans ? l.crUpT : l.crUp, err, "crt_apply_up");
  }
  launch(st,
         sweep::down_step<double>(r, dn(r), true, VV[L - 1], c, nullptr, nullptr, u[0], c, nullptr,
                                  c),
         trans ? r.crDnT : r.crDn, err, "crt_apply_root");
  int cur = 0;
  for (int t = L - 2; t >= 0; --t) {
    const Level& l = H.lv[t];
    const bool leaf = t == 0;
    launch(st,
           sweep::down_step<double>(l, dn(l), false, leaf ? X : VV[t], leaf ? ldx : c,
                                    leaf ? perm : nullptr, u[cur], leaf ? Y : u[cur ^ 1],
                                    leaf ? ldy : c, leaf ? perm : nullptr, c),
           trans ? l.crDnT : l.crDn, err, "crt_apply_down");
    cur ^= 1;
  }
}

}  // namespace slu
