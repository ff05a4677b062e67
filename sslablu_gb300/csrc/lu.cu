// LU with partial pivoting (LAPACK getrf's pivots and storage) and explicit
// inverses, batched: the pivot blocks of the red-black and Thomas
// eliminations (direct_solve/omsdirectsolve.py:89-94, 211, 333).
//
// Right-looking in two block sizes.  A panel of 32 columns is factored by one
// thread-block cluster per matrix with the panel in registers; its row swaps
// go to every other column at once; inside an outer block of 128 columns the
// following panels are updated on the float64 units, and right of it the
// trailing matrix takes one rank-128 update per outer block as a tensor-core
// product (gemm_f64), which carries nearly all flops of a large block.
#include <cooperative_groups.h>

#include <algorithm>

#include "hbs.cuh"

namespace cg = cooperative_groups;

namespace slu {
namespace {

constexpr int kPanel = 32;       // columns per panel
constexpr int kOuter = 128;      // columns per outer block
constexpr int kPanelRows = 512;  // rows (threads) per CTA of the panel kernel at most

// Largest v of the block and, of equal ones, the smallest idx.
__device__ inline void argmax_abs_block(double v, int idx, double* sv, int* si, double& out_v,
                                        int& out_i) {
  // warp reduce
  for (int o = 16; o > 0; o >>= 1) {
    double ov = __shfl_down_sync(0xffffffffu, v, o);
    int oi = __shfl_down_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  }
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { sv[w] = v; si[w] = idx; }
  __syncthreads();
  if (w == 0) {
    int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? sv[lane] : -1.0;
    idx = lane < nw ? si[lane] : 0x7fffffff;
    for (int o = 16; o > 0; o >>= 1) {
      double ov = __shfl_down_sync(0xffffffffu, v, o);
      int oi = __shfl_down_sync(0xffffffffu, idx, o);
      if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    if (lane == 0) { sv[0] = v; si[0] = idx; }
  }
  __syncthreads();
  out_v = sv[0];
  out_i = si[0];
  __syncthreads();
}

// Panels of more rows than a cluster holds: the panel in global memory, one
// CTA per matrix.  src[i] = the row that ends at row i.
__global__ void __launch_bounds__(1024)
lu_panel_global_kernel(int n, int k0, int kb, double* __restrict__ A, int lda, long long sA,
                       int* __restrict__ piv, long long sP, int* __restrict__ src, int* info,
                       int istep) {
  A += blockIdx.x * sA;
  piv += blockIdx.x * sP;
  src += (long long)blockIdx.x * n;
  __shared__ double sv[32];
  __shared__ int si[32];
  int first_zero = 0;
  const int k1 = k0 + kb;
  for (int i = k0 + threadIdx.x; i < n; i += blockDim.x) src[i] = i;
  __syncthreads();
  for (int j = k0; j < k1; ++j) {
    double best = -1.0;
    int bi = j;
    for (int i = j + threadIdx.x; i < n; i += blockDim.x) {
      const double v = fabs(A[(long long)i * lda + j]);
      if (v > best) { best = v; bi = i; }
    }
    double pv;
    int p;
    argmax_abs_block(best, bi, sv, si, pv, p);
    if (threadIdx.x == 0) {
      piv[j] = p;
      const int t = src[j];
      src[j] = src[p];
      src[p] = t;
    }
    if (p != j) {
      for (int c = k0 + threadIdx.x; c < k1; c += blockDim.x) {
        const double t = A[(long long)j * lda + c];
        A[(long long)j * lda + c] = A[(long long)p * lda + c];
        A[(long long)p * lda + c] = t;
      }
    }
    __syncthreads();
    const double d = A[(long long)j * lda + j];
    if (d == 0.0) {
      if (!first_zero) first_zero = j + 1;
      __syncthreads();
      continue;
    }
    const double inv = 1.0 / d;
    for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) A[(long long)i * lda + j] *= inv;
    __syncthreads();
    const int w = k1 - j - 1;   // panel columns right of j
    if (w > 0) {
      const long long tot = (long long)(n - j - 1) * w;
      for (long long e = threadIdx.x; e < tot; e += blockDim.x) {
        const int i = j + 1 + (int)(e / w), c = j + 1 + (int)(e % w);
        A[(long long)i * lda + c] -= A[(long long)i * lda + j] * A[(long long)j * lda + c];
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && first_zero && info) atomicCAS(info + istep * blockIdx.x, 0, first_zero);
}

// Panel factorisation by one cluster per matrix.  Thread = row, the row's kb
// panel entries in registers, so the rank-1 updates spread over the float64
// pipes of the cluster's SMs (2 FMA per clock each).  Rows are never moved: a
// thread carries the position its row has after the swaps and stores it there
// at the end.
// A column is a chain of latencies: largest entry, its row to all, multiplier,
// update of the next column.  It is kept short by
//  * no barrier: every warp sends its candidate (key, row, 1/d) straight to
//    every CTA of the cluster with asynchronous stores that complete on the
//    receiver's mbarrier, and every warp picks the winner of all candidates
//    itself; two buffers alternate (a warp sends for column j after all have
//    sent for j - 1, that is after all have read j - 2);
//  * only the next column's entry is updated at once; the other columns lag by
//    one update, applied while the messages travel.  A candidate's row is sent
//    as it stands with its multiplier, and the receiver applies the update.
//  * one loop body for all columns: the registers move down by one column, a
//    finished entry goes to shared memory.  Unrolled over the columns the code
//    runs once per launch and waits for its own instructions.
// Per column at 1024 rows, in clocks: candidate 200, reciprocal and row 490,
// sending 620 (the messages' bytes), lagging updates 90 per column still to go
// (1500 on average), winner 360, update of the next column 430.  1024 rows, 32
// columns, eight matrices, cold: 67 us (lu_panel_split_kernel takes those now);
// with a cluster barrier per column, the
// winner's row read through distributed shared memory and the loop unrolled
// 122 us; in one CTA, the panel in global memory, 422.
struct PanelMsg {
  double row[kPanel];
  unsigned long long key;   // bits of |entry| + 1; 0: no candidate
  long long pos;
  double lprev, inv;        // its multiplier of the column before; 1 / entry
};
constexpr uint32_t kMsgBytes = sizeof(PanelMsg);

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t remote_u32(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send_2b64(uint32_t addr, ulonglong2 v, uint32_t bar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
          addr),
      "l"(v.x), "l"(v.y), "r"(bar)
      : "memory");
}
// 1 / d: the hardware's approximation (PTX: from the upper 20 mantissa bits, so
// good to 2^-19 or better) and one step of the cubic hyperpower iteration (M.
// Altman, Pacific J. Math. 10, 1960), x (1 + e + e^2) with e = 1 - d x, which
// leaves e^3 < 2^-57: the two roundings after it count, 1 ulp at most (tested).
// Three dependent operations, half the division's time on a column's critical
// chain.  Outside its range (subnormal, near overflow, zero, infinite) the
// division.
__device__ __forceinline__ double reciprocal(double d) {
  const int f = (__double2hiint(d) >> 20) & 0x7ff;
  if (f < 64 || f > 1980) return 1.0 / d;
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  const double e = fma(-d, x, 1.0);
  return fma(x, fma(e, e, e), x);
}
__device__ __forceinline__ bool panel_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 22); ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__global__ void __launch_bounds__(kPanelRows)
lu_panel_kernel(int n, int k0, int kb, double* __restrict__ A, int lda, long long sA,
                int* __restrict__ piv, long long sP, int* __restrict__ src, int* info, int istep,
                volatile unsigned* err) {
  constexpr int KB = kPanel;
  extern __shared__ __align__(16) unsigned char s_raw[];
  cg::cluster_group cl = cg::this_cluster();
  const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.x / cs;
  A += b * sA;
  piv += b * sP;
  src += (long long)b * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nmsg = cs * nw;
  PanelMsg* msg = reinterpret_cast<PanelMsg*>(s_raw);                     // [2][nmsg]
  PanelMsg& out = msg[2 * nmsg + warp];                                   // this warp's candidate
  double* us = reinterpret_cast<double*>(msg + 2 * nmsg + nw) + KB * warp;   // its pivot row
  // finished entries, [column][thread]
  double* fin = reinterpret_cast<double*>(msg + 2 * nmsg + nw) + KB * nw + threadIdx.x;
  __shared__ __align__(8) unsigned long long bars[2];
  const uint32_t bar0 = smem_u32(bars);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const int R = n - k0, r = rank * blockDim.x + threadIdx.x;
  const bool have = r < R;
  double a[KB];
  {
    const double* row = A + (long long)(k0 + (have ? r : 0)) * lda + k0;
#pragma unroll
    for (int c = 0; c < KB; ++c) a[c] = (have && c < kb) ? row[c] : 0.0;
  }
  int pos = have ? r : -1;   // -1: no row
  int first_zero = 0;
  double lp = 0.0, up = 0.0;        // pending: multiplier, pivot row (lane = column)
  bool pend = false, lag = false;   // any; for this row
  bool ok = true;
  uint32_t slot[8], rbar[8];   // this warp's message and the barriers in every CTA
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    slot[q] = remote_u32(smem_u32(&msg[rank * nw + warp]), q < cs ? q : 0) + 16 * lane;
    rbar[q] = remote_u32(bar0, q < cs ? q : 0);
  }
  cl.sync();   // the barriers are there
  // a[i]: column j + i
#pragma unroll 1
  for (int j = 0; j < kb && ok; ++j) {
    const int buf = j & 1;
    const uint32_t bar = bar0 + 8 * buf;
    if (threadIdx.x == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(nmsg * kMsgBytes)
                   : "memory");
    // the warp's candidate (NaNs are none)
    const unsigned long long bits =
        (unsigned long long)__double_as_longlong(a[0]) & 0x7fffffffffffffffULL;
    const bool cand = pos >= j && bits <= 0x7ff0000000000000ULL;
    const uint32_t hi = cand ? (uint32_t)(bits >> 32) + 1 : 0, lo = (uint32_t)bits;
    const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0);
    const int mp =
        __reduce_min_sync(0xffffffffu, (cand && hi == mh && lo == ml) ? pos : 0x7fffffff);
    if (cand && pos == mp) {
#pragma unroll
      for (int c = 0; c < KB; c += 2)
        *reinterpret_cast<double2*>(&out.row[c]) = make_double2(a[c], a[c + 1]);
      out.lprev = lp;
      out.inv = reciprocal(a[0]);
    }
    __syncwarp();
    {
      // 16 bytes per lane
      ulonglong2 v = reinterpret_cast<const ulonglong2*>(&out)[lane < 18 ? lane : 0];
      if (lane == 16) v = make_ulonglong2(mh ? (unsigned long long)mh << 32 | ml : 0, mp);
      const uint32_t off = buf * nmsg * kMsgBytes;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < cs && lane < 18) send_2b64(slot[q] + off, v, rbar[q] + 8 * buf);
    }
    // the update that columns j + 1 .. lag by
    if (pend) {
      const double ln = lag ? -lp : 0.0;
#pragma unroll
      for (int c4 = 0; c4 < KB; c4 += 4) {
        if (c4 >= KB - j) break;   // a branch: predicated off, the pipe is taken all the same
#pragma unroll
        for (int c = c4 ? c4 : 1; c < c4 + 4; ++c)
          if (lag) a[c] = fma(ln, us[c], a[c]);
      }
    }
    ok = panel_wait(bar, (uint32_t)(j >> 1) & 1);
    if (!__all_sync(0xffffffffu, ok)) {
      ok = false;
      if (lane == 0 && err) *err = 1;
      break;
    }
    // the winner: largest entry, then the first position
    const PanelMsg* m = msg + buf * nmsg;
    unsigned long long key = lane < nmsg ? m[lane].key : 0;
    int kp = lane < nmsg ? (int)m[lane].pos : 0x7fffffff, ki = lane;
    for (int q = lane + 32; q < nmsg; q += 32) {
      const unsigned long long qk = m[q].key;
      const int qp = (int)m[q].pos;
      if (qk > key || (qk == key && qp < kp)) {
        key = qk;
        kp = qp;
        ki = q;
      }
    }
    const uint32_t kh = (uint32_t)(key >> 32), kl = (uint32_t)key;
    const uint32_t wh = __reduce_max_sync(0xffffffffu, kh);
    const uint32_t wl = __reduce_max_sync(0xffffffffu, kh == wh ? kl : 0);
    const int wp = __reduce_min_sync(0xffffffffu, (kh == wh && kl == wl) ? kp : 0x7fffffff);
    const unsigned own = __ballot_sync(0xffffffffu, kh == wh && kl == wl && kp == wp);
    const int wi = __shfl_sync(0xffffffffu, ki, __ffs(own) - 1);
    // no key: every remaining entry of the column is NaN; the row at position j
    // is its own pivot, wherever it is held
    const int p = wh ? wp : j;
    const double ul = __shfl_down_sync(0xffffffffu, up, 1);   // of the column before
    double u, inv;
    if (wh) {
      u = m[wi].row[lane];
      inv = m[wi].inv;
      if (pend && lane > 0) u = fma(-m[wi].lprev, ul, u);
    } else {
      u = inv = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (rank == 0 && threadIdx.x == 0) piv[k0 + j] = k0 + p;
    // position swap j <-> p
    const bool retire = pos == p;
    if (pos == j) pos = p;
    if (retire) pos = j;
    // the pivot is zero when its key says so
    if (wh == 1 && wl == 0) {
      if (!first_zero) first_zero = k0 + j + 1;
      pend = lag = false;
    } else {
      up = u;
      pend = true;
      lag = pos > j;
      const double u1 = __shfl_sync(0xffffffffu, u, 1);
      __syncwarp();
      if (lane > 0) us[lane - 1] = u;   // for the next column's a[]
      __syncwarp();
      if (lag) {
        lp = a[0] * inv;
        a[0] = lp;
        a[1] = fma(-lp, u1, a[1]);
      }
    }
    fin[j * blockDim.x] = a[0];
#pragma unroll
    for (int c = 0; c + 1 < KB; ++c) a[c] = a[c + 1];
    a[KB - 1] = 0.0;
  }
  cl.sync();   // no CTA leaves while another may still write to its shared memory
  if (have) {
    double* row = A + (long long)(k0 + pos) * lda + k0;
    for (int c = 0; c < kb; ++c) row[c] = fin[c * blockDim.x];
    src[k0 + pos] = k0 + r;
  }
  if (rank == 0 && threadIdx.x == 0 && first_zero && info) atomicCAS(info + istep * b, 0, first_zero);
}

// The same for up to 1024 rows, four warps per 32 rows: warp g of them holds
// columns g, g + 4, .. of its rows, so that a column's lagging updates (72
// clocks of a scheduler's float64 pipe each) spread over the four schedulers.
// The warp of the pivot's column finds the candidate and shows the others its
// entries; each sends its eight columns of the candidate's row (one
// asynchronous store per lane serves all CTAs) and forms the multipliers
// itself once the winner is known.
// 256 rows, 32 columns: 63 -> 42 us (cold); over the panels of a 1024-row
// factorisation 61 -> 47 us on average, at 1024 rows the same (four warps per
// scheduler there).  More rows take the kernel above.
constexpr int kSplitRows = 1024;
__global__ void __launch_bounds__(512)
lu_panel_split_kernel(int n, int k0, int kb, double* __restrict__ A, int lda, long long sA,
                      int* __restrict__ piv, long long sP, int* __restrict__ src, int* info, int istep,
                      volatile unsigned* err) {
  constexpr int KB = kPanel, NC = KB / 4;   // columns per warp
  extern __shared__ __align__(16) unsigned char s_raw[];
  cg::cluster_group cl = cg::this_cluster();
  const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.x / cs;
  A += b * sA;
  piv += b * sP;
  src += (long long)b * n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nrg = blockDim.x >> 7, rg = warp >> 2, g = warp & 3;   // row and column groups
  const int nmsg = cs * nrg, rows = 32 * nrg;
  PanelMsg* msg = reinterpret_cast<PanelMsg*>(s_raw);   // [2][nmsg]
  PanelMsg& out = msg[2 * nmsg + rg];                   // this row group's candidate
  double* colv = reinterpret_cast<double*>(msg + 2 * nmsg + nrg);   // [2][rows]: pivot column
  double* us = colv + 2 * rows + NC * warp;             // pivot row, own columns
  double* fin = colv + 2 * rows + NC * 4 * nrg + 32 * rg + lane;    // finished: [column][row]
  __shared__ int4 s_cand[2][4];                         // key, position, lane
  __shared__ __align__(8) unsigned long long bars[2];
  const uint32_t bar0 = smem_u32(bars);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const int R = n - k0, r = rank * rows + 32 * rg + lane;
  const bool have = r < R;
  double a[NC];   // a[i]: column 4 (j4 + i) + g
  {
    const double* row = A + (long long)(k0 + (have ? r : 0)) * lda + k0;
#pragma unroll
    for (int i = 0; i < NC; ++i) a[i] = (have && 4 * i + g < kb) ? row[4 * i + g] : 0.0;
  }
  int pos = have ? r : -1;
  int first_zero = 0;
  double lp = 0.0, up = 0.0;        // pending: multiplier, pivot row (lane = own column)
  bool pend = false, lag = false;
  bool ok = true;
  // four lanes per CTA send 64 bytes of the row, two the rest of the message
  const uint32_t own = smem_u32(&msg[rank * nrg + rg]);
  const int to4 = lane >> 2, to2 = lane >> 1;
  const uint32_t row_to = remote_u32(own, to4 < cs ? to4 : 0) + 64 * g + 16 * (lane & 3);
  const uint32_t row_bar = remote_u32(bar0, to4 < cs ? to4 : 0);
  const uint32_t key_to = remote_u32(own, to2 < cs ? to2 : 0) + 8 * KB + 16 * (lane & 1);
  const uint32_t key_bar = remote_u32(bar0, to2 < cs ? to2 : 0);
  cl.sync();   // the barriers are there
#pragma unroll 1
  for (int j4 = 0; 4 * j4 < kb; ++j4) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int j = 4 * j4 + s;
      if (j >= kb) break;   // uniform
      if (!ok) {
        // given up: only the barriers, which know no limit, for the warps that
        // have not found out yet
        asm volatile("bar.sync %0, 128;" ::"r"(1 + rg) : "memory");
        continue;
      }
      const int buf = s & 1;
      const uint32_t bar = bar0 + 8 * buf;
      if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(nmsg * kMsgBytes)
                     : "memory");
      double pv = a[0];   // this row's entry of column j
      if (g == s) {
        // the row group's candidate (NaNs are none)
        const unsigned long long bits =
            (unsigned long long)__double_as_longlong(pv) & 0x7fffffffffffffffULL;
        const bool cand = pos >= j && bits <= 0x7ff0000000000000ULL;
        const uint32_t hi = cand ? (uint32_t)(bits >> 32) + 1 : 0, lo = (uint32_t)bits;
        const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
        const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0);
        const int mp =
            __reduce_min_sync(0xffffffffu, (cand && hi == mh && lo == ml) ? pos : 0x7fffffff);
        const unsigned at = __ballot_sync(0xffffffffu, cand && pos == mp);
        colv[buf * rows + 32 * rg + lane] = pv;
        if (lane == 0) s_cand[buf][rg] = make_int4((int)mh, (int)ml, mp, at ? __ffs(at) - 1 : -1);
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + rg) : "memory");
      const int4 cd = s_cand[buf][rg];
      if (g != s) pv = colv[buf * rows + 32 * rg + lane];
      if (lane == cd.w) {
#pragma unroll
        for (int i = 0; i < NC; i += 2)
          *reinterpret_cast<double2*>(&out.row[NC * g + i]) = make_double2(a[i], a[i + 1]);
        if (g == s) {
          out.lprev = lp;
          out.inv = reciprocal(pv);
        }
      }
      __syncwarp();
      const uint32_t off = buf * nmsg * kMsgBytes;
      if (to4 < cs)
        send_2b64(row_to + off,
                  reinterpret_cast<const ulonglong2*>(&out.row[NC * g])[lane & 3],
                  row_bar + 8 * buf);
      if (g == s && to2 < cs) {
        ulonglong2 v = reinterpret_cast<const ulonglong2*>(&out.lprev)[0];
        if ((lane & 1) == 0)
          v = make_ulonglong2(cd.x ? (unsigned long long)(uint32_t)cd.x << 32 | (uint32_t)cd.y : 0,
                              (unsigned long long)(long long)cd.z);
        send_2b64(key_to + off, v, key_bar + 8 * buf);
      }
      // the update that columns j + 1 .. lag by
      if (pend) {
        const double ln = lag ? -lp : 0.0;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          if (i >= NC - j4) break;
          if (i == 0 && g <= s) continue;
          if (lag) a[i] = fma(ln, us[i], a[i]);
        }
      }
      ok = panel_wait(bar, (uint32_t)(j >> 1) & 1);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        if (lane == 0 && err) *err = 1;
        continue;
      }
      // the winner: largest entry, then the first position
      const PanelMsg* m = msg + buf * nmsg;
      const unsigned long long key = lane < nmsg ? m[lane].key : 0;
      const int kp = lane < nmsg ? (int)m[lane].pos : 0x7fffffff;
      const uint32_t kh = (uint32_t)(key >> 32), kl = (uint32_t)key;
      const uint32_t wh = __reduce_max_sync(0xffffffffu, kh);
      const uint32_t wl = __reduce_max_sync(0xffffffffu, kh == wh ? kl : 0);
      const int wp = __reduce_min_sync(0xffffffffu, (kh == wh && kl == wl) ? kp : 0x7fffffff);
      const unsigned win = __ballot_sync(0xffffffffu, kh == wh && kl == wl && kp == wp);
      const int wi = __ffs(win) - 1;
      // no key: every remaining entry of the column is NaN; the row at position
      // j is its own pivot, wherever it is held
      const int p = wh ? wp : j;
      double u, inv;
      if (wh) {
        u = m[wi].row[NC * g + (lane & (NC - 1))];
        inv = m[wi].inv;
        if (pend && ((lane & (NC - 1)) > 0 || g > s)) u = fma(-m[wi].lprev, up, u);
      } else {
        u = inv = __longlong_as_double(0x7ff8000000000000LL);
      }
      if (rank == 0 && threadIdx.x == 0) piv[k0 + j] = k0 + p;
      // position swap j <-> p
      const bool retire = pos == p;
      if (pos == j) pos = p;
      if (retire) pos = j;
      // the pivot is zero when its key says so
      if (wh == 1 && wl == 0) {
        if (!first_zero) first_zero = k0 + j + 1;
        pend = lag = false;
      } else {
        up = u;
        pend = true;
        lag = pos > j;
        // the next column: s + 1's first, or group 0's second
        const int nx = s < 3 ? 0 : 1;
        const double u1 = __shfl_sync(0xffffffffu, u, nx);
        __syncwarp();
        // (the registers move down after s = 3)
        if (s < 3 ? lane < NC : (lane > 0 && lane < NC)) us[s < 3 ? lane : lane - 1] = u;
        __syncwarp();
        if (lag) {
          lp = pv * inv;
          if (g == s) a[0] = lp;
          if (g == ((s + 1) & 3)) a[nx] = fma(-lp, u1, a[nx]);
        }
      }
      if (g == s) fin[j * rows] = a[0];
    }
#pragma unroll
    for (int i = 0; i + 1 < NC; ++i) a[i] = a[i + 1];
    a[NC - 1] = 0.0;
    up = __shfl_down_sync(0xffffffffu, up, 1);
  }
  cl.sync();   // no CTA leaves while another may still write to its shared memory
  if (have) {
    double* row = A + (long long)(k0 + pos) * lda + k0;
#pragma unroll
    for (int i = 0; i < NC; ++i)
      if (4 * i + g < kb) row[4 * i + g] = fin[(4 * i + g) * rows];
    if (g == 0) src[k0 + pos] = k0 + r;
  }
  if (rank == 0 && threadIdx.x == 0 && first_zero && info) atomicCAS(info + istep * b, 0, first_zero);
}

// The panel's row swaps on every column outside it, from the net permutation
// (src[i]: the row that ends at row i): the kb top rows and the up to kb
// pivot rows below, all reads before the writes.  For columns k1 .. ct the top
// rows are then solved with the panel's unit lower triangle: a warp per
// column, lane = row, a finished entry broadcast by shuffle.  Eight columns
// per CTA: a step of a solve holds a quarter of the SM's float64 pipe for 72
// clocks (a column per lane instead, 32 per warp: 17 us for the 496 steps).
constexpr int kSwapCols = 8;
__global__ void __launch_bounds__(32 * kSwapCols)
lu_swap_trsm_kernel(int n, int k0, int kb, int ct, double* __restrict__ A, int lda, long long sA,
                    const int* __restrict__ piv, long long sP, const int* __restrict__ src) {
  A += blockIdx.y * sA;
  piv += blockIdx.y * sP;
  src += (long long)blockIdx.y * n;
  __shared__ double X[kPanel][kSwapCols + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k1 = k0 + kb;
  const int cb = blockIdx.x * kSwapCols;
  const bool solve = cb < ct && cb + kSwapCols > k1;   // uniform
  // L11: lane = row
  double l[kPanel];
  if (solve) {
#pragma unroll
    for (int r = 0; r < kPanel; ++r)
      l[r] = r < lane && lane < kb ? A[(long long)(k0 + lane) * lda + k0 + r] : 0.0;
  }
  const int i = threadIdx.x / kSwapCols, w = threadIdx.x % kSwapCols, c = cb + w;
  const bool on = i < kb && c < n && (c < k0 || c >= k1);
  double x = 0.0, y = 0.0;
  int to = -1;
  if (on) {
    const int rt = src[k0 + i];
    to = piv[k0 + i];
    x = A[(long long)rt * lda + c];
    if (to >= k1) y = A[(long long)src[to] * lda + c];
  }
  X[i][w] = x;
  __syncthreads();   // all reads before the writes
  if (on && to >= k1) A[(long long)to * lda + c] = y;
  const int cs = cb + warp;
  if (solve && cs >= k1 && cs < ct) {
    double v = X[lane][warp];
#pragma unroll
    for (int r = 0; r + 1 < kPanel; ++r) {
      const double xr = __shfl_sync(0xffffffffu, v, r);
      if (lane > r) v = fma(-l[r], xr, v);
    }
    X[lane][warp] = v;
  }
  __syncthreads();
  if (on) A[(long long)(k0 + i) * lda + c] = X[i][w];
}

// U12 = L11^{-1} A12 for the nb rows of an outer block, columns c0 .. n-1:
// eight columns per CTA (so a few hundred columns fill the GPU), the columns
// in shared memory, 32 rows at a time: the diagonal tile by one warp per
// column (lane = row, finished entries broadcast by shuffle), then the rows
// below it as products.  Float64-pipe bound: nb^2 / 2 FMA per column.
constexpr int kTrsmCols = 8;
__global__ void __launch_bounds__(256)
lu_block_trsm_kernel(int n, int k0, int nb, int c0, double* __restrict__ A, int lda,
                     long long sA) {
  A += blockIdx.y * sA;
  __shared__ double X[kOuter][kTrsmCols + 1];
  __shared__ double Lt[kPanel][kPanel + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cb = c0 + blockIdx.x * kTrsmCols, nc = min(kTrsmCols, n - cb);
  for (int e = tid; e < nb * kTrsmCols; e += 256) {
    const int i = e / kTrsmCols, c = e % kTrsmCols;
    X[i][c] = c < nc ? A[(long long)(k0 + i) * lda + cb + c] : 0.0;
  }
  for (int t0 = 0; t0 < nb; t0 += kPanel) {
    const int tn = min(kPanel, nb - t0);
    __syncthreads();
    for (int e = tid; e < tn * tn; e += 256) {
      const int i = e / tn, j = e - i * tn;
      Lt[i][j] = A[(long long)(k0 + t0 + i) * lda + k0 + t0 + j];
    }
    __syncthreads();
    {
      double x = lane < tn ? X[t0 + lane][warp] : 0.0;
      for (int i = 0; i < tn; ++i) {
        const double xi = __shfl_sync(0xffffffffu, x, i);
        if (lane > i && lane < tn) x = fma(-Lt[lane][i], xi, x);
      }
      if (lane < tn) X[t0 + lane][warp] = x;
    }
    __syncthreads();
    // rows below: thread = (row, column)
    const int c = tid & 7;
    for (int i = t0 + tn + (tid >> 3); i < nb; i += 32) {
      const double* l = A + (long long)(k0 + i) * lda + k0 + t0;
      double acc = X[i][c];
      if (tn == kPanel) {
#pragma unroll
        for (int j = 0; j < kPanel; ++j) acc = fma(-__ldg(l + j), X[t0 + j][c], acc);
      } else {
        for (int j = 0; j < tn; ++j) acc = fma(-__ldg(l + j), X[t0 + j][c], acc);
      }
      X[i][c] = acc;
    }
  }
  __syncthreads();
  for (int e = tid; e < nb * kTrsmCols; e += 256) {
    const int i = e / kTrsmCols, c = e % kTrsmCols;
    if (c < nc) A[(long long)(k0 + i) * lda + cb + c] = X[i][c];
  }
}

void launch_panel(cudaStream_t st, int n, int k0, int kb, double* A, int lda, long long sA,
                  int* piv, long long sP, int* src, int batch, int* info, int istep,
                  volatile unsigned* err) {
  const int R = n - k0;
  // 32 rows per CTA (four warps), then up to 128, in clusters of up to eight
  // (the portable size); above 1024 rows a thread per row
  const bool split = R <= kSplitRows;
  int cs = 1;
  while (cs < 8 && R > (split ? 32 : 128) * cs) cs *= 2;
  const int warps = ((R + cs - 1) / cs + 31) / 32;   // row groups of 32
  const int threads = 32 * warps * (split ? 4 : 1);
  if (threads > kPanelRows) {
    lu_panel_global_kernel<<<batch, 1024, 0, st>>>(n, k0, kb, A, lda, sA, piv, sP, src, info,
                                                   istep);
    check_launch("lu_panel_global_kernel");
    return;
  }
  // messages, (pivot column), pivot rows, finished entries
  const size_t sm = (size_t)(2 * cs * warps + warps) * sizeof(PanelMsg) +
                    8 * (size_t)warps * (kPanel + (split ? 64 : 0) + 32 * kPanel);
  auto kern = split ? lu_panel_split_kernel : lu_panel_kernel;
  ensure_smem(reinterpret_cast<const void*>(kern), sm);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(batch * cs));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SLU_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, n, k0, kb, A, lda, sA, piv, sP, src,
                                    info, istep, err));
  check_launch("lu_panel_kernel");
}

// ---------------------------------------------------------------- inverses
// Lp (np x np) = L with identity padding, Ut = U^T likewise (both lower
// triangular, zeros above); perm: the net row permutation of the pivots
// (P A = L U, (P A)_i = A_perm[i]), by one extra CTA per matrix.
__global__ void __launch_bounds__(256)
tri_pack_kernel(int n, int np, const double* __restrict__ LU, int lda, long long sA,
                const int* __restrict__ piv, long long sP, double* __restrict__ T,
                int* perm, int in_place) {
  const int b = blockIdx.z, tid = threadIdx.x;
  LU += b * sA;
  extern __shared__ int s_perm[];
  if (blockIdx.y == gridDim.y - 1) {
    if (blockIdx.x != 0) return;
    piv += b * sP;
    if (in_place) {   // too large for shared memory
      int* pm = perm + (long long)b * n;
      for (int i = tid; i < n; i += 256) pm[i] = i;
      __syncthreads();
      if (tid == 0)
        for (int i = 0; i < n; ++i) {
          const int p = piv[i], t = pm[i];
          pm[i] = pm[p];
          pm[p] = t;
        }
      return;
    }
    int* pv = s_perm + n;
    for (int i = tid; i < n; i += 256) {
      s_perm[i] = i;
      pv[i] = piv[i];
    }
    __syncthreads();
    if (tid == 0)
      for (int i = 0; i < n; ++i) {
        const int p = pv[i], t = s_perm[i];
        s_perm[i] = s_perm[p];
        s_perm[p] = t;
      }
    __syncthreads();
    for (int i = tid; i < n; i += 256) perm[(long long)b * n + i] = s_perm[i];
    return;
  }
  const long long nn = (long long)np * np;
  double* Lp = T + 2 * b * nn;
  double* Ut = Lp + nn;
  __shared__ double tile[32][33];
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32, tx = tid & 31, ty = tid >> 5;
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + r, j = j0 + tx;
    double v = 0.0;
    if (i < n && j < n) v = LU[(long long)i * lda + j];
    tile[r][tx] = v;
    if (i < np && j < np)
      Lp[(long long)i * np + j] = i == j ? 1.0 : (i > j && i < n ? v : 0.0);
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int i = j0 + r, j = i0 + tx;   // Ut[i][j] = U[j][i]
    if (i < np && j < np)
      Ut[(long long)i * np + j] =
          i < n ? (j <= i ? tile[tx][r] : 0.0) : (i == j ? 1.0 : 0.0);
  }
}

// In-place inverses of the w x w (w <= 32) diagonal blocks of lower triangular
// matrices: one warp per block, lane = column, forward substitution with the
// column in registers.
__global__ void __launch_bounds__(32)
tri_base_kernel(int np, int w, double* __restrict__ T) {
  double* D = T + (long long)blockIdx.y * np * np + (long long)blockIdx.x * w * (np + 1);
  __shared__ double L[32][33];
  const int lane = threadIdx.x;
  for (int i = 0; i < w; ++i)
    if (lane < w) L[i][lane] = D[(long long)i * np + lane];
  __syncwarp();
  const double rd = lane < w ? 1.0 / L[lane][lane] : 0.0;
  double x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const double ri = __shfl_sync(0xffffffffu, rd, i);
    double acc = i == lane ? 1.0 : 0.0;
    if (i < w) {
#pragma unroll
      for (int j = 0; j < i; ++j) acc = fma(-L[i][j], x[j], acc);
    }
    x[i] = acc * ri;
  }
  if (lane < w)
    for (int i = 0; i < w; ++i) {
      double v = 0.0;
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (q == i) v = x[q];
      D[(long long)i * np + lane] = v;
    }
}

// Y (np x n) = columns of X permuted: Y[:, perm[i]] = X[:, i]
__global__ void __launch_bounds__(256)
permute_cols_kernel(int n, int np, const double* __restrict__ X, long long sX,
                    const int* __restrict__ perm, double* __restrict__ Y, long long sY) {
  X += blockIdx.z * sX;
  Y += blockIdx.z * sY;
  perm += (long long)blockIdx.z * n;
  const int r = blockIdx.y;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += 256 * gridDim.x)
    Y[(long long)r * n + perm[i]] = X[(long long)r * np + i];
}

}  // namespace

void lu_factor(Handle& h, int n, double* A, int lda, long long sA, int* piv, long long sP,
               int batch, int* info, int istep) {
  if (n <= 0 || batch <= 0) return;
  constexpr int kMaxBatch = 65535;   // matrices of a launch (grid dimensions)
  if (batch > kMaxBatch) {
    for (int b0 = 0; b0 < batch; b0 += kMaxBatch)
      lu_factor(h, n, A + b0 * sA, lda, sA, piv + b0 * sP, sP, std::min(kMaxBatch, batch - b0),
                info ? info + (long long)istep * b0 : nullptr, istep);
    return;
  }
  cudaStream_t st = h.stream;
  Scratch scratch(h.lu_ws, st);
  scratch.w.reserve(sizeof(int) * (size_t)n * batch + 256, st);
  int* src = scratch.w.take<int>((size_t)n * batch);
  for (int K0 = 0; K0 < n; K0 += kOuter) {
    const int K1 = std::min(K0 + kOuter, n);
    for (int k0 = K0; k0 < K1; k0 += kPanel) {
      const int kb = std::min(kPanel, K1 - k0), k1 = k0 + kb;
      launch_panel(st, n, k0, kb, A, lda, sA, piv, sP, src, batch, info, istep,
                   h.err_word());
      if (n > kb) {
        lu_swap_trsm_kernel<<<dim3((n + kSwapCols - 1) / kSwapCols, batch), 32 * kSwapCols, 0, st>>>(
            n, k0, kb, K1, A, lda, sA, piv, sP, src);
        check_launch("lu_swap_trsm_kernel");
      }
      if (k1 < K1)
        gemm_batched<double>(st, false, false, n - k1, K1 - k1, kb, -1.0,
                             A + (long long)k1 * lda + k0, lda, sA, 0,
                             A + (long long)k0 * lda + k1, lda, sA, 0, 1.0,
                             A + (long long)k1 * lda + k1, lda, sA, 0, batch);
    }
    if (K1 < n) {
      lu_block_trsm_kernel<<<dim3((n - K1 + kTrsmCols - 1) / kTrsmCols, batch), 256, 0, st>>>(
          n, K0, K1 - K0, K1, A, lda, sA);
      check_launch("lu_block_trsm_kernel");
      gemm_f64(h, false, false, n - K1, n - K1, K1 - K0, -1.0, A + (long long)K1 * lda + K0, lda,
               sA, 0, A + (long long)K0 * lda + K1, lda, sA, 0, 1.0, A + (long long)K1 * lda + K1,
               lda, sA, 0, batch);
    }
  }
}

// Inv = U^{-1} L^{-1} P.  L and U^T are inverted together by doubling: blocks
// of at most 32 rows by substitution, then for pairs of inverted neighbours
// the off-diagonal block becomes -C^{-1} (B A^{-1}), two batched products per
// level over every pair of both triangles of all matrices; the last product
// joins them.  ~log2(n / 32) levels of wide products instead of n / 32
// dependent substitution steps (against the identity, by 32-row tiles, eight
// 1024 blocks took 18 ms; the inverses of a whole 8 x 1024 red-black
// factorisation, 15 blocks, now take about 3 ms).
void lu_inverse(Handle& h, int n, const double* LU, int lda, long long sA, const int* piv,
                long long sP, double* Inv, int ldi, long long sI, int batch) {
  if (n <= 0 || batch <= 0) return;
  cudaStream_t st = h.stream;
  int q = 0;
  while (((n + (1 << q) - 1) >> q) > 32) ++q;
  const int w = (n + (1 << q) - 1) >> q, np = w << q;
  const size_t nn = (size_t)np * np;
  const size_t per = 8 * (3 * nn + (size_t)np * n) + sizeof(int) * (size_t)n + 4 * 256;
  const int fit = (int)std::max<size_t>(1, std::min<size_t>(Handle::kScratchMax / per, 65535 >> (q + 1)));
  for (int b0 = 0; b0 < batch; b0 += fit) {
    const int nb = std::min(fit, batch - b0);
    Scratch scratch(h.lu_ws, st);
    Workspace& ws = scratch.w;
    ws.reserve(per * nb + 4096, st);
    double* T = ws.take<double>(2 * nn * nb);
    double* W = ws.take<double>(nn * nb);
    double* LP = ws.take<double>((size_t)np * n * nb);
    int* perm = ws.take<int>((size_t)n * nb);
    const int in_place = 2 * sizeof(int) * (size_t)n > 200 * 1024;
    const size_t sm = in_place ? 0 : 2 * sizeof(int) * (size_t)n;
    ensure_smem(reinterpret_cast<const void*>(tri_pack_kernel), sm);
    const int tl = (np + 31) / 32;
    tri_pack_kernel<<<dim3(tl, tl + 1, nb), 256, sm, st>>>(n, np, LU + b0 * sA, lda, sA,
                                                           piv + b0 * sP, sP, T, perm,
                                                           in_place);
    check_launch("tri_pack_kernel");
    tri_base_kernel<<<dim3(1 << q, 2 * nb), 32, 0, st>>>(np, w, T);
    check_launch("tri_base_kernel");
    for (int s = w; s < np; s *= 2) {
      const int pairs = np / (2 * s);
      const long long sd = 2LL * s * (np + 1), ss = (long long)s * s;
      double* B = T + (long long)s * np;           // below the first block of a pair
      double* C = T + (long long)s * (np + 1);     // the second block
      gemm_f64(h, false, false, s, s, s, 1.0, B, np, sd, (long long)nn, T, np, sd, (long long)nn,
               0.0, W, s, ss, ss * pairs, pairs, 2 * nb);
      gemm_f64(h, false, false, s, s, s, -1.0, C, np, sd, (long long)nn, W, s, ss, ss * pairs, 0.0,
               B, np, sd, (long long)nn, pairs, 2 * nb);
    }
    permute_cols_kernel<<<dim3(std::min((n + 255) / 256, 8), np, nb), 256, 0, st>>>(
        n, np, T, 2 * (long long)nn, perm, LP, (long long)np * n);
    check_launch("permute_cols_kernel");
    gemm_f64(h, true, false, n, n, np, 1.0, T + nn, np, 2 * (long long)nn, 0, LP, n,
             (long long)np * n, 0, 0.0, Inv + b0 * sI, ldi, sI, 0, nb);
  }
}

}  // namespace slu
