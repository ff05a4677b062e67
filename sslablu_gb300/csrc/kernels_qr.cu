// Householder QR panels, reflector application and one-sided Jacobi SVD.
//
// These implement the per-block LAPACK work of the HBS compression and ULV
// factorisation:
//   * complete QR of each sketch block Om_blk^T and the projection of Y onto
//     the trailing columns of Q (matAssembly/HBS/HBSnew.py:20-28 compute_UV),
//     which also yields Y*Q_1 and R for the right pseudo-inverse solves of
//     construct_D / block_solve_r (HBSnew.py:11-19, 48-62);
//   * the SVD whose leading left singular vectors become U (HBSnew.py:27);
//   * complete QR of V (W1, ULVsparse.py:18-25) and square QR of D*W
//     (ULVsparse.py:51-61).
// Reflectors follow the LAPACK geqrf convention (beta = -sign(alpha)*norm,
// v[0] = 1), so the trailing columns of Q match LAPACK's to rounding.
#include <cooperative_groups.h>

#include <algorithm>

#include "slablu_internal.cuh"

namespace cg = cooperative_groups;

namespace slu {
namespace {

__device__ inline double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ inline double block_sum(double v, double* red) {
  v = warp_sum(v);
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  double t = 0.0;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}

// QR of the first nfac columns of an m x ncol column-major work array `a`
// (leading dimension lda), applying each reflector to every later column.
__device__ void panel_qr_dev(int m, int nfac, int ncol, double* a, int lda, double* tau) {
  __shared__ double red[32];
  __shared__ double s_tau, s_scale;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int j = 0; j < nfac && j < m; ++j) {
    double* col = a + (long long)j * lda;
    double ss = 0.0;
    for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) ss += col[i] * col[i];
    ss = block_sum(ss, red);
    if (threadIdx.x == 0) {
      double alpha = col[j];
      if (ss == 0.0) {
        s_tau = 0.0;
        s_scale = 0.0;
      } else {
        double beta = -copysign(sqrt(alpha * alpha + ss), alpha);
        s_tau = (beta - alpha) / beta;
        s_scale = 1.0 / (alpha - beta);
        col[j] = beta;
      }
      tau[j] = s_tau;
    }
    __syncthreads();
    const double t = s_tau, sc = s_scale;
    if (t != 0.0)
      for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) col[i] *= sc;
    __syncthreads();
    if (t != 0.0) {
      for (int c = j + 1 + warp; c < ncol; c += nwarps) {
        double* cc = a + (long long)c * lda;
        double d = (lane == 0) ? cc[j] : 0.0;
        for (int i = j + 1 + lane; i < m; i += 32) d += col[i] * cc[i];
        d = warp_sum(d) * t;
        if (lane == 0) cc[j] -= d;
        for (int i = j + 1 + lane; i < m; i += 32) cc[i] -= d * col[i];
      }
    }
    __syncthreads();
  }
}

// Panels too large for one CTA's shared memory, in global memory.
__global__ void __launch_bounds__(512)
panel_qr_kernel(int m, int nfac, int ncol, double* __restrict__ W, int ldw, long long sW,
                double* __restrict__ tau, long long sTau, double* __restrict__ W2,
                double* __restrict__ tau2, int nsplit) {
  // blocks nsplit.. work on the second batch (W2, tau2), same shapes
  const bool second = (int)blockIdx.x >= nsplit;
  const long long b = second ? blockIdx.x - nsplit : blockIdx.x;
  panel_qr_dev(m, nfac, ncol, (second ? W2 : W) + b * sW, ldw, (second ? tau2 : tau) + b * sTau);
}

// C <- Q C (transpose = false) or Q^T C for tall columns; each warp owns whole
// columns of C.
__global__ void __launch_bounds__(256)
apply_q_kernel(bool transpose, int m, int k, const double* __restrict__ V, int ldv, long long sV,
               const double* __restrict__ tau, long long sTau, double* __restrict__ C, int ldc,
               long long sC, int nc) {
  V += blockIdx.y * sV;
  tau += blockIdx.y * sTau;
  C += blockIdx.y * sC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int c = blockIdx.x * nwarps + warp;
  if (c >= nc) return;
  double* cc = C + (long long)c * ldc;
  for (int s = 0; s < k; ++s) {
    const int j = transpose ? s : (k - 1 - s);
    const double t = tau[j];
    if (t == 0.0) continue;
    const double* v = V + (long long)j * ldv;
    double d = (lane == 0) ? cc[j] : 0.0;
    for (int i = j + 1 + lane; i < m; i += 32) d += v[i] * cc[i];
    d = warp_sum(d) * t;
    if (lane == 0) cc[j] -= d;
    for (int i = j + 1 + lane; i < m; i += 32) cc[i] -= d * v[i];
    __syncwarp();
  }
}

// ---------------------------------------------------------------- float64 economy
// One warp instruction on the float64 pipe takes 64 clocks of its SM
// sub-partition, so scalars are formed from bit patterns and float32 seeds.
__device__ __forceinline__ uint32_t hi32(double v) { return (uint32_t)__double2hiint(v); }
// mantissa in [1, 2) as a float32 (the leading 23 bits)
__device__ __forceinline__ float mantissa(double v) {
  return __uint_as_float(0x3f800000u | (hi32(v) & 0xfffffu) << 3 |
                         (uint32_t)__double2loint(v) >> 29);
}
__device__ __forceinline__ int expo(double v) { return (int)(hi32(v) >> 20 & 0x7ff); }
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
// float32 -> float64 on the integer units (normal numbers and zero)
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f), mag = u & 0x7fffffffu;
  const uint32_t h = mag < 0x00800000u ? 0u : (mag >> 3) + 0x38000000u;
  return __hiloint2double((int)((u & 0x80000000u) | h),
                          mag < 0x00800000u ? 0 : (int)(u << 29));
}

template <int LANES>
__device__ __forceinline__ double lanes_sum(double v, uint32_t mask) {
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// 1 / sqrt(t): float32 seed (relative error below 2^-21, with the mantissa cut to
// 23 bits) and one step of Householder's iteration of third order (The Numerical
// Treatment of a Single Nonlinear Equation, 1970), y (1 + r / 2 + 3 r^2 / 8) with
// r = 1 - t y^2: 5 r^3 / 16 < 2^-60 before the roundings; t positive, finite and
// normal
__device__ __forceinline__ double inv_sqrt(double t) {
  const int e = expo(t) - 1023, e2 = e & ~1;
  const double q = __hiloint2double((int)hi32(t) - (e2 << 20), __double2loint(t));   // in [1, 4)
  const double y = widen(rsqrtf(mantissa(t) * (float)(1 + (e & 1))));
  const double r = fma(-q * y, y, 1.0);
  const double z = fma(y * r, fma(0.375, r, 0.5), y);
  return __hiloint2double((int)hi32(z) - (e2 / 2 << 20), __double2loint(z));
}
// 1 / q by the cubic hyperpower iteration (M. Altman, Pacific J. Math. 10, 1960):
// z (1 + r + r^2), r = 1 - q z; q positive, finite and normal, 1 / q normal
__device__ __forceinline__ double inv_pos(double q) {
  const int e = expo(q) - 1023;
  const double m = __hiloint2double((int)hi32(q) - (e << 20), __double2loint(q));   // in [1, 2)
  const double z = widen(__frcp_rn(mantissa(q)));
  const double r = fma(-m, z, 1.0);
  const double w = fma(z, fma(r, r, r), z);
  return __hiloint2double((int)hi32(w) - (e << 20), __double2loint(w));
}

// Householder reflector of a column with diagonal entry alpha and ss the sum
// of squares below it: v = (v0, rest), H = I - f v v^T, new diagonal beta.
struct Reflector {
  double v0, f, beta, tau, sc;   // tau, sc = 1 / v0: the LAPACK form (v[0] = 1)
};
__device__ __forceinline__ Reflector make_reflector(double alpha, double ss) {
  Reflector h{0.0, 0.0, alpha, 0.0, 0.0};
  if (ss == 0.0) return h;
  const double t = fma(alpha, alpha, ss);
  const int e = expo(t);
  if (e > 1023 - 900 && e < 1023 + 900) {
    const double y = inv_sqrt(t), nrm = t * y;
    h.beta = -copysign(nrm, alpha);
    h.v0 = alpha - h.beta;
    const double a = fabs(h.v0);
    h.f = inv_pos(nrm * a);
    h.tau = a * y;
    h.sc = copysign(nrm * h.f, h.v0);
  } else {   // near the ends of the range, or not finite
    h.beta = -copysign(sqrt(t), alpha);
    h.v0 = alpha - h.beta;
    h.tau = -h.v0 / h.beta;
    h.sc = 1.0 / h.v0;
    h.f = h.tau * h.sc * h.sc;
  }
  return h;
}

// ---------------------------------------------------------------- clusters
// Sums over the CTAs of a cluster: every CTA sends its terms to the others with
// asynchronous stores that complete on the receiver's mbarrier, and adds all
// of them in the same order, so all CTAs hold the same values.  Two
// buffers alternate; a warp sends for one exchange after it has read the one
// before, so nobody overwrites what is still to be read.
template <int C>
struct Exchange {
  double* buf;         // [2][C][terms]
  int terms, rank;
  uint32_t bar;        // two mbarriers
  int n = 0;           // exchanges so far
  __device__ void init(double* b, int t, int r, unsigned long long* bars) {
    buf = b;
    terms = t;
    rank = r;
    bar = static_cast<uint32_t>(__cvta_generic_to_shared(bars));
    if (threadIdx.x == 0) {
      for (int i = 0; i < 2; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * i) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cg::this_cluster().sync();
  }
  __device__ double* slot(int r, int i) const { return buf + ((n & 1) * C + r) * terms + i; }
  // one thread per CTA: `count` terms from the other CTAs are to come
  __device__ void expect(int count) const {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar + 8 * (n & 1)),
                 "r"(count * 8)
                 : "memory");
  }
  __device__ void send(int i, double v) const {
    *slot(rank, i) = v;
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(slot(rank, i)));
#pragma unroll
    for (int q = 1; q < C; ++q) {
      const int to = (rank + q) % C;
      uint32_t d, b;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(to));
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(bar + 8 * (n & 1)), "r"(to));
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                       d),
                   "l"(__double_as_longlong(v)), "r"(b)
                   : "memory");
    }
  }
  __device__ bool wait() const {
    for (int i = 0; i < (1 << 22); ++i) {
      uint32_t done;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(done)
          : "r"(bar + 8 * (n & 1)), "r"((uint32_t)(n >> 1) & 1)
          : "memory");
      if (done) return true;
    }
    return false;
  }
  __device__ double sum(int i) const {
    double v[C];
#pragma unroll
    for (int r = 0; r < C; ++r) v[r] = *slot(r, i);
#pragma unroll
    for (int h = 1; h < C; h *= 2)
#pragma unroll
      for (int r = 0; r + h < C; r += 2 * h) v[r] += v[r + h];
    return v[0];
  }
};

// ---------------------------------------------------------------- panels in shared memory
// QR of an m x n column-major panel, one CTA, the panel in shared memory
// (column stride ld, 8 mod 16: the 2 x 8 entries of a wavefront hit distinct
// banks).  Warp 0 carries the chain: it applies reflector j to column j + 1
// with all its lanes and forms reflector j + 1 at once; meanwhile the other
// warps apply reflector j to the columns after it, eight lanes per column
// (three butterfly additions per product instead of five).  One barrier per
// column.  Bound by the float64 pipe for wide panels, by warp 0's chain of
// ~50 float64 instructions per column for the last ones.
// 128 panels of 261 x 64 with 64 carried columns: 0.40 ms, and 0.64 for the
// carried ones (apply_q_reg_kernel); 1.71 by panel_qr_kernel in global memory.
__global__ void __launch_bounds__(512)
panel_qr_smem_kernel(int m, int n, double* __restrict__ W, int ldw, long long sW,
                     double* __restrict__ tau, long long sTau, int ld, double* __restrict__ W2,
                     double* __restrict__ tau2, int nsplit) {
  extern __shared__ double sm[];
  double* s_sc = sm + (size_t)ld * n;   // n: 1 / v0
  __shared__ double s_v0[2], s_f[2];
  const bool second = (int)blockIdx.x >= nsplit;
  const long long b = second ? blockIdx.x - nsplit : blockIdx.x;
  double* w = (second ? W2 : W) + b * sW;
  double* tg = (second ? tau2 : tau) + b * sTau;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  for (int c = warp; c < n; c += nwarps)
    for (int i = lane; i < m; i += 32) sm[(size_t)c * ld + i] = w[(long long)c * ldw + i];
  __syncthreads();
  const int steps = min(n, m);
  // reflector of column j from its entries below the diagonal (warp 0)
  auto reflect = [&](int j) {
    double* col = sm + (size_t)j * ld;
    double ss = 0.0, s1 = 0.0;
    int i = j + 1 + lane;
    for (; i + 32 < m; i += 64) {
      ss = fma(col[i], col[i], ss);
      s1 = fma(col[i + 32], col[i + 32], s1);
    }
    if (i < m) ss = fma(col[i], col[i], ss);
    ss = warp_sum(ss + s1);
    const Reflector h = make_reflector(col[j], ss);
    __syncwarp();
    if (lane == 0) {
      s_v0[j & 1] = h.v0;
      s_f[j & 1] = h.f;
      s_sc[j] = h.sc;
      col[j] = h.beta;
      tg[j] = h.tau;
    }
  };
  if (warp == 0) reflect(0);
  __syncthreads();
  for (int j = 0; j < steps; ++j) {
    const double* v = sm + (size_t)j * ld;
    const double v0 = s_v0[j & 1], f = s_f[j & 1];
    if (warp == 0) {
      if (j + 1 < n) {
        double* cc = sm + (size_t)(j + 1) * ld;
        if (f != 0.0) {
          double d = lane == 0 ? v0 * cc[j] : 0.0, d1 = 0.0;
          int i = j + 1 + lane;
          for (; i + 32 < m; i += 64) {
            d = fma(v[i], cc[i], d);
            d1 = fma(v[i + 32], cc[i + 32], d1);
          }
          if (i < m) d = fma(v[i], cc[i], d);
          d = f * warp_sum(d + d1);
          for (i = j + 1 + lane; i < m; i += 32) cc[i] = fma(-d, v[i], cc[i]);
          if (lane == 0) cc[j] = fma(-d, v0, cc[j]);
          __syncwarp();
        }
        if (j + 1 < steps) reflect(j + 1);
      }
    } else if (f != 0.0) {
      const int part = lane & 7, per = 4 * (nwarps - 1);
      for (int c0 = j + 2; c0 < n; c0 += per) {
        const int c = c0 + 4 * (warp - 1) + (lane >> 3);
        if (c0 + 4 * (warp - 1) >= n) break;   // uniform
        const bool on = c < n;
        double* cc = sm + (size_t)(on ? c : j) * ld;
        const int i0 = ((j + 1) & ~7) + part;
        double d = part == 0 ? v0 * cc[j] : 0.0, d1 = 0.0;
        int i = i0 > j ? i0 : i0 + 8;
        const int first = i;
        for (; i + 8 < m; i += 16) {
          d = fma(v[i], cc[i], d);
          d1 = fma(v[i + 8], cc[i + 8], d1);
        }
        if (i < m) d = fma(v[i], cc[i], d);
        d = f * lanes_sum<8>(d + d1, 0xffffffffu);
        if (on) {
#pragma unroll 4
          for (i = first; i < m; i += 8) cc[i] = fma(-d, v[i], cc[i]);
          if (part == 0) cc[j] = fma(-d, v0, cc[j]);
        }
      }
    }
    __syncthreads();
  }
  for (int c = warp; c < n; c += nwarps) {
    const double sc = c < steps ? s_sc[c] : 0.0;
    for (int i = lane; i < m; i += 32) {
      const double x = sm[(size_t)c * ld + i];
      w[(long long)c * ldw + i] = (i > c && sc != 0.0) ? x * sc : x;
    }
  }
}

// The same by a cluster of C CTAs per panel where there are few of them: each
// CTA holds its rows of every column, four lanes per column.  Per column one
// exchange: the partial products of the column with itself and all later ones,
// and from the owner of the diagonal that row; every thread forms the
// reflector's v0 and f, and the updates are local.  The float64 pipe of one SM
// bounds panel_qr_smem_kernel (a 261 x 64 panel 360 us, alone or one of 128);
// here up to 38 panels take 268 us (four CTAs each): 2K clocks of a column the
// reflector, 1.2K the exchange.
// A thread's entries (at most R of its column) stay in registers between the
// product and the update; a multiplication of a warp takes 72 clocks however
// few of its lanes it serves, so rows that are done are branched over.
template <int C, int R>
__global__ void __launch_bounds__(256)
panel_qr_cluster_kernel(int m, int n, double* __restrict__ W, int ldw, long long sW,
                        double* __restrict__ tau, long long sTau, int ld, double* __restrict__ W2,
                        double* __restrict__ tau2, int nsplit, int* info) {
  extern __shared__ double sm[];
  double* s_sc = sm + (size_t)ld * n;   // n: 1 / v0
  __shared__ __align__(8) unsigned long long s_bar[2];
  __shared__ double s_v0, s_f;
  const int prob = blockIdx.x / C, rank = (int)blockIdx.x % C;
  const bool second = prob >= nsplit;
  const long long b = second ? prob - nsplit : prob;
  double* w = (second ? W2 : W) + b * sW;
  double* tg = (second ? tau2 : tau) + b * sTau;
  Exchange<C> ex;
  ex.init(s_sc + n, 2 * n, rank, s_bar);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int part = tid & 3, group = tid >> 2, ngroups = blockDim.x >> 2;
  const int mr = (m + C - 1) / C, own0 = rank * mr, ml = max(0, min(m - own0, mr));
  for (int c = warp; c < n; c += nwarps)
    for (int i = lane; i < ml; i += 32) sm[(size_t)c * ld + i] = w[(long long)c * ldw + own0 + i];
  __syncthreads();
  const int steps = min(n, m);
  bool failed = false;
  for (int j = 0; j < steps && !failed; ++j) {
    const int owner = j / mr, lj = j - own0;   // lj: local row of the diagonal, in its owner
    const double* v = sm + (size_t)j * ld;
    if (tid == 0) ex.expect((C - 1) * (n - j) + (rank != owner ? n - j : 0));
    // rows lo .. ml - 1 are below the diagonal: entries u0 .. u1 - 1
    const int lo = max(0, lj + 1), u0 = lo >> 2, u1 = (ml + 3) >> 2;
    double y[R], x[R];   // the column's entries and the first product's
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = 4 * u + part;
      y[u] = i >= lo && i < ml ? v[i] : 0.0;
    }
    for (int c0 = j; c0 < n; c0 += ngroups) {
      const int c = c0 + group;
      const bool on = c < n;
      if (c0 + (group & ~7) >= n) break;   // the whole warp
      const double* cc = sm + (size_t)(on ? c : j) * ld;
      double z[R], d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int i = 4 * u + part;
        z[u] = i >= lo && i < ml ? cc[i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        if (u < u0) continue;
        if (u >= u1) break;
        d[u & 3] = fma(y[u], z[u], d[u & 3]);
      }
      const double s = lanes_sum<4>((d[0] + d[1]) + (d[2] + d[3]), 0xffffffffu);
      if (on && part == 0) {
        ex.send(c, s);
        if (rank == owner) ex.send(n + c, cc[lj]);
      }
      if (c0 == j) {
#pragma unroll
        for (int u = 0; u < R; ++u) x[u] = z[u];
      }
    }
    failed = __syncthreads_or(!ex.wait()) != 0;   // (and the own terms are there)
    if (failed) break;
    // warp 0 forms the reflector, the others add up their products meanwhile
    const int c1 = j + group;   // the column whose entries are in x
    const bool on1 = group > 0 && c1 < n;
    const double r1 = on1 ? *ex.slot(owner, n + c1) : 0.0, d1 = on1 ? ex.sum(c1) : 0.0;
    if (warp == 0) {
      const Reflector h = make_reflector(*ex.slot(owner, n + j), ex.sum(j));
      if (lane == 0) {
        s_v0 = h.v0;
        s_f = h.f;
        s_sc[j] = h.sc;
        if (rank == owner) {
          tg[j] = h.tau;
          sm[(size_t)j * ld + lj] = h.beta;
        }
      }
    }
    __syncthreads();
    const double v0 = s_v0, f = s_f;
    if (f != 0.0) {
      for (int c0 = j; c0 < n; c0 += ngroups) {
        const int c = c0 + group;
        if (c0 + (group & ~7) >= n) break;
        const bool on = c > j && c < n;
        double* cc = sm + (size_t)(on ? c : j) * ld;
        double rc = r1, t = d1;
        if (c0 > j && on) {
          rc = *ex.slot(owner, n + c);
          t = ex.sum(c);
#pragma unroll
          for (int u = 0; u < R; ++u) {
            const int i = 4 * u + part;
            x[u] = i >= lo && i < ml ? cc[i] : 0.0;
          }
        }
        t = f * fma(v0, rc, t);
#pragma unroll
        for (int u = 0; u < R; ++u) {
          if (u < u0) continue;
          if (u >= u1) break;
          const int i = 4 * u + part;
          const double q = fma(-t, y[u], x[u]);
          if (on && i >= lo && i < ml) cc[i] = q;
        }
        if (rank == owner && part == 0 && on) cc[lj] = fma(-t, v0, rc);
      }
    }
    ++ex.n;
    __syncthreads();
  }
  if (tid == 0 && failed && info) atomicCAS(info, 0, 1);
  for (int c = warp; c < n; c += nwarps) {
    const double sc = c < steps ? s_sc[c] : 0.0;
    for (int i = lane; i < ml; i += 32) {
      const double x = sm[(size_t)c * ld + i];
      w[(long long)c * ldw + own0 + i] = (own0 + i > c && sc != 0.0) ? x * sc : x;
    }
  }
  cg::this_cluster().sync();   // nobody sends to a CTA that has left
}

// C <- Q^T C (transpose) or Q C for the m x k reflectors of a factored panel,
// columns of C in registers (eight lanes per column, RPL rows each), the
// reflectors through shared memory kRefl at a time with their unit diagonal
// and the zeros above it.  Few problems spread their columns over more CTAs.
// Bound by the float64 pipe (2 FMA per row, reflector and column).
constexpr int kRefl = 16;
template <int RPL>
__global__ void __launch_bounds__(512)
apply_q_reg_kernel(bool transpose, int m, int k, const double* __restrict__ V, int ldv,
                   long long sV, const double* __restrict__ tau, long long sTau,
                   double* __restrict__ C, int ldc, long long sC, int nc,
                   const double* __restrict__ V2, const double* __restrict__ tau2,
                   double* __restrict__ C2, int nsplit) {
  extern __shared__ double sv[];   // kRefl x 8 RPL
  __shared__ double st[kRefl];
  const bool second = (int)blockIdx.y >= nsplit;
  const long long b = second ? blockIdx.y - nsplit : blockIdx.y;
  V = (second ? V2 : V) + b * sV;
  tau = (second ? tau2 : tau) + b * sTau;
  C = (second ? C2 : C) + b * sC;
  constexpr int P = 8 * RPL;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int part = lane & 7, c = (blockIdx.x * nwarps + warp) * 4 + (lane >> 3);
  const bool on = c < nc;
  double* cc = C + (long long)(on ? c : 0) * ldc;
  double x[RPL];
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = part + 8 * i;
    x[i] = (on && r < m) ? cc[r] : 0.0;
  }
  const int chunks = (k + kRefl - 1) / kRefl;
  for (int q = 0; q < chunks; ++q) {
    const int j0 = (transpose ? q : chunks - 1 - q) * kRefl, nj = min(kRefl, k - j0);
    __syncthreads();
    for (int e = tid; e < nj * P; e += blockDim.x) {
      const int jj = e / P, r = e - jj * P, j = j0 + jj;
      sv[e] = r < j ? 0.0 : (r == j ? 1.0 : (r < m ? V[(long long)j * ldv + r] : 0.0));
    }
    if (tid < nj) st[tid] = tau[j0 + tid];
    __syncthreads();
    for (int s = 0; s < nj; ++s) {
      const int jj = transpose ? s : nj - 1 - s;
      const double t = st[jj];
      if (t == 0.0) continue;   // uniform
      const double* v = sv + jj * P + part;
      double d[2] = {0.0, 0.0};
#pragma unroll
      for (int i = 0; i < RPL; ++i)
        if (8 * i + 7 >= j0) d[i & 1] = fma(v[8 * i], x[i], d[i & 1]);
      const double g = t * lanes_sum<8>(d[0] + d[1], 0xffffffffu);
#pragma unroll
      for (int i = 0; i < RPL; ++i)
        if (8 * i + 7 >= j0) x[i] = fma(-g, v[8 * i], x[i]);
    }
  }
  if (!on) return;
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = part + 8 * i;
    if (r < m) cc[r] = x[i];
  }
}

// ---------------------------------------------------------------- Jacobi SVD
// One-sided (Hestenes) Jacobi on the columns of A (m x n), round-robin pair
// ordering.  A column pair belongs to LANES consecutive lanes of a warp; a
// lane owns rows part, part + LANES, ... of both columns, in registers from
// the inner product to the rotation (RPL rows; RPL = 0: more rows than
// registers, read twice).
//
// Bound by the float64 pipe: one warp instruction per 64 clocks and SM
// sub-partition, so what counts is float64 instructions per round, and
// everything that need not be float64 runs on the integer and float32 units:
//   * the squared column norms are kept in shared memory and updated by the
//     rotation (exact for whatever angle is taken; recomputed each sweep, and
//     at once where a norm falls by cancellation), so a round forms one inner
//     product instead of three;
//   * the convergence test and the rotation angle come from the bit patterns
//     of the norms and the inner product (exponents as integers, mantissas as
//     float32).  An angle good to 1e-6 still cuts the inner product by that
//     factor per rotation, and the test (|gamma| <= m eps sqrt(alpha beta)
//     for every pair) needs no more;
//   * the rotation is applied as three shears (x -= tau y, y += s x,
//     x -= tau y; tau = tan(theta / 2), s = 2 tau / (1 + tau^2) to float64
//     rounding), three FMAs per row instead of two and two products; it is
//     orthogonal to float64 rounding whatever the angle.
// 64 x 64: 82 float64 instructions per round and warp; with float64 angles
// and three inner products 160 (128 problems: 10.99 -> 5.76 ms).
// Before the sweeps, A^T P = Q R by Householder QR with column pivoting (in
// shared memory): the left singular vectors of A are those of R^T with their
// rows permuted, and the columns of R^T, graded and nearly orthogonal, need
// 8-9 sweeps where those of a sketch block need 18-25 (Z. Drmac and K.
// Veselic, SIAM J. Matrix Anal. Appl. 29, 2008).  The QR costs about one
// sweep; 128 problems of 64 x 64: 5.76 -> 2.17 ms.
// Columns live in shared memory with an odd leading dimension.  At
// convergence the columns are sigma_j u_j; the r largest are normalised and
// written as U (m x r).
constexpr int JAC_MAX_SWEEPS = 40;

// Rotation of a pair with squared norms al, be and inner product ga: false
// where the pair is orthogonal to |ga| <= tol sqrt(al be) (tol2 = tol^2).
__device__ __forceinline__ bool jac_angle(double al, double be, double ga, float tol2, double& tau,
                                          double& s) {
  const int eg = expo(ga), ea = expo(al), eb = expo(be);
  const uint32_t gbits = (hi32(ga) & 0x7fffffffu) | (uint32_t)__double2loint(ga);
  if (gbits == 0 || eg == 0x7ff || ea == 0x7ff || eb == 0x7ff) return false;
  const float mg = mantissa(ga);
  const float q = mg * mg / (mantissa(al) * mantissa(be));
  if (q * pow2f(min(max(2 * eg - ea - eb, -120), 60)) <= tol2) return false;
  const double d = be - al;
  const int ez = expo(d) - eg - 1;   // exponent of zeta = d / (2 ga)
  if (ez > 100) {   // t below 2^-100: t = s = ga / d, c = 1
    s = ga / d;
    tau = 0.5 * s;
    return s != 0.0;
  }
  const float az = expo(d) == 0 ? 0.f : __fdividef(mantissa(d), mg) * pow2f(max(ez, -100));
  const float t = az > 1e9f ? __fdividef(0.5f, az)
                            : __fdividef(1.0f, az + sqrtf(fmaf(az, az, 1.0f)));
  const float h = __fdividef(t, 1.0f + sqrtf(fmaf(t, t, 1.0f)));   // tan(theta / 2) <= 0.42
  const uint32_t neg = (hi32(d) ^ hi32(ga)) & 0x80000000u;
  const float hs = __uint_as_float(__float_as_uint(h) | (az == 0.f ? 0u : neg));
  tau = widen(hs);
  // s = 2 tau / (1 + tau^2): float32 reciprocal and one cubic Newton step
  const double u = fma(tau, tau, 1.0);
  const double r0 = widen(__frcp_rn(fmaf(hs, hs, 1.0f)));
  const double e = fma(-u, r0, 1.0);
  s = (tau + tau) * fma(r0, fma(e, e, e), r0);
  return true;
}

// |v| as a float32 relative to 2^(E0 - 1023), E0 the largest exponent field
// (20 mantissa bits; below 2^-126 of it: 0): pivot choices on the integer and
// float32 units.
__device__ __forceinline__ float rough(double v, int E0) {
  const int h = (int)(hi32(v) & 0x7fffffffu) - ((E0 - 126) << 20);
  return h > 0 ? __int_as_float(h << 3) : 0.f;
}

// Householder QR with column pivoting of the nr x nc array b (column-major,
// leading dimension ld) in shared memory by the whole block; perm[c] = the
// original column.  R is left on and above the diagonal.  LANES lanes share
// a column; the reflector is not normalised (H = I - f v v^T).
template <int LANES>
__device__ void pivoted_qr_dev(int nr, int nc, double* b, int ld, int* perm, float* vn, int E0) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int part = tid & (LANES - 1), group = tid / LANES, ngroups = blockDim.x / LANES;
  __shared__ double s_beta;
  for (int c0 = 0; c0 < nc; c0 += ngroups) {
    const int c = c0 + group;
    float v = 0.f;
    if (c < nc)
      for (int i = part; i < nr; i += LANES) {
        const float f = rough(b[(long long)c * ld + i], E0);
        v = fmaf(f, f, v);
      }
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (part == 0 && c < nc) vn[c] = v;
  }
  for (int c = tid; c < nc; c += blockDim.x) perm[c] = c;
  __syncthreads();
  const int steps = min(nr, nc);
  for (int j = 0; j < steps; ++j) {
    // largest remaining column (every warp on its own; NaN norms never win)
    uint32_t best = 0;
    for (int c = j + lane; c < nc; c += 32) best = max(best, __float_as_uint(fmaxf(vn[c], 0.f)));
    best = __reduce_max_sync(0xffffffffu, best);
    int p = nc;
    for (int c = j + lane; c < nc; c += 32)
      if (__float_as_uint(fmaxf(vn[c], 0.f)) == best) p = min(p, c);
    p = __reduce_min_sync(0xffffffffu, p);
    if (p >= nc) p = j;
    __syncthreads();
    double* bj = b + (long long)j * ld;
    if (p != j) {
      double* bp = b + (long long)p * ld;
      for (int i = tid; i < nr; i += blockDim.x) {
        const double t = bj[i];
        bj[i] = bp[i];
        bp[i] = t;
      }
      if (tid == 0) {
        const int t = perm[j];
        perm[j] = perm[p];
        perm[p] = t;
        vn[p] = vn[j];
      }
      __syncthreads();
    }
    double ss = 0.0;
    for (int i = j + 1 + lane; i < nr; i += 32) ss = fma(bj[i], bj[i], ss);
    ss = warp_sum(ss);
    const double alpha = bj[j], t = fma(alpha, alpha, ss);
    // nothing below the diagonal (or not finite): no reflection
    const bool reflect = ss > 0.0 && t < 1e300;
    double f = 0.0, v0 = 0.0;
    if (reflect) {
      const double nrm = sqrt(t);
      v0 = alpha + copysign(nrm, alpha);
      f = 1.0 / (nrm * fabs(v0));
      if (tid == 0) s_beta = -copysign(nrm, alpha);
    }
    // columns j + 1 .., several per pass
    for (int c0 = j + 1; c0 < nc; c0 += ngroups) {
      const int c = c0 + group;
      const bool on = c < nc;
      double* bc = b + (long long)(on ? c : j) * ld;
      const int i0 = j + 1 + ((part - (j + 1)) & (LANES - 1));
      double d0 = 0.0, d1 = 0.0;
      if (on && reflect) {
        int i = i0;
        for (; i + LANES < nr; i += 2 * LANES) {
          d0 = fma(bj[i], bc[i], d0);
          d1 = fma(bj[i + LANES], bc[i + LANES], d1);
        }
        if (i < nr) d0 = fma(bj[i], bc[i], d0);
        if (part == 0) d1 = fma(v0, bc[j], d1);
      }
      const double w = f * lanes_sum<LANES>(d0 + d1, 0xffffffffu);
      float v = 0.f;
      if (on) {
        for (int i = i0; i < nr; i += LANES) {
          const double x = reflect ? fma(-w, bj[i], bc[i]) : bc[i];
          if (reflect) bc[i] = x;
          const float r = rough(x, E0);
          v = fmaf(r, r, v);
        }
        if (part == 0 && reflect) bc[j] = fma(-w, v0, bc[j]);
      }
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (on && part == 0) vn[c] = v;
    }
    __syncthreads();
    if (tid == 0 && reflect) bj[j] = s_beta;
  }
  __syncthreads();
}

constexpr int JAC_THREADS = 512;
constexpr int JAC_CLUSTER_THREADS = 320;   // of a CTA where several share a problem
// ld: column stride of the shared array, cols its columns (see jacobi_smem);
// pre: QR preconditioning first.
// C > 1 (with pre): a cluster of C CTAs per problem.  Each does the whole QR
// and then keeps its own rows of every column: a round is the partial inner
// products, one exchange of them, the angles (in every CTA) and the rotation
// of the own rows.  The float64 pipe of one SM bounds a round of 64 columns
// of 64 rows (83 instructions of 72 clocks per warp); with four CTAs it is 37
// and the exchange.  64 x 64, up to 38 problems: 2140 -> 1390 us, up to 76 with
// two CTAs 1580; 80 x 80: 3640 -> 2210.
template <int LANES, int RPL, int C>
__global__ void __launch_bounds__(C > 1 ? JAC_CLUSTER_THREADS : JAC_THREADS)
jacobi_kernel(int m, int n_in, const double* __restrict__ A, int lda, long long sA, int r,
              double* __restrict__ U, int ldu, long long sU, double* __restrict__ sv,
              long long sS, int* info, int lower, const double* __restrict__ A2,
              double* __restrict__ U2, int nsplit, int ld, int cols, int pre) {
  extern __shared__ double sm[];
  const int n = pre ? min(m, n_in) : n_in;   // columns of the sweeps
  const int np = n + (n & 1);            // even number of columns (a zero pad column)
  const int lda_s = ld;
  double* a = sm;                        // column-major, column c at a + c * lda_s
  double* nrm = a + (long long)lda_s * cols;   // np: squared norms, then norms
  int* order = reinterpret_cast<int*>(nrm + cols);   // np
  int* rows = order + cols;                          // m: row i of the sweeps = row rows[i] of A
  __shared__ int s_rot, s_e0;
  __shared__ __align__(8) unsigned long long s_bar[2];
  // problems nsplit.. are the second batch (A2 -> U2), same shapes
  const int prob = blockIdx.x / C, rank = C > 1 ? (int)blockIdx.x % C : 0;
  const bool second = prob >= nsplit;
  const long long bi = second ? prob - nsplit : prob;
  Exchange<C> ex;
  if constexpr (C > 1) {
    ex.init(reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(rows + m) + 15) &
                                      ~uintptr_t(15)),
            np, rank, s_bar);
  }
  A = (second ? A2 : A) + bi * sA;
  if (pre) {
    // columns of A^T = rows of A; with `lower`, only A's lower triangle is read
    if (threadIdx.x == 0) s_e0 = 0;
    __syncthreads();
    int e0 = 0;
    for (int e = threadIdx.x; e < m * n_in; e += blockDim.x) {
      const int i = e / n_in, c = e - i * n_in;
      const double v = (!lower || c <= i) ? A[(long long)i * lda + c] : 0.0;
      a[(long long)i * lda_s + c] = v;
      e0 = max(e0, expo(v));
    }
    atomicMax(&s_e0, e0);
    __syncthreads();
    pivoted_qr_dev<LANES>(n_in, m, a, lda_s, rows, reinterpret_cast<float*>(nrm),
                          max(s_e0, 127));
    // R^T in place: column j, rows i >= j, from row j of R; zeros above
    for (int e = threadIdx.x; e < m * n; e += blockDim.x) {
      const int i = e / n, j = e - i * n;
      if (i > j) {
        const double v = a[(long long)i * lda_s + j];
        a[(long long)j * lda_s + i] = v;
        if (i < np) a[(long long)i * lda_s + j] = 0.0;
      }
    }
    __syncthreads();
    if (np > n)
      for (int i = threadIdx.x; i < m; i += blockDim.x) a[(long long)n * lda_s + i] = 0.0;
  } else {
    for (long long e = threadIdx.x; e < (long long)m * np; e += blockDim.x) {
      int c = (int)(e / m), i = (int)(e % m);
      // A row-major; with `lower`, only its lower triangle (c <= i) is read
      a[(long long)c * lda_s + i] =
          (c < n && (!lower || c <= i)) ? A[(long long)i * lda + c] : 0.0;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const float tolf = 2.220446049250313e-16f * (float)m, tol2 = tolf * tolf;
  const int npairs = np / 2, ring = np - 1;
  const int part = threadIdx.x & (LANES - 1), group = threadIdx.x / LANES;
  const int ngroups = blockDim.x / LANES;
  const uint32_t gmask = LANES == 32 ? 0xffffffffu
                                     : ((1u << LANES) - 1) << (lane & ~(LANES - 1));
  // own rows of every column
  const int mr = (m + C - 1) / C, own0 = rank * mr, ml = C > 1 ? max(0, min(m - own0, mr)) : m;
  double* al0 = a + own0;
  bool failed = false;   // a wait ran out (the same on all threads)
  // squared norms of all columns
  auto norms = [&]() {
    if (C > 1 && threadIdx.x == 0) ex.expect((C - 1) * np);
    // (loops of the same length on every lane: the whole warp joins the sums)
    for (int c0 = 0; c0 < np; c0 += ngroups) {
      const int c = c0 + group;
      double v = 0.0;
      if (c < np) {
        const double* ac = al0 + (long long)c * lda_s;
        for (int i = part; i < ml; i += LANES) v = fma(ac[i], ac[i], v);
      }
      v = lanes_sum<LANES>(v, 0xffffffffu);
      if (part == 0 && c < np) {
        if constexpr (C > 1) ex.send(c, v);
        else nrm[c] = v;
      }
    }
    if constexpr (C > 1) {
      // (the barrier: the own terms are there too)
      failed = __syncthreads_or(!ex.wait()) != 0;
      for (int c = threadIdx.x; c < np; c += blockDim.x) nrm[c] = ex.sum(c);
      __syncthreads();
      ++ex.n;
    }
  };
  int sweep = 0;
  for (; sweep < JAC_MAX_SWEEPS; ++sweep) {
    norms();
    if (threadIdx.x == 0) s_rot = 0;
    __syncthreads();
    if (C > 1 && failed) break;
    for (int rnd = 0; rnd < ring; ++rnd) {
      bool fresh = false, late = false;
      if (C > 1 && threadIdx.x == 0) ex.expect((C - 1) * npairs);
      for (int p0 = 0; p0 < npairs; p0 += ngroups) {
        // circle method: slot 0 fixed, others rotate
        const bool on = p0 + group < npairs;
        const int pi = on ? p0 + group : 0;
        int p = pi - 1 + rnd, q = np - 2 - pi + rnd;
        p = pi == 0 ? 0 : 1 + (p >= ring ? p - ring : p);
        q = 1 + (q >= ring ? q - ring : q);
        double* ap = al0 + (long long)p * lda_s;
        double* aq = al0 + (long long)q * lda_s;
        double x[RPL > 0 ? RPL : 1], y[RPL > 0 ? RPL : 1];
        double g[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (RPL > 0) {
#pragma unroll
          for (int i = 0; i < RPL; ++i) {
            const int row = part + LANES * i;
            x[i] = row < ml ? ap[row] : 0.0;
            y[i] = row < ml ? aq[row] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < RPL; ++i) g[i & 3] = fma(x[i], y[i], g[i & 3]);
        } else {
          for (int row = part; row < ml; row += LANES) g[0] = fma(ap[row], aq[row], g[0]);
        }
        double ga = RPL > 2 ? (g[0] + g[2]) + (g[1] + g[3]) : g[0] + g[1];
        ga = lanes_sum<LANES>(ga, 0xffffffffu);
        if constexpr (C > 1) {
          // (ngroups >= npairs: one pass)
          if (on && part == 0) ex.send(pi, ga);
          late = !ex.wait();
          __syncwarp();
          ga = ex.sum(pi);
        }
        const double al = nrm[p], be = nrm[q];
        double tau, s;
        if (!on || !jac_angle(al, be, ga, tol2, tau, s)) continue;
        double na = 0.0, nb = 0.0;
        if constexpr (RPL > 0) {
#pragma unroll
          for (int i = 0; i < RPL; ++i) {
            const int row = part + LANES * i;
            x[i] = fma(-tau, y[i], x[i]);
            y[i] = fma(s, x[i], y[i]);
            x[i] = fma(-tau, y[i], x[i]);
            if (row < ml) {
              ap[row] = x[i];
              aq[row] = y[i];
            }
          }
        } else {
          for (int row = part; row < ml; row += LANES) {
            double xv = ap[row], yv = aq[row];
            xv = fma(-tau, yv, xv);
            yv = fma(s, xv, yv);
            xv = fma(-tau, yv, xv);
            ap[row] = xv;
            aq[row] = yv;
          }
        }
        // |x'|^2 = al + s (s (be - al) - 2 c ga), c = 1 - tau s
        const double c = fma(-tau, s, 1.0);
        const double w = s * fma(s, be - al, -(c + c) * ga);
        na = al + w;
        nb = be - w;
        // a norm that fell by cancellation has lost its digits: form it anew
        // (the whole group sees the same values)
        if constexpr (C > 1) {
          if ((int)hi32(na) < 0 || expo(na) < expo(al) - 3 || (int)hi32(nb) < 0 ||
              expo(nb) < expo(be) - 3)
            fresh = true;   // after the round, for all columns
        } else if ((int)hi32(na) < 0 || expo(na) < expo(al) - 3) {
          na = 0.0;
          if constexpr (RPL > 0) {
#pragma unroll
            for (int i = 0; i < RPL; ++i) na = fma(x[i], x[i], na);
          } else {
            for (int row = part; row < m; row += LANES) na = fma(ap[row], ap[row], na);
          }
          na = lanes_sum<LANES>(na, gmask);
        }
        if (C == 1 && ((int)hi32(nb) < 0 || expo(nb) < expo(be) - 3)) {
          nb = 0.0;
          if constexpr (RPL > 0) {
#pragma unroll
            for (int i = 0; i < RPL; ++i) nb = fma(y[i], y[i], nb);
          } else {
            for (int row = part; row < m; row += LANES) nb = fma(aq[row], aq[row], nb);
          }
          nb = lanes_sum<LANES>(nb, gmask);
        }
        if (part == 0) {
          nrm[p] = na;
          nrm[q] = nb;
          s_rot = 1;
        }
      }
      if constexpr (C > 1) {
        // decisions by the barrier itself, the same on all threads
        const bool act = __syncthreads_or(fresh || late) != 0;
        ++ex.n;
        if (act) {
          failed = __syncthreads_or(late) != 0;
          if (failed) break;
          norms();
          if (failed) break;
        }
      } else {
        __syncthreads();
      }
    }
    if (!s_rot || (C > 1 && failed)) break;
    __syncthreads();
  }
  if (threadIdx.x == 0 && (sweep >= JAC_MAX_SWEEPS || failed) && info)
    atomicCAS(info, 0, 1);
  // column norms
  if constexpr (C > 1) {
    __syncthreads();
    if (!failed) norms();
    __syncthreads();
    for (int c = threadIdx.x; c < np; c += blockDim.x) nrm[c] = sqrt(nrm[c]);
  } else {
    for (int c = warp; c < np; c += nwarps) {
      double s = 0.0;
      for (int i = lane; i < m; i += 32)
        s += a[(long long)c * lda_s + i] * a[(long long)c * lda_s + i];
      s = warp_sum(s);
      if (lane == 0) nrm[c] = sqrt(s);
    }
  }
  __syncthreads();
  // rank of each column by decreasing norm (ties by index).  A NaN norm
  // (non-finite input) ranks below every number, so the ranks stay a
  // permutation and every order[] slot is written
  for (int c = threadIdx.x; c < np; c += blockDim.x) {
    int rk = 0;
    const double v = nrm[c] == nrm[c] ? nrm[c] : -1.0;
    for (int o = 0; o < np; ++o) {
      const double w = nrm[o] == nrm[o] ? nrm[o] : -1.0;
      rk += (w > v) || (w == v && o < c);
    }
    order[rk] = c;
  }
  __syncthreads();
  double* Ub = (second ? U2 : U) + bi * sU;
  double* svb = (sv && !second) ? sv + bi * sS : nullptr;
  const double smax = nrm[order[0]];
  const double tiny = (smax > 0.0) ? smax * 1e-150 : 1e-300;
  // normalised leading columns; columns that carry no direction are
  // completed below
  for (int j = warp; j < r; j += nwarps) {
    const int c = min(max(order[j < np ? j : np - 1], 0), np - 1);
    double s = nrm[c];
    if (svb && lane == 0 && rank == 0) svb[j] = (j < n) ? s : 0.0;
    bool ok = (j < n) && s > tiny;
    for (int i = own0 + lane; i < own0 + ml; i += 32)
      Ub[(long long)(pre ? rows[i] : i) * ldu + j] = ok ? a[(long long)c * lda_s + i] / s : 0.0;
  }
  __syncthreads();
  // completion by unit vectors, orthogonalised against the columns before
  // (classical Gram-Schmidt twice, over the whole block).  Every boundary
  // coupling of a red-black level is a zero block, so this is no rare case.
  // A unit vector once rejected stays rejected (its residual only shrinks as
  // columns join), so each is tried once: the compression of a zero 512-point
  // block (rank 24) takes 9 ms where retrying all of them for every column
  // took 30.
  if constexpr (C > 1) {
    // all rows are written; nothing is sent any more
    cg::this_cluster().sync();
    if (rank != 0) return;
  }
  int j0 = 0;
  while (j0 < r && j0 < n && nrm[min(max(order[j0 < np ? j0 : np - 1], 0), np - 1)] > tiny) ++j0;
  __syncthreads();
  double* v = a;        // candidate (the columns are no longer needed)
  double* d = a + m;    // its products with the columns before
  double thr = 0.5;
  int cand = 0;
  for (int j = j0; j < r; ++j) {
    for (;;) {
      if (cand >= m) {
        // fewer than r unit vectors leave half their length outside: some
        // vector still has 1 / sqrt(m) of it
        if (thr < 0.5) break;
        thr = 0.5 / sqrt((double)m);
        cand = 0;
      }
      for (int i = threadIdx.x; i < m; i += blockDim.x) v[i] = (i == cand) ? 1.0 : 0.0;
      __syncthreads();
      for (int pass = 0; pass < 2; ++pass) {
        for (int q = warp; q < j; q += nwarps) {
          double s = 0.0;
          for (int i = lane; i < m; i += 32) s = fma(Ub[(long long)i * ldu + q], v[i], s);
          s = warp_sum(s);
          if (lane == 0) d[q] = s;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
          double x = v[i];
          for (int q = 0; q < j; ++q) x = fma(-d[q], Ub[(long long)i * ldu + q], x);
          v[i] = x;
        }
        __syncthreads();
      }
      double s = 0.0;
      for (int i = lane; i < m; i += 32) s = fma(v[i], v[i], s);
      s = sqrt(warp_sum(s));
      ++cand;
      if (s > thr) {
        for (int i = threadIdx.x; i < m; i += blockDim.x) Ub[(long long)i * ldu + j] = v[i] / s;
        break;
      }
      __syncthreads();
    }
    __syncthreads();
  }
}
// Compact WY form of a factored panel of jb reflectors (LAPACK larft,
// forward, columnwise): Vc (jb x mp, row-major) holds the reflectors with
// their unit diagonal and zeros above it written out, and T (jb x jb, upper)
// satisfies H_0 H_1 ... H_{jb-1} = I - V T V^T (V = Vc^T).  One CTA per
// matrix; the panel is read from the column-major work array (column a at
// P + a * ldw, rows 0..mp-1 relative to the panel's diagonal).
constexpr int kWY = 32;   // panel width of the blocked QR
__global__ void __launch_bounds__(256)
wy_kernel(int mp, int jb, const double* __restrict__ P, int ldw, long long sW,
          const double* __restrict__ tau, long long sTau, double* __restrict__ Vc, long long sV,
          double* __restrict__ T, long long sT) {
  __shared__ double G[kWY][kWY + 1];
  __shared__ double Ts[kWY][kWY + 1];
  const long long b = blockIdx.x;
  P += b * sW;
  tau += b * sTau;
  Vc += b * sV;
  T += b * sT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (long long e = threadIdx.x; e < (long long)jb * mp; e += blockDim.x) {
    const int a = (int)(e / mp), r = (int)(e - (long long)a * mp);
    Vc[e] = r < a ? 0.0 : (r == a ? 1.0 : P[(long long)a * ldw + r]);
  }
  // G(a, c) = v_a . v_c for a < c: v_c starts at row c (unit), v_a there
  // holds P(a, c) (a < c), both below
  for (int q = warp; q < jb * jb; q += nwarps) {
    const int a = q / jb, c = q - a * jb;
    if (a >= c) continue;
    double d = 0.0;
    for (int r = c + 1 + lane; r < mp; r += 32)
      d += P[(long long)a * ldw + r] * P[(long long)c * ldw + r];
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) G[a][c] = d + P[(long long)a * ldw + c];
  }
  __syncthreads();
  // T(i, i) = tau_i; T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i), one column
  // at a time by the first warp (lane r owns row r)
  if (warp == 0) {
    for (int i = 0; i < jb; ++i) {
      const double ti = tau[i];
      double v = 0.0;
      if (lane < i) {
        for (int c = lane; c < i; ++c) v += Ts[lane][c] * G[c][i];
        v *= -ti;
      }
      __syncwarp();
      if (lane < i) Ts[lane][i] = v;
      if (lane == i) Ts[i][i] = ti;
      if (lane > i && lane < jb) Ts[lane][i] = 0.0;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < jb * jb; e += blockDim.x) T[e] = Ts[e / jb][e % jb];
}

}  // namespace

size_t qr_blocked_ws_elems(int m, int ncol, int batch) {
  return (size_t)batch * ((size_t)kWY * m + (size_t)kWY * kWY + 2 * (size_t)ncol * kWY) + 64;
}

void qr_blocked(cudaStream_t st, int m, int nfac, int ncol, double* W, int ldw, long long sW,
                double* tau, long long sTau, int batch, double* ws) {
  if (batch <= 0 || m <= 0 || nfac <= 0) return;
  if (nfac <= 2 * kWY) {
    panel_qr(st, m, nfac, ncol, W, ldw, sW, tau, sTau, batch);
    return;
  }
  SLU_REQUIRE(ws, "qr_blocked: workspace missing");
  const long long sV = (long long)kWY * m, sT = (long long)kWY * kWY, sX = (long long)ncol * kWY;
  double* Vc = ws;
  double* T = Vc + batch * sV;
  double* X1 = T + batch * sT;
  double* X2 = X1 + batch * sX;
  const int nf = std::min(nfac, m);
  for (int j0 = 0; j0 < nf; j0 += kWY) {
    const int jb = std::min(kWY, nf - j0), mp = m - j0;
    double* Pj = W + (long long)j0 * ldw + j0;
    panel_qr(st, mp, jb, jb, Pj, ldw, sW, tau + j0, sTau, batch);
    const int nc = ncol - j0 - jb;
    if (nc <= 0) continue;
    wy_kernel<<<batch, 256, 0, st>>>(mp, jb, Pj, ldw, sW, tau + j0, sTau, Vc, sV, T, sT);
    check_launch("wy_kernel");
    // trailing columns C (mp x nc, column-major: C^T row-major with ld ldw)
    // <- Q^T C, i.e. C^T <- C^T - (C^T V) T V^T
    double* Ct = Pj + (long long)jb * ldw;
    gemm_batched<double>(st, false, true, nc, jb, mp, 1.0, Ct, ldw, sW, 0, Vc, mp, sV, 0, 0.0, X1,
                         jb, sX, 0, batch);
    gemm_batched<double>(st, false, false, nc, jb, jb, 1.0, X1, jb, sX, 0, T, jb, sT, 0, 0.0, X2,
                         jb, sX, 0, batch);
    gemm_batched<double>(st, false, false, nc, mp, jb, -1.0, X2, jb, sX, 0, Vc, mp, sV, 0, 1.0, Ct,
                         ldw, sW, 0, batch);
  }
}

namespace {

template <int RPL>
void launch_apply(cudaStream_t st, bool transpose, int m, int k, const double* V, int ldv,
                  long long sV, const double* tau, long long sTau, double* C, int ldc,
                  long long sC, int nc, const double* V2, const double* tau2, double* C2,
                  int nsplit, int batch) {
  // up to 16 warps (64 columns) per CTA, fewer while SMs would stay empty
  int warps = std::min(16, (nc + 3) / 4);
  while (warps > 2 && (long long)batch * ((nc + 4 * warps - 1) / (4 * warps)) < num_sms())
    warps = (warps + 1) / 2;
  const size_t sm = sizeof(double) * kRefl * 8 * RPL;
  auto kern = apply_q_reg_kernel<RPL>;
  ensure_smem(reinterpret_cast<const void*>(kern), sm);
  kern<<<dim3((nc + 4 * warps - 1) / (4 * warps), batch), 32 * warps, sm, st>>>(
      transpose, m, k, V, ldv, sV, tau, sTau, C, ldc, sC, nc, V2, tau2, C2, nsplit);
  check_launch("apply_q_reg_kernel");
}

// Rows that eight lanes hold in registers; taller columns stay in memory.
constexpr int kApplyRows = 320;
// Rows from which few panels are shared by clusters of eight or four CTAs.  At
// 64 rows the exchange and the reflector of a column take as long as one CTA's
// column; with two CTAs per panel of 261 x 64 nothing is gained (398 -> 385 us).
constexpr int kClusterRows = 128;

void apply_q_dispatch(cudaStream_t st, bool transpose, int m, int k, const double* V, int ldv,
                      long long sV, const double* tau, long long sTau, double* C, int ldc,
                      long long sC, int nc, const double* V2, const double* tau2, double* C2,
                      int nsplit, int batch) {
#define SLU_APPLY(R)                                                                           \
  return launch_apply<R>(st, transpose, m, k, V, ldv, sV, tau, sTau, C, ldc, sC, nc, V2, tau2, \
                         C2, nsplit, batch)
  if (m <= 32) SLU_APPLY(4);
  if (m <= 64) SLU_APPLY(8);
  if (m <= 96) SLU_APPLY(12);
  if (m <= 128) SLU_APPLY(16);
  if (m <= 192) SLU_APPLY(24);
  if (m <= 264) SLU_APPLY(33);
  SLU_APPLY(40);
#undef SLU_APPLY
}

// One or two (W2 != W) batches of panels.  The factored columns in shared
// memory where they fit, the carried columns afterwards from registers; else
// everything by the one-CTA kernel in global memory.
void panel_qr_any(cudaStream_t st, int m, int nfac, int ncol, double* W, double* W2, int ldw,
                  long long sW, double* tau, double* tau2, long long sTau, int batch, int total,
                  int* info) {
  if (info && m >= kClusterRows && 4LL * total <= num_sms()) {
    const int C = 8LL * total <= num_sms() ? 8 : 4;
    const int mr = (m + C - 1) / C, ldc = (mr + 11) / 16 * 16 + 4;   // >= mr, 4 mod 16
    const size_t smc = sizeof(double) * ((size_t)ldc * nfac + nfac + 4 * (size_t)C * nfac);
    const int rl = (mr + 3) / 4;   // rows per lane
    if (rl <= 17 && smc <= 220 * 1024 && (ncol == nfac || m <= kApplyRows)) {
      auto kern = C == 8 ? (rl <= 9 ? panel_qr_cluster_kernel<8, 9> : panel_qr_cluster_kernel<8, 17>)
                         : (rl <= 9 ? panel_qr_cluster_kernel<4, 9> : panel_qr_cluster_kernel<4, 17>);
      ensure_smem(reinterpret_cast<const void*>(kern), smc);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(total * C));
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = smc;
      cfg.stream = st;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)C;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      SLU_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, m, nfac, W, ldw, sW, tau, sTau, ldc, W2, tau2,
                                        batch, info));
      check_launch("panel_qr_cluster_kernel");
      if (ncol > nfac)
        apply_q_dispatch(st, true, m, std::min(nfac, m), W, ldw, sW, tau, sTau,
                         W + (long long)nfac * ldw, ldw, sW, ncol - nfac, W2, tau2,
                         W2 + (long long)nfac * ldw, batch, total);
      return;
    }
  }
  const int ld = (m + 7) / 16 * 16 + 8;   // >= m, 8 mod 16
  const size_t sm = sizeof(double) * ((size_t)ld * nfac + nfac);
  if (sm <= 220 * 1024 && (ncol == nfac || m <= kApplyRows)) {
    ensure_smem(reinterpret_cast<const void*>(panel_qr_smem_kernel), sm);
    const int warps = std::min(16, std::max(2, 1 + (nfac + 3) / 4));
    panel_qr_smem_kernel<<<total, 32 * warps, sm, st>>>(m, nfac, W, ldw, sW, tau, sTau, ld, W2,
                                                        tau2, batch);
    check_launch("panel_qr_smem_kernel");
    if (ncol > nfac)
      apply_q_dispatch(st, true, m, std::min(nfac, m), W, ldw, sW, tau, sTau,
                       W + (long long)nfac * ldw, ldw, sW, ncol - nfac, W2, tau2,
                       W2 + (long long)nfac * ldw, batch, total);
    return;
  }
  panel_qr_kernel<<<total, 512, 0, st>>>(m, nfac, ncol, W, ldw, sW, tau, sTau, W2, tau2, batch);
  check_launch("panel_qr_kernel");
}

}  // namespace

void panel_qr(cudaStream_t st, int m, int nfac, int ncol, double* W, int ldw, long long sW,
              double* tau, long long sTau, int batch, int* info) {
  if (batch <= 0 || m <= 0 || nfac <= 0) return;
  panel_qr_any(st, m, nfac, ncol, W, W, ldw, sW, tau, tau, sTau, batch, batch, info);
}

void panel_qr2(cudaStream_t st, int m, int nfac, int ncol, double* W, double* W2, int ldw,
               long long sW, double* tau, double* tau2, long long sTau, int batch, int* info) {
  if (batch <= 0 || m <= 0 || nfac <= 0) return;
  panel_qr_any(st, m, nfac, ncol, W, W2, ldw, sW, tau, tau2, sTau, batch, 2 * batch, info);
}

void apply_q(cudaStream_t st, bool transpose, int m, int k, const double* V, int ldv,
             long long sV, const double* tau, long long sTau, double* C, int ldc, long long sC,
             int nc, int batch) {
  if (batch <= 0 || nc <= 0 || m <= 0) return;
  if (m <= kApplyRows) {
    apply_q_dispatch(st, transpose, m, k, V, ldv, sV, tau, sTau, C, ldc, sC, nc, V, tau, C, batch,
                     batch);
    return;
  }
  dim3 grid((nc + 7) / 8, batch);
  apply_q_kernel<<<grid, 256, 0, st>>>(transpose, m, k, V, ldv, sV, tau, sTau, C, ldc, sC, nc);
  check_launch("apply_q_kernel");
}

namespace {
template <int LANES, int RPL, int C>
void launch_jacobi(cudaStream_t st, int grid, int threads, size_t sm, int m, int n,
                   const double* A, int lda, long long sA, int r, double* U, int ldu,
                   long long sU, double* sv, long long sS, int* info, bool lower,
                   const double* A2, double* U2, int nsplit, int ld, int cols, int pre) {
  auto kern = jacobi_kernel<LANES, RPL, C>;
  ensure_smem(reinterpret_cast<const void*>(kern), sm);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(grid * C));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  SLU_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, m, n, A, lda, sA, r, U, ldu, sU, sv, sS, info,
                                    lower ? 1 : 0, A2, U2, nsplit, ld, cols, pre));
  check_launch("jacobi_kernel");
}

// Lanes per pair and rows per lane: the float64 instructions of the busiest
// SM sub-partition, (warps on it) x (4 per row + ~19), are least.  Four lanes
// put the 32 pairs of 64 columns on exactly one warp per sub-partition; other
// column counts fill it more evenly with eight.
void jacobi_dispatch(cudaStream_t st, int grid, int m, int n, const double* A, int lda,
                     long long sA, int r, double* U, int ldu, long long sU, double* sv,
                     long long sS, int* info, bool lower, const double* A2, double* U2,
                     int nsplit) {
  SLU_REQUIRE(r <= m, "jacobi: rank larger than rows");
  // shared memory: the columns, their norms, ranks and the row order.  The QR
  // needs A^T (m columns of n) in the same array: left out where that does not
  // fit, or where there is nothing to gain (one or two columns)
  auto bytes = [&](int ld, int cols, int pre) {
    return ((size_t)ld + 1) * cols * sizeof(double) +
           ((size_t)cols + (pre ? m : 0)) * sizeof(int);
  };
  const int k = std::min(m, n);
  int ld = std::max(m, n) | 1, cols = std::max(m, k + (k & 1)), pre = 1;
  if (n < 3 || m < 3 || bytes(ld, cols, 1) > 220 * 1024) {
    pre = 0;
    ld = m | 1;
    cols = n + (n & 1);
  }
  size_t sm = bytes(ld, cols, pre);
  SLU_REQUIRE(sm <= 220 * 1024, "jacobi: block too large for shared memory");
  const int swept = pre ? k : n, pairs = (swept + (swept & 1)) / 2;
  auto rows = [&](int lanes) { return (m + lanes - 1) / lanes; };
  auto cost = [&](int lanes) {
    const int warps = (pairs * lanes + 31) / 32;
    return (warps + 3) / 4 * (4 * rows(lanes) + 19);
  };
  int lanes = 4;
  if (rows(4) > 16 || cost(8) < cost(4)) lanes = 8;
  const int threads = std::min(JAC_THREADS, std::max(64, (pairs * lanes + 31) / 32 * 32));
#define SLU_JACOBI_C(L, R, C)                                                                  \
  return launch_jacobi<L, R, C>(st, grid, threads, sm, m, n, A, lda, sA, r, U, ldu, sU, sv, sS, \
                                info, lower, A2, U2, nsplit, ld, cols, pre)
#define SLU_JACOBI(L, R) SLU_JACOBI_C(L, R, 1)
  // few problems: four or two CTAs each, while every CTA gets an SM
  if (pre && k >= 32 && pairs * 4 <= JAC_CLUSTER_THREADS && 2LL * grid <= num_sms()) {
    const int C = 4LL * grid <= num_sms() ? 4 : 2, np = k + (k & 1);
    const int rc = ((m + C - 1) / C + 3) / 4;   // rows per lane, four lanes per pair
    const size_t more = 2 * sizeof(double) * C * np + 16;
    if (rc <= 10 && sm + more <= 220 * 1024) {
      sm += more;
      const int threads = std::max(64, (pairs * 4 + 31) / 32 * 32);
      if (C == 4) {
        if (rc <= 4) SLU_JACOBI_C(4, 4, 4);
        if (rc <= 6) SLU_JACOBI_C(4, 6, 4);
        SLU_JACOBI_C(4, 10, 4);
      }
      if (rc <= 8) SLU_JACOBI_C(4, 8, 2);
      SLU_JACOBI_C(4, 10, 2);
    }
  }
  const int rp = rows(lanes);
  if (lanes == 4) {
    if (rp <= 4) SLU_JACOBI(4, 4);
    if (rp <= 8) SLU_JACOBI(4, 8);
    if (rp <= 10) SLU_JACOBI(4, 10);
    if (rp <= 12) SLU_JACOBI(4, 12);
    if (rp <= 14) SLU_JACOBI(4, 14);
    SLU_JACOBI(4, 16);
  }
  if (rp <= 4) SLU_JACOBI(8, 4);
  if (rp <= 8) SLU_JACOBI(8, 8);
  if (rp <= 10) SLU_JACOBI(8, 10);
  if (rp <= 12) SLU_JACOBI(8, 12);
  if (rp <= 16) SLU_JACOBI(8, 16);
  SLU_JACOBI(8, 0);
#undef SLU_JACOBI
#undef SLU_JACOBI_C
}
}  // namespace

void jacobi_left_sv(cudaStream_t st, int m, int n, const double* A, int lda, long long sA, int r,
                    double* U, int ldu, long long sU, double* sv, long long sS, int batch,
                    int* info, bool lower) {
  if (batch <= 0 || r <= 0) return;
  jacobi_dispatch(st, batch, m, n, A, lda, sA, r, U, ldu, sU, sv, sS, info, lower, A, U, batch);
}

void jacobi_left_sv2(cudaStream_t st, int m, int n, const double* A, const double* A2, int lda,
                     long long sA, int r, double* U, double* U2, int ldu, long long sU, int batch,
                     int* info, bool lower) {
  if (batch <= 0 || r <= 0) return;
  jacobi_dispatch(st, 2 * batch, m, n, A, lda, sA, r, U, ldu, sU, nullptr, 0, info, lower, A2, U2,
                  batch);
}

}  // namespace slu
