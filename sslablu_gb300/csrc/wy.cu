// Columns carried along a QR of sketch blocks (matAssembly/HBS/HBSnew.py:20-28:
// Y_blk times the complete Q of Om_blk^T) in the compact WY form: with the
// reflectors' vectors as the rows of V (k x m), Q = H_0 H_1 .. = I - V^T T V and
//   C^T <- C^T - ((C^T V^T) T) V
// (C^T row-major: the columns carried, one per row).  T is the inverse of the
// upper triangle of V V^T with 1 / tau on the diagonal (C. Puglisi, SIAM J. Sci.
// Stat. Comput. 13, 1992).  One reflector after the other is twice m per column
// and reflector on the float64 pipe, whatever the number of columns; here all
// but T are products, exact residue products where they are large enough.  64
// reflectors of 261 rows on 64 columns: 128 panels 640 -> 280 us, 16 of them
// 298 -> 110.
#include <algorithm>

#include "hbs.cuh"

namespace slu {
namespace {

// V (k x m row-major) of a factored panel with unit diagonal and zeros in
// front of it; a reflector with tau = 0 (H = I) has a row of zeros.
__global__ void __launch_bounds__(256)
wy_vectors_kernel(int m, int k, const double* __restrict__ P, const double* __restrict__ P2,
                  int ldw, long long sW, const double* __restrict__ tau,
                  const double* __restrict__ tau2, long long sTau, double* __restrict__ V,
                  int nsplit) {
  const int a = blockIdx.x, i = blockIdx.y;
  const bool second = i >= nsplit;
  const int b = second ? i - nsplit : i;
  const double* p = (second ? P2 : P) + b * sW + (long long)a * ldw;
  const bool on = (second ? tau2 : tau)[b * sTau + a] != 0.0;
  double* v = V + ((long long)i * k + a) * m;
  for (int r = threadIdx.x; r < m; r += 256)
    v[r] = !on || r < a ? 0.0 : (r == a ? 1.0 : p[r]);
}

// T (k x k, upper) from G = V V^T and tau, by one CTA in shared memory: blocks
// of 16 by back substitution (a lane per column; the diagonal's reciprocals are
// the taus), then T12 = -T11 G12 T22 for pairs of neighbours, doubling.
__global__ void __launch_bounds__(256)
wy_tri_kernel(int k, const double* __restrict__ G, const double* __restrict__ tau,
              const double* __restrict__ tau2, long long sTau, double* __restrict__ T,
              int nsplit) {
  extern __shared__ double sm[];
  const int ld = k + 1, tid = threadIdx.x, i = blockIdx.x;
  double* S = sm;             // k x ld
  double* W = S + k * ld;     // the products of one level
  const bool second = i >= nsplit;
  const double* t = (second ? tau2 + (long long)(i - nsplit) * sTau : tau + (long long)i * sTau);
  G += (long long)i * k * k;
  T += (long long)i * k * k;
  for (int e = tid; e < k * k; e += 256) {
    const int r = e / k, c = e - r * k;
    S[r * ld + c] = c > r ? G[e] : 0.0;
  }
  __syncthreads();
  {
    const int c = tid, b0 = c & ~15;   // k <= 256 columns
    double x[16];
#pragma unroll
    for (int r = 15; r >= 0; --r) {
      x[r] = 0.0;
      if (b0 + r < k && b0 + r <= c && c < k) {
        double acc = b0 + r == c ? 1.0 : 0.0;
#pragma unroll
        for (int j = r + 1; j < 16; ++j)
          if (b0 + j < k) acc = fma(-S[(b0 + r) * ld + b0 + j], x[j], acc);
        x[r] = t[b0 + r] * acc;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (b0 + r < k && b0 + r <= c && c < k) S[(b0 + r) * ld + c] = x[r];
  }
  __syncthreads();
  for (int h = 16; h < k; h *= 2) {
    // pairs at b0: rows b0 .. b0 + h - 1, columns b0 + h .. min(b0 + 2 h, k) - 1
    const int pairs = (k + 2 * h - 1) / (2 * h), tot = pairs * h * h;
    for (int pass = 0; pass < 2; ++pass) {
      for (int e = tid; e < tot; e += 256) {
        const int q = e / (h * h), f = e - q * h * h, r = f / h, c = f - r * h, b0 = 2 * h * q;
        const int col = b0 + h + c;
        if (col >= k) continue;
        double a0 = 0.0, a1 = 0.0;
        if (pass == 0) {   // G12 T22
          const double* g = S + (b0 + r) * ld + b0 + h;
          const double* u = S + (b0 + h) * ld + col;
          int j = 0;
          for (; j < c; j += 2) {
            a0 = fma(g[j], u[j * ld], a0);
            a1 = fma(g[j + 1], u[(j + 1) * ld], a1);
          }
          if (j == c) a0 = fma(g[j], u[j * ld], a0);
          W[e] = a0 + a1;
        } else {           // -T11 (G12 T22)
          const double* u = S + (b0 + r) * ld + b0;
          const double* w = W + q * h * h + c;
          int j = r;
          for (; j + 1 < h; j += 2) {
            a0 = fma(u[j], w[j * h], a0);
            a1 = fma(u[j + 1], w[(j + 1) * h], a1);
          }
          if (j < h) a0 = fma(u[j], w[j * h], a0);
          S[(b0 + r) * ld + col] = -(a0 + a1);
        }
      }
      __syncthreads();
    }
  }
  for (int e = tid; e < k * k; e += 256) T[e] = S[e / k * ld + e % k];
}

constexpr int kMaxK = 128;

}  // namespace

// The reflectors one by one hold a row per eight lanes in registers and are
// bound by the float64 pipe or, with few blocks, by a chain of k steps: below
// 96 rows they are the faster way.
bool wy_pays(int m, int k, int nc) { return m >= 96 && m >= k && k >= 16 && k <= kMaxK && nc >= 16; }

// C <- Q^T C for the nc columns behind the k factored ones of two batches of
// panels (W2 == nullptr: one).
void apply_wy(Handle& h, int m, int k, double* W, double* W2, int ldw, long long sW, double* tau,
              double* tau2, long long sTau, int nc, int batch) {
  cudaStream_t st = h.stream;
  const int sets = W2 ? 2 : 1;
  const long long sV = (long long)k * m, sT = (long long)k * k, sX = (long long)nc * k;
  const size_t per = 8 * (size_t)sets * (sV + 2 * sT + 2 * sX) + 5 * 256;
  const int fit = (int)std::max<size_t>(
      1, std::min<size_t>(Handle::kScratchMax / per, (size_t)65535 / sets));
  const int sm = 8 * (k * (k + 1) + k * k / 2 + 2 * k * 16);
  ensure_smem(reinterpret_cast<const void*>(wy_tri_kernel), sm);
  for (int b0 = 0; b0 < batch; b0 += fit) {
    const int nb = std::min(fit, batch - b0), total = sets * nb;
    Scratch scratch(h.lu_ws, st);
    Workspace& ws = scratch.w;
    ws.reserve(per * nb + 4096, st);
    double* V = ws.take<double>(sV * total);
    double* G = ws.take<double>(sT * total);
    double* T = ws.take<double>(sT * total);
    double* X1 = ws.take<double>(sX * total);
    double* X2 = ws.take<double>(sX * total);
    double* Wa = W + b0 * sW;
    double* Wb = W2 ? W2 + b0 * sW : Wa;
    const double* ta = tau + b0 * sTau;
    const double* tb = W2 ? tau2 + b0 * sTau : ta;
    wy_vectors_kernel<<<dim3(k, total), 256, 0, st>>>(m, k, Wa, Wb, ldw, sW, ta, tb, sTau, V, nb);
    check_launch("wy_vectors_kernel");
    gemm_f64(h, false, true, k, k, m, 1.0, V, m, sV, 0, V, m, sV, 0, 0.0, G, k, sT, 0, total, 1);
    wy_tri_kernel<<<total, 256, sm, st>>>(k, G, ta, tb, sTau, T, nb);
    check_launch("wy_tri_kernel");
    double* Ct = Wa + (long long)k * ldw;
    const long long s2 = Wb - Wa;   // from one set to the other
    gemm_f64(h, false, true, nc, k, m, 1.0, Ct, ldw, sW, s2, V, m, sV, sV * nb, 0.0, X1, k, sX,
             sX * nb, nb, sets);
    gemm_f64(h, false, false, nc, k, k, 1.0, X1, k, sX, 0, T, k, sT, 0, 0.0, X2, k, sX, 0, total, 1);
    gemm_f64(h, false, false, nc, m, k, -1.0, X2, k, sX, sX * nb, V, m, sV, sV * nb, 1.0, Ct, ldw,
             sW, s2, nb, sets);
  }
}

}  // namespace slu
