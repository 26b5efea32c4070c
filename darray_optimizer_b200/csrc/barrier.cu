// FP64 device kernels of the log-barrier SVM dual solver (Newton step by Sherman-Morrison-Woodbury).
//
// Restates include/dbarrier.h:14-81 (f, gg, Grad_f, Grad_Phi, Grad, Hess_Phi) and the Newton / line-search
// arithmetic of tests/testsvm.cpp:243-321, with the Newton system solved as
//   (Z Z^T + diag(D)) s = -g   ->   (I + Z^T D^-1 Z) u = -Z^T D^-1 g,   s = -D^-1 (g + Z u)
// instead of the reference's PCG on (Z Z^T + D + n I) x = e_1 (include/dbarrier.h:84-139).
// Every pass over Z (n x r, column major, FP64) is HBM-bound.  Row passes (Z times an r-vector) give a CTA 64 rows and
// each of its 8 warps every eighth column of them (16-byte loads, a warp reads 512 contiguous bytes), the r-vector in
// shared memory; column passes (Z^T times an n-vector) give a warp four columns of a row range, so that the n-vector
// is read once for four of them.
#include <algorithm>
#include <cfloat>

#include "barrier.h"
#include "internal.h"

namespace db200 {
namespace {

constexpr int THREADS = 256;
constexpr int MAX_R_SMEM = 4096;  // r-vector staged in shared memory (32 KB)

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-reduce NV sums and atomically add them to out[0..NV).
template <int NV>
__device__ __forceinline__ void block_sum_add(double (&v)[NV], double* out) {
  __shared__ double red[NV][THREADS / 32];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const double s = warp_sum(v[k]);
    if (lane == 0) red[k][warp] = s;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
    for (int w = 0; w < THREADS / 32; ++w) s += red[threadIdx.x][w];
    atomicAdd(out + threadIdx.x, s);
  }
  __syncthreads();
}

// atomic max / min on non-negative doubles through their (monotone) bit patterns
__device__ __forceinline__ void atomic_max_pos(double* p, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void atomic_min_pos(double* p, double v) {
  atomicMin(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}

// part[w][i] = sum over the columns k = w (mod 8) of Z(i0 + i, k) s_k for the CTA's 64 rows, then their sum over w in
// the threads i < 64 (0 past n).  VEC: 16-byte loads.  Thread-per-row passes with 8-byte loads ran at 0.6 to 0.8 of the
// copy rate (131072 x 528: 106 - 140 us), 3.5 CTAs per SM of one wave.
constexpr int ROWS = 64;
template <bool VEC>
__device__ __forceinline__ double row_dots(const double* __restrict__ Z, long long ld, int i0, int n, int r,
                                           const double* s, double (*part)[ROWS]) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int i = i0 + (VEC ? 2 * lane : lane);
  const double* z = Z + i;
  double a0 = 0.0, a1 = 0.0;
  if (VEC && i + 1 < n) {
#pragma unroll 8
    for (int k = warp; k < r; k += 8) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(z + (long long)k * ld));
      a0 = fma(v.x, s[k], a0);
      a1 = fma(v.y, s[k], a1);
    }
  } else {
    const int step = VEC ? 1 : 32;  // the second row of this lane
    const bool p0 = i < n, p1 = i + step < n;
#pragma unroll 4
    for (int k = warp; k < r; k += 8) {
      if (p0) a0 = fma(__ldg(z + (long long)k * ld), s[k], a0);
      if (p1) a1 = fma(__ldg(z + (long long)k * ld + step), s[k], a1);
    }
  }
  __syncthreads();  // the sums of the row block before have been read
  part[warp][VEC ? 2 * lane : lane] = a0;
  part[warp][VEC ? 2 * lane + 1 : lane + 32] = a1;
  __syncthreads();
  double sum = 0.0;
  if (threadIdx.x < ROWS) {
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) sum += part[w][threadIdx.x];
  }
  return sum;
}

// Gradient and Hessian diagonal at a (Grad_f + Grad_Phi = Grad, Hess_Phi):
//   zw = Z (Z^T a),  g = zw - 1 + (-1/a + 1/(C - a))/t,  D = (1/a^2 + 1/(C - a)^2)/t,  dinv = 1/D
// Reductions into red[]: [0] sum(a), [1] sum(log a + log(C - a)), [2] max D, [3] min D.
template <bool VEC>
__global__ void __launch_bounds__(THREADS) grad_hess_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                            const double* __restrict__ w, const double* __restrict__ a,
                                                            double C, double t, double* __restrict__ g,
                                                            double* __restrict__ dinv, double* red,
                                                            const double* __restrict__ zw_in,
                                                            double* __restrict__ zw_out) {
  __shared__ double sw[MAX_R_SMEM];
  if (!zw_in)
    for (int k = threadIdx.x; k < r; k += blockDim.x) sw[k] = w[k];
  __syncthreads();
  double sums[2] = {0.0, 0.0};
  double dmax = 0.0, dmin = DBL_MAX;
  __shared__ double part[THREADS / 32][ROWS];
  for (int i0 = blockIdx.x * ROWS; i0 < n; i0 += gridDim.x * ROWS) {
    const double dot = zw_in ? 0.0 : row_dots<VEC>(Z, ld, i0, n, r, sw, part);
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= ROWS || i >= n) continue;
    const double ai = a[i], ci = C - ai;
    const double zw = zw_in ? zw_in[i] : dot;
    if (zw_out) zw_out[i] = zw;
    g[i] = (zw - 1.0) + ((-1.0 / ai) + (1.0 / ci)) / t;
    const double D = ((1.0 / (ai * ai)) + (1.0 / (ci * ci))) / t;
    dinv[i] = 1.0 / D;
    sums[0] += ai;
    sums[1] += log(ai) + log(ci);
    dmax = fmax(dmax, D);
    dmin = fmin(dmin, D);
  }
  block_sum_add<2>(sums, red);
  // max / min through warp shuffles then one atomic per warp
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
  }
  if (threadIdx.x % 32 == 0) {
    atomic_max_pos(red + 2, dmax);
    atomic_min_pos(red + 3, dmin);
  }
}

// Newton direction from u:  s = -dinv * (g + Z u).  Reductions: [0] g.s, [1] sum(s), [2] max feasible step
// (min over i of -a/s for s < 0 and (C - a)/s for s > 0).
template <bool VEC>
__global__ void __launch_bounds__(THREADS) direction_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                            const double* __restrict__ u, const double* __restrict__ g,
                                                            const double* __restrict__ dinv,
                                                            const double* __restrict__ a, double C,
                                                            double* __restrict__ s, double* red) {
  __shared__ double su[MAX_R_SMEM];
  for (int k = threadIdx.x; k < r; k += blockDim.x) su[k] = u[k];
  __syncthreads();
  double sums[2] = {0.0, 0.0};
  double tmax = DBL_MAX;
  __shared__ double part[THREADS / 32][ROWS];
  for (int i0 = blockIdx.x * ROWS; i0 < n; i0 += gridDim.x * ROWS) {
    const double zu = row_dots<VEC>(Z, ld, i0, n, r, su, part);
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= ROWS || i >= n) continue;
    const double gi = g[i];
    const double si = -dinv[i] * (gi + zu);
    s[i] = si;
    sums[0] += gi * si;
    sums[1] += si;
    const double ai = a[i];
    if (si < 0.0) tmax = fmin(tmax, -ai / si);
    else if (si > 0.0) tmax = fmin(tmax, (C - ai) / si);
  }
  block_sum_add<2>(sums, red);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tmax = fmin(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
  if (threadIdx.x % 32 == 0) atomic_min_pos(red + 2, tmax);
}

// out[k] += sign sum_i Z[i, k] * (scale_i * v_i)  (scale may be null): Z^T v.  A warp owns GT_COLS neighbouring columns and
// the rows of blockIdx.y, whose products scale_i v_i it forms once for all of them; FP64 atomics combine the row
// splits.  131072 x 528: 86 us (a column per warp, 8-byte loads, the vectors read per column: 106 - 117).
constexpr int GT_COLS = 4;
template <bool VEC>
__global__ void __launch_bounds__(THREADS) gemv_t_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                         const double* __restrict__ v, const double* __restrict__ scale,
                                                         double sign, double* out, int rows_per_split) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int k0 = (blockIdx.x * (THREADS / 32) + warp) * GT_COLS;
  if (k0 >= r) return;
  const int r0 = blockIdx.y * rows_per_split, r1 = min(n, r0 + rows_per_split);
  const double* z[GT_COLS];
  double acc[GT_COLS];
#pragma unroll
  for (int c = 0; c < GT_COLS; ++c) {
    z[c] = Z + (long long)min(k0 + c, r - 1) * ld;  // columns past r repeat the last and are not stored
    acc[c] = 0.0;
  }
  int i = r0 + (VEC ? 2 : 1) * lane;
  if (VEC) {
#pragma unroll 2
    for (; i + 1 < r1; i += 64) {
      double2 x = __ldg(reinterpret_cast<const double2*>(v + i));
      if (scale) {
        const double2 w = __ldg(reinterpret_cast<const double2*>(scale + i));
        x.x *= w.x;
        x.y *= w.y;
      }
#pragma unroll
      for (int c = 0; c < GT_COLS; ++c) {
        const double2 q = __ldg(reinterpret_cast<const double2*>(z[c] + i));
        acc[c] = fma(q.x, x.x, acc[c]);
        acc[c] = fma(q.y, x.y, acc[c]);
      }
    }
  }
  for (; i < r1; i += VEC ? 64 : 32) {  // VEC: an odd last row
    const double x = scale ? scale[i] * v[i] : v[i];
#pragma unroll
    for (int c = 0; c < GT_COLS; ++c) acc[c] = fma(__ldg(z[c] + i), x, acc[c]);
  }
#pragma unroll
  for (int c = 0; c < GT_COLS; ++c) {
    const double sum = warp_sum(acc[c]);
    if (lane == 0 && k0 + c < r) atomicAdd(out + k0 + c, sign * sum);
  }
}

// Log-barrier sums at the 16 candidate steps: out[k] += sum_i log(a_i + tau_k s_i) + log(C - a_i - tau_k s_i); a candidate
// that leaves the open box anywhere counts its infeasible rows in out[16 + k].  A thread per row and candidate (lane %
// 16): bound by the logarithms' issue, which needs the warps.  n = 4096: 2.7 us (a thread per row with all 16
// candidates, 16 CTAs and 32 block sums: 8.9); 131072: 16 us (22).
__global__ void __launch_bounds__(THREADS) linesearch16_kernel(int n, const double* __restrict__ a,
                                                               const double* __restrict__ s, double C,
                                                               const double* __restrict__ taus, double* out) {
  __shared__ double part[2][THREADS / 32][16];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, k = lane % 16;
  const double tau = taus[k];
  double sum = 0.0, bad = 0.0;
  for (int i = (blockIdx.x * THREADS + threadIdx.x) / 16; i < n; i += gridDim.x * (THREADS / 16)) {
    const double ai = a[i], si = s[i];
    const double x = fma(tau, si, ai), y = C - x;
    if (x > 0.0 && y > 0.0)
      sum += log(x) + log(y);
    else
      bad += 1.0;
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  bad += __shfl_xor_sync(0xffffffffu, bad, 16);
  if (lane < 16) {
    part[0][warp][k] = sum;
    part[1][warp][k] = bad;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) v += part[threadIdx.x / 16][w][k];
    if (threadIdx.x < 16 || v != 0.0) atomicAdd(out + threadIdx.x, v);
  }
}

// gradf = Z w - 1, gradphi = (-1/a + 1/(C-a))/t, grad = gradf + gradphi, D = (1/a^2 + 1/(C-a)^2)/t
// (include/dbarrier.h:48-81 one by one); red: [0] += sum a, [1] += sum(log a + log(C - a)).
template <bool VEC>
__global__ void __launch_bounds__(THREADS) terms_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                        const double* __restrict__ w, const double* __restrict__ a,
                                                        double C, double t, double* gf, double* gp, double* g,
                                                        double* D, double* red) {
  __shared__ double sw[MAX_R_SMEM];
  for (int k = threadIdx.x; k < r; k += blockDim.x) sw[k] = w[k];
  __syncthreads();
  double sums[2] = {0.0, 0.0};
  __shared__ double part[THREADS / 32][ROWS];
  for (int i0 = blockIdx.x * ROWS; i0 < n; i0 += gridDim.x * ROWS) {
    const double f1 = row_dots<VEC>(Z, ld, i0, n, r, sw, part) - 1.0;
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= ROWS || i >= n) continue;
    const double ai = a[i], ci = C - ai;
    const double p1 = ((-1.0 / ai) + (1.0 / ci)) / t;
    gf[i] = f1;
    gp[i] = p1;
    g[i] = f1 + p1;
    D[i] = ((1.0 / (ai * ai)) + (1.0 / (ci * ci))) / t;
    sums[0] += ai;
    sums[1] += log(ai) + log(ci);
  }
  block_sum_add<2>(sums, red);
}

// Negated residual of the Newton system (Z Z^T + D) s = -g:  res = g + Z v + s / dinv  with v = Z^T s.
// red: [0] += |res|^2, [1] += |g|^2.
template <bool VEC>
__global__ void __launch_bounds__(THREADS) residual_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                           const double* __restrict__ v, const double* __restrict__ g,
                                                           const double* __restrict__ dinv,
                                                           const double* __restrict__ s, double* __restrict__ res,
                                                           double* red, double* __restrict__ zv_out) {
  __shared__ double sv[MAX_R_SMEM];
  for (int k = threadIdx.x; k < r; k += blockDim.x) sv[k] = v[k];
  __syncthreads();
  double sums[2] = {0.0, 0.0};
  __shared__ double part[THREADS / 32][ROWS];
  for (int i0 = blockIdx.x * ROWS; i0 < n; i0 += gridDim.x * ROWS) {
    const double zv = row_dots<VEC>(Z, ld, i0, n, r, sv, part);
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= ROWS || i >= n) continue;
    const double gi = g[i];
    if (zv_out) zv_out[i] = zv;
    const double ri = gi + zv + s[i] / dinv[i];
    res[i] = ri;
    sums[0] += ri * ri;
    sums[1] += gi * gi;
  }
  block_sum_add<2>(sums, red);
}

// Line-search inputs for a direction s: red [0] += g.s, [1] += sum s, [2] min feasible step (init DBL_MAX).
__global__ void __launch_bounds__(THREADS) step_stats_kernel(int n, const double* __restrict__ g,
                                                             const double* __restrict__ s,
                                                             const double* __restrict__ a, double C, double* red) {
  double sums[2] = {0.0, 0.0};
  double tmax = DBL_MAX;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double si = s[i], ai = a[i];
    sums[0] += g[i] * si;
    sums[1] += si;
    if (si < 0.0) tmax = fmin(tmax, -ai / si);
    else if (si > 0.0) tmax = fmin(tmax, (C - ai) / si);
  }
  block_sum_add<2>(sums, red);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tmax = fmin(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
  if (threadIdx.x % 32 == 0) atomic_min_pos(red + 2, tmax);
}

__global__ void reciprocal_kernel(int n, const double* x, double* y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = 1.0 / x[i];
}

__global__ void vec_update_kernel(int n, double alpha, const double* x, double beta, double* y, double gamma) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = (x ? alpha * x[i] : 0.0) + (beta != 0.0 ? beta * y[i] : 0.0) + gamma;
}

__global__ void negate_kernel(int n, const double* x, double* y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = -x[i];
}

__global__ void axpy_kernel(int n, double alpha, const double* __restrict__ x, double* __restrict__ y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = fma(alpha, x[i], y[i]);
}

// Primal value pieces at w = Z^T a:  sum_i max(0, 1 - (Z w)_i)
template <bool VEC>
__global__ void __launch_bounds__(THREADS) hinge_kernel(int n, int r, const double* __restrict__ Z, long long ld,
                                                        const double* __restrict__ w, double* red,
                                                        const double* __restrict__ y, double b) {
  __shared__ double sw[MAX_R_SMEM];
  for (int k = threadIdx.x; k < r; k += blockDim.x) sw[k] = w[k];
  __syncthreads();
  double sums[1] = {0.0};
  __shared__ double part[THREADS / 32][ROWS];
  for (int i0 = blockIdx.x * ROWS; i0 < n; i0 += gridDim.x * ROWS) {
    const double zw = row_dots<VEC>(Z, ld, i0, n, r, sw, part);
    const int i = i0 + threadIdx.x;
    if (threadIdx.x < ROWS && i < n) sums[0] += fmax(0.0, 1.0 - zw - (y ? y[i] * b : 0.0));
  }
  block_sum_add<1>(sums, red);
}

__global__ void scale_diag_kernel(double* M, int ldm, int r, double factor) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r; i += gridDim.x * blockDim.x) M[(long long)i * ldm + i] *= factor;
}

__global__ void add_identity_kernel(double* M, int ldm, int r) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r; i += gridDim.x * blockDim.x) M[(long long)i * ldm + i] += 1.0;
}

__global__ void init_red_kernel(double* red, int nsum, int nmax, int nmin) {
  const int i = threadIdx.x;
  if (i < nsum) red[i] = 0.0;
  else if (i < nsum + nmax) red[i] = 0.0;
  else if (i < nsum + nmax + nmin) red[i] = DBL_MAX;
}

// One CTA's scalars of a Newton step in one launch (six nodes of a graph before): wv[0] = w.v, wv[1] = v.v, the line
// search's sums ls[0..32) cleared, and taus[k] = t0 beta^k (k < 16), t0 = min(1, 0.99 * *step_max), by repeated
// multiplication (the host forms the same values the same way).
__global__ void __launch_bounds__(THREADS) step_scalars_kernel(int r, const double* __restrict__ w,
                                                               const double* __restrict__ v, double* wv,
                                                               const double* step_max, double beta, double* taus,
                                                               double* ls) {
  double s[2] = {0.0, 0.0};
  for (int k = threadIdx.x; k < r; k += THREADS) {
    s[0] += w[k] * v[k];
    s[1] += v[k] * v[k];
  }
  if (threadIdx.x < 2) wv[threadIdx.x] = 0.0;  // before block_sum_add's barrier, added to after it by the same threads
  if (threadIdx.x >= 32 && threadIdx.x < 64) ls[threadIdx.x - 32] = 0.0;
  if (threadIdx.x == 64) {
    const double m = 0.99 * *step_max;
    double t = (m < 1.0) ? m : 1.0;  // as std::min(1.0, m): 1 when m is NaN
    for (int k = 0; k < 16; ++k) {
      taus[k] = t;
      t *= beta;
    }
  }
  block_sum_add<2>(s, wv);
}

__global__ void dot_kernel(int r, const double* x, const double* y, double* out) {
  double s = 0.0;
  for (int k = threadIdx.x; k < r; k += blockDim.x) s += x[k] * y[k];
  double v[1] = {s};
  if (threadIdx.x == 0) out[0] = 0.0;  // this thread adds the sum to it
  block_sum_add<1>(v, out);
}

// grid of the row passes: 64 rows per CTA, up to eight CTAs per SM
inline int blocks64(db200_context* ctx, int n) { return std::max(1, std::min((n + ROWS - 1) / ROWS, 8 * ctx->num_sms)); }
inline bool vec_ok(const double* Z, long long ld) { return reinterpret_cast<uintptr_t>(Z) % 16 == 0 && ld % 2 == 0; }

inline int rows_grid(db200_context* ctx, int n) {
  int b = (n + THREADS - 1) / THREADS;
  const int cap = 4 * ctx->num_sms;
  return b < 1 ? 1 : (b > cap ? cap : b);
}

}  // namespace

int bar_init_red(db200_context* ctx, double* red, int nsum, int nmax, int nmin) {
  init_red_kernel<<<1, 64, 0, ctx->stream>>>(red, nsum, nmax, nmin);
  count_launch(ctx);
  return cudaGetLastError() == cudaSuccess ? DB200_OK : cuda_fail(ctx, cudaGetLastError(), "init_red");
}

int bar_grad_hess(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* w, const double* a,
                  double C, double t, double* g, double* dinv, double* red, const double* zw_in, double* zw_out) {
  if (r > MAX_R_SMEM) return fail(ctx, DB200_ERR_UNSUPPORTED, "barrier: rank > 4096");
  auto k = vec_ok(Z, ld) ? grad_hess_kernel<true> : grad_hess_kernel<false>;
  k<<<blocks64(ctx, n), THREADS, 0, ctx->stream>>>(n, r, Z, ld, w, a, C, t, g, dinv, red, zw_in, zw_out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_direction(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* u, const double* g,
                  const double* dinv, const double* a, double C, double* s, double* red) {
  auto k = vec_ok(Z, ld) ? direction_kernel<true> : direction_kernel<false>;
  k<<<blocks64(ctx, n), THREADS, 0, ctx->stream>>>(n, r, Z, ld, u, g, dinv, a, C, s, red);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_gemv_t(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* v, const double* scale,
               double sign, double* out) {
  DB200_CUDA(ctx, cudaMemsetAsync(out, 0, sizeof(double) * r, ctx->stream));
  // about eight CTAs per SM, no split shorter than 128 rows
  const int per = GT_COLS * THREADS / 32, col_blocks = (r + per - 1) / per;
  int splits = std::max(1, std::min((n + 127) / 128, 8 * ctx->num_sms / col_blocks));
  const int rows = round_up((n + splits - 1) / splits, 64);
  splits = (n + rows - 1) / rows;
  const bool vec = vec_ok(Z, ld) && vec_ok(v, 2) && (!scale || vec_ok(scale, 2));
  auto k = vec ? gemv_t_kernel<true> : gemv_t_kernel<false>;
  k<<<dim3(col_blocks, splits), THREADS, 0, ctx->stream>>>(n, r, Z, ld, v, scale, sign, out, rows);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_linesearch16(db200_context* ctx, int n, const double* a, const double* s, double C, const double* taus,
                     double* out) {
  const int blocks = std::max(1, std::min((n + THREADS / 16 - 1) / (THREADS / 16), 8 * ctx->num_sms));
  linesearch16_kernel<<<blocks, THREADS, 0, ctx->stream>>>(n, a, s, C, taus, out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_terms(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* w, const double* a,
              double C, double t, double* gf, double* gp, double* g, double* D, double* red) {
  if (r > MAX_R_SMEM) return fail(ctx, DB200_ERR_UNSUPPORTED, "barrier: rank > 4096");
  auto k = vec_ok(Z, ld) ? terms_kernel<true> : terms_kernel<false>;
  k<<<blocks64(ctx, n), THREADS, 0, ctx->stream>>>(n, r, Z, ld, w, a, C, t, gf, gp, g, D, red);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_residual(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* v, const double* g,
                 const double* dinv, const double* s, double* res, double* red, double* zv_out) {
  auto k = vec_ok(Z, ld) ? residual_kernel<true> : residual_kernel<false>;
  k<<<blocks64(ctx, n), THREADS, 0, ctx->stream>>>(n, r, Z, ld, v, g, dinv, s, res, red, zv_out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_step_stats(db200_context* ctx, int n, const double* g, const double* s, const double* a, double C,
                   double* red) {
  step_stats_kernel<<<rows_grid(ctx, n), THREADS, 0, ctx->stream>>>(n, g, s, a, C, red);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_reciprocal(db200_context* ctx, int n, const double* x, double* y) {
  reciprocal_kernel<<<rows_grid(ctx, n), THREADS, 0, ctx->stream>>>(n, x, y);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_vec_update(db200_context* ctx, int n, double alpha, const double* x, double beta, double* y, double gamma) {
  vec_update_kernel<<<rows_grid(ctx, n), THREADS, 0, ctx->stream>>>(n, alpha, x, beta, y, gamma);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_negate(db200_context* ctx, int n, const double* x, double* y) {
  negate_kernel<<<rows_grid(ctx, n), THREADS, 0, ctx->stream>>>(n, x, y);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_axpy(db200_context* ctx, int n, double alpha, const double* x, double* y) {
  axpy_kernel<<<rows_grid(ctx, n), THREADS, 0, ctx->stream>>>(n, alpha, x, y);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_hinge(db200_context* ctx, int n, int r, const double* Z, long long ld, const double* w, double* red,
              const double* y, double b) {
  DB200_CUDA(ctx, cudaMemsetAsync(red, 0, sizeof(double), ctx->stream));
  auto k = vec_ok(Z, ld) ? hinge_kernel<true> : hinge_kernel<false>;
  k<<<blocks64(ctx, n), THREADS, 0, ctx->stream>>>(n, r, Z, ld, w, red, y, b);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_add_identity(db200_context* ctx, double* M, int ldm, int r) {
  add_identity_kernel<<<(r + 255) / 256, 256, 0, ctx->stream>>>(M, ldm, r);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_scale_diag(db200_context* ctx, double* M, int ldm, int r, double factor) {
  scale_diag_kernel<<<(r + 255) / 256, 256, 0, ctx->stream>>>(M, ldm, r, factor);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_step_scalars(db200_context* ctx, int r, const double* w, const double* v, double* wv, const double* step_max,
                     double beta, double* taus, double* ls) {
  step_scalars_kernel<<<1, THREADS, 0, ctx->stream>>>(r, w, v, wv, step_max, beta, taus, ls);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int bar_dot(db200_context* ctx, int r, const double* x, const double* y, double* out) {
  dot_kernel<<<1, THREADS, 0, ctx->stream>>>(r, x, y, out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

}  // namespace db200
