// FP64 dense linear algebra for the 1 x 1 DMatrix path: tall-skinny Gram (matrix_multiply T,N), tall GEMM,
// blocked Cholesky (cholesky_factorize 'U'), triangular inverse / solves (triangular_solve), GEMV pairs.
//
// Restated from include/lapack_like.h:10-56 (blocked right-looking Cholesky: potrf on the diagonal block, trsm on
// the panel, syrk on the trailing matrix), include/blas_like.h:63-127 (matrix_multiply T,N; triangular_solve
// L,U,T,N) and include/cblas_like.h:40-69, in FP64 on the GPU.  All matrices are column major.
#include <cstdio>
#include <type_traits>

#include "dmm64.cuh"
#include "internal.h"
#include "la64.h"
#include "potrf64.cuh"

namespace db200 {

namespace {

// The Cholesky's trailing matrix takes whole DMM tiles once it holds a wave of them (128 x 128 upper tiles).
constexpr int GT = 128;

// One block column of the right-looking blocked upper Cholesky: the kb x kb diagonal block (kb <= 64) is factored
// in every CTA (redundantly), whose other four warps solve 64 columns of the block row, the columns
// [k0 + kb + 64 blockIdx.x, +64), at the same time (p64_run, potrf64.cuh).  The last CTA to have read the block writes
// R11 back (zeros below its diagonal), and that write waits for nothing: every CTA counts itself in `arrivals` after
// its reads of A11, and the CTA that arrives last, when every other one has read A11, is the one that overwrites
// it (and re-arms the counter for the next launch).  On a non-positive or NaN pivot nothing is written, status <-
// DB200_ERR_NOT_SPD and *bad <- k0 (first failing block).  A block column after a failed one writes nothing.  Follows
// cholesky_factorize (include/lapack_like.h:10-57): potrf of the diagonal block, trsm of the panel, syrk of the
// trailing matrix (launched after this one).
template <bool VEC>
__global__ void __launch_bounds__(P64_THREADS) potrf_block_kernel(double* A, int lda, int k0, int kb, int l,
                                                                  int* status, int* bad, int* arrivals, double* W) {
  extern __shared__ __align__(16) unsigned char raw[];
  P64Smem& S = *reinterpret_cast<P64Smem*>(raw);
  const int t = threadIdx.x, warp = t / 32;
  int group = warp, col = k0 + 16 * warp, cl = k0 + kb;
  if (warp >= 4) {
    col = k0 + kb + 64 * (int)blockIdx.x + 16 * (warp - 4);
    cl = l;
    group = col < l ? warp : -1;
  }
  double acc[8][4];
  if (group >= 0) p64_load<VEC>(acc, A, lda, k0, kb, col, cl, warp < 4 ? warp : -1);
  __syncthreads();  // this CTA's reads of A11 are done
  if (t == 0) {
    __threadfence();
    const int before = atomicAdd(arrivals, 1);
    S.flag = (before == (int)gridDim.x - 1);
    if (S.flag) *arrivals = 0;  // every CTA has arrived: re-armed for the next launch
    __threadfence();
  }
  if (*(volatile int*)status) return;  // an earlier block column failed (checked after counting in)
  const bool ok = p64_run(S, acc, group, P64_NB);  // (a constant: a bound here costs each of many full blocks 0.4 us)
  const bool writer = S.flag != 0;  // visible: p64_run passed a barrier
  if (!ok) {
    if (writer && t == 0 && atomicCAS(status, 0, DB200_ERR_NOT_SPD) == 0) *bad = k0;
    return;
  }
  if (writer) {
    for (int e = t; e < kb * P64_NB; e += P64_THREADS) {
      const int i = e % P64_NB, j = e / P64_NB;
      if (i < kb) A[(long long)(k0 + j) * lda + k0 + i] = (i <= j) ? S.R[j * P64_RLD + i] : 0.0;
    }
    if (W) p64_store_inverses(S, W + (long long)k0 * 16, kb);
  }
  if (group >= 4) p64_store<VEC>(acc, A, lda, k0, kb, col, cl);
}

// Trailing update of the blocked Cholesky: C[m x m] (upper triangle) -= P^T P for the kb x m panel P (kb <= 64, the
// rows of R12 just solved).  One 32 x 32 tile of C per CTA (upper tiles only) so that the few hundred tiles of an
// r ~ 500..4000 factor spread over the whole GPU; the two 64 x 32 panel slices sit in shared memory and each of the
// 256 threads forms 4 outputs with 64-long FP64 dot products.
__global__ void __launch_bounds__(256) syrk_update_kernel(const double* __restrict__ P, int ldp, int kb, int m,
                                                          double* C, int ldc, const int* status) {
  if (*(volatile const int*)status) return;
  int idx = blockIdx.x, bi = 0;
  const int nt = (m + 31) / 32;
  while (idx >= nt - bi) {  // upper tile pairs (bi <= bj), row by row
    idx -= nt - bi;
    ++bi;
  }
  const int bj = bi + idx;
  const int i0 = bi * 32, j0 = bj * 32;
  __shared__ double pi[64][33], pj[64][33];
  for (int e = threadIdx.x; e < 64 * 32; e += 256) {
    const int k = e & 63, c = e >> 6;  // consecutive threads walk k: one column of P is contiguous
    pi[k][c] = (k < kb && i0 + c < m) ? P[(long long)(i0 + c) * ldp + k] : 0.0;
    pj[k][c] = (k < kb && j0 + c < m) ? P[(long long)(j0 + c) * ldp + k] : 0.0;
  }
  __syncthreads();
  const int ti = threadIdx.x & 31, tj = threadIdx.x >> 5;  // rows ti; columns tj + 8 b
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int k = 0; k < 64; ++k) {
    const double a = pi[k][ti];
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[b] = fma(a, pj[k][tj + 8 * b], acc[b]);
  }
  const int i = i0 + ti;
  if (i >= m) return;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int j = j0 + tj + 8 * b;
    if (j < m && i <= j) C[(long long)j * ldc + i] -= acc[b];
  }
}

// Zero the strictly lower triangle of an l x l matrix.
__global__ void zero_lower_kernel(double* A, int lda, int l) {
  const long long total = (long long)l * l;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % l), j = (int)(e / l);
    if (i > j) A[(long long)j * lda + i] = 0.0;
  }
}

// U <- the upper triangle of R, zeros below.
__global__ void copy_upper_kernel(const double* R, int ldr, int l, double* U, int ldu) {
  const long long total = (long long)l * l;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % l), j = (int)(e / l);
    U[(long long)j * ldu + i] = i <= j ? R[(long long)j * ldr + i] : 0.0;
  }
}

// Diagonal blocks of X = R^-1 (upper triangular, l x l): one warp per 32 x 32 block, lane j holding column j of the
// block's inverse in registers (column-oriented back substitution; R's columns are read from shared memory as
// broadcasts).  Rows and columns past l behave as identity and are not stored.
constexpr int TI = 32;
constexpr int TI_WARPS = 4;
__global__ void __launch_bounds__(32 * TI_WARPS) trinv_diag_kernel(const double* R, int ldr, int l, double* X,
                                                                   int ldx) {
  __shared__ double sR[TI_WARPS][TI][TI + 1];  // column i of the block at sR[i]
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int r0 = (blockIdx.x * TI_WARPS + warp) * TI;
  if (r0 >= l) return;
  double(*S)[TI + 1] = sR[warp];
#pragma unroll 4
  for (int i = 0; i < TI; ++i) {
    const bool in = r0 + i < l && r0 + lane < l;
    S[i][lane] = in ? R[(long long)(r0 + i) * ldr + r0 + lane] : (i == lane ? 1.0 : 0.0);
  }
  __syncwarp();
  double x[TI];
#pragma unroll
  for (int i = 0; i < TI; ++i) x[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll
  for (int i = TI - 1; i >= 0; --i) {
    x[i] = x[i] / S[i][i];
#pragma unroll
    for (int k = 0; k < i; ++k) x[k] = fma(-S[i][k], x[i], x[k]);
  }
  if (r0 + lane < l) {
    double* col = X + (long long)(r0 + lane) * ldx + r0;
#pragma unroll
    for (int i = 0; i < TI; ++i)
      if (r0 + i < l) col[i] = x[i];
  }
}

// Clears the rows below the diagonal of every block pair (blockIdx.y) of trinv_doubling's level h.
__global__ void trinv_clear_kernel(double* X, int ldx, int l, int h) {
  const int r0 = 2 * h * (int)blockIdx.y, q = min(h, l - r0 - h);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < q * h; e += gridDim.x * blockDim.x)
    X[(long long)(r0 + e / q) * ldx + r0 + h + e % q] = 0.0;
}

// x <- R^-1 R^-T x for an upper factor R (l <= 4096) with the inverses W = R_bb^-T of its 16 x 16 diagonal blocks, in one
// CTA: the forward solve R^T z = x (block b needs its columns above the block, a warp per column), then R u = z (block b
// needs its 16 rows right of the block, 16 contiguous entries per column; no transposed copy).  Per block: the off-block
// products, their reduction, and y = W r, y += W (r - R_bb^T y), three 16 x 16 products of one warp, instead of 16 dependent
// substitution steps (the correction keeps the substitution's backward error).  What a block reads depends on nothing
// computed: every thread holds its part of the next panel (16 x 256) in registers, and warp 0 of the next W and R_bb, loaded
// one block ahead, so the chain holds no memory latency.  Bound by that chain of l / 16 blocks each way, about 1.5 us a
// block: l = 528 106 us, l = 138 23 us (shared-memory rings fed by cp.async or bulk copies 121 - 139 and 27, their issue in
// the chain's way; a global load, a 32-step shuffle chain and a transposed copy per block of 32: 2 x 82 and 2 x 16 us and
// the copy).
// Follows triangular_solve (include/blas_like.h:96-140) for one column.
constexpr int TV_THREADS = 512, TV_NB = 16, TV_LEN = 256, TV_MAX_L = 4096;
struct TrsvSmem {
  double x[TV_MAX_L + TV_LEN];
  double part[16][16];
  double r[16], e[16];
};

// One direction's blocks (a template: the addresses of the two differ by constants that the loop then carries as
// immediates; chosen at run time they made the loop's integer work its bound, 360 instructions per warp and block).
template <bool FWD>
__device__ __forceinline__ void trsv_sweep(TrsvSmem& S, const double* __restrict__ R, int ld, int l,
                                           const double* __restrict__ W, int nb) {
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int i = lane % 16, h = 8 * (lane / 16);  // warp 0's solve: row i, half h of its products
  const int first = FWD ? lane : tid / 16;       // this thread's first off-block index, then every 32nd
  const long long step = FWD ? 32 : 32LL * ld;
  // forward: rows 0 .. b0 - 1 of column b0 + warp; backward: row b0 + tid % 16 of the columns b0 + 16 .. l - 1
  auto base = [&](int b) -> const double* {
    const int b0 = b * TV_NB;
    return FWD ? R + (long long)min(b0 + warp, l - 1) * ld + first
               : R + (long long)(b0 + TV_NB + first) * ld + b0 + tid % 16;
  };
  auto off_len = [&](int b) -> int { return FWD ? b * TV_NB : l - (b + 1) * TV_NB; };
  auto load = [&](const double* p, int left, double (&v)[8]) {  // left: entries from `first` of this piece on
    if (left >= TV_LEN) {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(p + u * step);
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u] = 0.0;
        if (first + 32 * u < left) v[u] = __ldg(p + u * step);
      }
    }
  };
  // forward: W(i, h + k) and R_bb(h + k, i); backward: W(h + k, i) and R_bb(i, h + k)
  auto load_diag = [&](int b, double (&w)[8], double (&d)[8]) {
    const int b0 = b * TV_NB;
    const double* Wb = W + (long long)b * 256 + (FWD ? i * 16 + h : h * 16 + i);
    const double* Rb = FWD ? R + (long long)min(b0 + i, l - 1) * ld + b0 + h : R + (long long)(b0 + h) * ld + b0 + i;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      w[k] = __ldg(Wb + (FWD ? k : 16 * k));
      const bool in = FWD ? (h + k <= i && b0 + i < l) : (i <= h + k && b0 + h + k < l);
      d[k] = in ? __ldg(Rb + (FWD ? k : (long long)k * ld)) : 0.0;
    }
  };
  int b = FWD ? 0 : nb - 1;
  const double* p = base(b);
  double nxt[8], wn[8], dn[8];
  load(p, off_len(b), nxt);
  if (warp == 0) load_diag(b, wn, dn);
#pragma unroll 1
  for (int k = 0; k < nb; ++k) {
    const int b0 = b * TV_NB, len = off_len(b), bn = FWD ? b + 1 : b - 1;
    const bool more = k + 1 < nb;
    double w[8], d[8];
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        w[q] = wn[q];
        d[q] = dn[q];
      }
      if (more) load_diag(bn, wn, dn);
    }
    double acc0 = 0.0, acc1 = 0.0;
    const double* xp = S.x + first + (FWD ? 0 : b0 + TV_NB);
    int left = len;
#pragma unroll 1
    do {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = nxt[u];
      if (left > TV_LEN) {
        p += 8 * step;
        load(p, left - TV_LEN, nxt);
      } else if (more) {
        p = base(bn);
        load(p, off_len(bn), nxt);
      }
      if (left == len) __syncthreads();  // x of the block before is written
      // past the end v is zero and x (cleared beyond l) finite
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        acc0 = fma(v[u], xp[32 * u], acc0);
        acc1 = fma(v[u + 1], xp[32 * u + 32], acc1);
      }
      xp += TV_LEN;
      left -= TV_LEN;
    } while (left > 0);
    acc0 += acc1;
    acc0 += __shfl_xor_sync(0xffffffffu, acc0, 16);
    if (FWD) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) acc0 += __shfl_xor_sync(0xffffffffu, acc0, o);
      if (lane == 0) S.r[warp] = b0 + warp < l ? S.x[b0 + warp] - acc0 : 0.0;
    } else {
      if (lane < 16) S.part[warp][lane] = acc0;
    }
    __syncthreads();
    if (warp == 0) {
      if (!FWD) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += S.part[h + q][i];
        t += __shfl_xor_sync(0xffffffffu, t, 16);
        if (lane < 16) S.r[i] = b0 + i < l ? S.x[b0 + i] - t : 0.0;
        __syncwarp();
      }
      auto apply = [&](const double (&m)[8], const double* v) -> double {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
          const double2 z = *reinterpret_cast<const double2*>(v + h + q);
          s0 = fma(m[q], z.x, s0);
          s1 = fma(m[q + 1], z.y, s1);
        }
        s0 += s1;
        return s0 + __shfl_xor_sync(0xffffffffu, s0, 16);
      };
      double y = apply(w, S.r);
      if (lane < 16) S.x[b0 + i] = y;
      __syncwarp();
      const double ry = apply(d, S.x + b0);
      if (lane < 16) S.e[i] = S.r[i] - ry;
      __syncwarp();
      y += apply(w, S.e);
      if (lane < 16) S.x[b0 + i] = y;
    }
    b = bn;
  }
}

__global__ void __launch_bounds__(TV_THREADS, 1) trsv_pair_kernel(const double* __restrict__ R, int ld, int l,
                                                                  const double* __restrict__ W, double* x) {
  __shared__ __align__(16) TrsvSmem S;
  const int nb = (l + TV_NB - 1) / TV_NB;
  for (int k = threadIdx.x; k < nb * TV_NB + TV_LEN; k += TV_THREADS) S.x[k] = k < l ? x[k] : 0.0;
  trsv_sweep<true>(S, R, ld, l, W, nb);   // R^T z = x (its first barrier also ends the staging)
  trsv_sweep<false>(S, R, ld, l, W, nb);  // R u = z
  __syncthreads();
  for (int k = threadIdx.x; k < l; k += TV_THREADS) x[k] = S.x[k];
}

__global__ void scale_kernel(double* C, int ldc, int m, int n, double beta, int upper_only) {
  const long long total = (long long)m * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % m), j = (int)(e / m);
    if (upper_only && i > j) continue;
    double* p = C + (long long)j * ldc + i;
    *p = (beta == 0.0) ? 0.0 : beta * *p;
  }
}

__global__ void symmetrize_kernel(double* C, int ldc, int l, double shift) {
  // C <- (C + C^T)/2 + shift I, full matrix
  const long long total = (long long)l * l;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % l), j = (int)(e / l);
    if (i > j) continue;
    double* a = C + (long long)j * ldc + i;
    double* b = C + (long long)i * ldc + j;
    double v = 0.5 * (*a + *b);
    if (i == j) v += shift;
    *a = v;
    *b = v;
  }
}

__global__ void fill_upper_from_lower_kernel(double* C, int ldc, int l) {
  const long long total = (long long)l * l;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % l), j = (int)(e / l);
    if (i > j) C[(long long)j * ldc + i] = C[(long long)i * ldc + j];
  }
}

template <typename TS, typename TD>
__global__ void convert_kernel(const TS* src, long long lds, TD* dst, long long ldd, int m, int n) {
  const long long total = (long long)m * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % m), j = (int)(e / m);
    dst[j * ldd + i] = (TD)src[j * lds + i];
  }
}

// C (float) = alpha * T (double) + beta * C
__global__ void axpby_f32_kernel(float* C, long long ldc, const double* T, long long ldt, int m, int n, double alpha,
                                 double beta) {
  const long long total = (long long)m * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % m), j = (int)(e / m);
    float* c = C + j * ldc + i;
    double v = alpha * T[j * ldt + i];
    if (beta != 0.0) v += beta * (double)*c;
    *c = (float)v;
  }
}

// out[0] += sum of squares of the m x n float block
__global__ void sumsq_f32_kernel(const float* A, long long lda, int m, int n, double* out) {
  double s = 0.0;
  const long long total = (long long)m * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const double v = A[(e / m) * lda + (e % m)];
    s = fma(v, v, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double w[32];
  if (threadIdx.x % 32 == 0) w[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x / 32); ++k) t += w[k];
    atomicAdd(out, t);
  }
}

// s_i = sum_k x_ik^2 in FP64 for point-major X (d x n, ldx): vecnorm (include/dkernel.cu:102-114) in FP64
__global__ void rownorm_f64_kernel(const float* X, long long ldx, int n, int d, double* s) {
  const int lane = threadIdx.x % 32;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long i = blockIdx.x * (long long)(blockDim.x / 32) + threadIdx.x / 32; i < n; i += warps) {
    double acc = 0.0;
    for (int k = lane; k < d; k += 32) {
      const double x = X[i * ldx + k];
      acc = fma(x, x, acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s[i] = acc;
  }
}

// Sort v[0..n) descending in place (rank sort, one CTA, n <= 8192).
__global__ void sort_desc_kernel(double* v, int n) {
  extern __shared__ double sv[];
  for (int i = threadIdx.x; i < n; i += blockDim.x) sv[i] = v[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double x = sv[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double yj = sv[j];
      rank += (yj > x) || (yj == x && j < i);
    }
    v[rank] = x;
  }
}

__global__ void trace_kernel(const double* C, int ldc, int l, double* out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < l; i += blockDim.x) s += C[(long long)i * ldc + i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double w[32];
  if (threadIdx.x % 32 == 0) w[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x / 32); ++k) t += w[k];
    *out = t;
  }
}

// One-sided Jacobi (Hestenes) on the columns of an n x n matrix held in global memory, one CTA: every round
// orthogonalises n/2 disjoint column pairs (round-robin tournament order), one warp per pair.  The singular
// values are the final column norms.  status <- 1 if `max_sweeps` sweeps did not converge.
__global__ void __launch_bounds__(1024) jacobi_svd_kernel(double* A, int lda, int n, int max_sweeps, double tol,
                                                          double* S, int* status) {
  __shared__ unsigned long long worst;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nw = blockDim.x / 32;
  const int np = (n + 1) & ~1;  // even number of players; index n is a dummy when n is odd
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) worst = 0ull;
    __syncthreads();
    for (int round = 0; round < np - 1; ++round) {
      for (int k = warp; k < np / 2; k += nw) {
        int p = (k == 0) ? 0 : ((k + round - 1) % (np - 1)) + 1;
        int q = ((np - 1 - k + round - 1) % (np - 1)) + 1;
        if (p >= n || q >= n) continue;
        double* ap = A + (long long)p * lda;
        double* aq = A + (long long)q * lda;
        double al = 0, be = 0, ga = 0;
        for (int i = lane; i < n; i += 32) {
          const double x = ap[i], y = aq[i];
          al = fma(x, x, al);
          be = fma(y, y, be);
          ga = fma(x, y, ga);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, o);
          be += __shfl_xor_sync(0xffffffffu, be, o);
          ga += __shfl_xor_sync(0xffffffffu, ga, o);
        }
        const double denom = sqrt(al * be);
        const double ratio = (denom > 0.0) ? fabs(ga) / denom : 0.0;
        if (lane == 0) atomicMax(&worst, (unsigned long long)__double_as_longlong(ratio));
        if (ratio > tol) {
          const double zeta = (be - al) / (2.0 * ga);
          const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
          const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
          for (int i = lane; i < n; i += 32) {
            const double x = ap[i], y = aq[i];
            ap[i] = c * x - s * y;
            aq[i] = s * x + c * y;
          }
        }
      }
      __syncthreads();
    }
    if (__longlong_as_double((long long)worst) <= tol) break;
    __syncthreads();
  }
  for (int p = warp; p < n; p += nw) {
    const double* ap = A + (long long)p * lda;
    double s2 = 0;
    for (int i = lane; i < n; i += 32) s2 = fma(ap[i], ap[i], s2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    if (lane == 0) S[p] = sqrt(s2);
  }
  if (threadIdx.x == 0) *status = (sweep >= max_sweeps) ? 1 : 0;
}

inline unsigned grid_for(long long total, int threads, int cap) {
  long long b = (total + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

}  // namespace

template <typename TA, typename TBt>
int gram(db200_context* ctx, int n, int p, int q, const TA* A, long long lda, const TBt* B, long long ldb,
         const double* w, double alpha, double beta, double* C, int ldc, bool upper_only) {
  if (p <= 0 || q <= 0) return DB200_OK;
  scale_kernel<<<grid_for((long long)p * q, 256, 4096), 256, 0, ctx->stream>>>(C, ldc, p, q, beta, upper_only ? 1 : 0);
  count_launch(ctx);
  if (n <= 0) return DB200_OK;
  DmmArgs g;
  g.m = p;
  g.q = q;
  g.p = n;
  g.A = A;
  g.lda = lda;
  g.B = B;
  g.ldb = ldb;
  g.w = w;
  g.alpha = alpha;
  g.C = C;
  g.ldc = ldc;
  g.upper = upper_only ? 1 : 0;
  // Row splits, added with FP64 atomics: about eight waves of two CTAs per SM (upper tiles carry unequal strips, so
  // several waves are needed for the SMs to end together: with four, the busiest SM had 0.77 of its tensor pipe in use
  // and the idlest 0.55), no split shorter than 64 rows (a CTA's prologue and its atomics then outweigh its stages).
  const long long tp = (p + DMM_BM - 1) / DMM_BM, tq = (q + 63) / 64;
  const long long tiles = upper_only ? std::max(1LL, tp * tq / 2 + tp) : tp * tq;
  int splits = (int)std::max(1LL, std::min((long long)n / 64, 16LL * ctx->num_sms / tiles));
  g.kps = round_up((n + splits - 1) / splits, DMM_KS);
  splits = (n + g.kps - 1) / g.kps;
  g.epi = splits > 1 ? DMM_ATOMIC : DMM_ADD;
  return dmm_launch<TA, TBt, double, true, true>(ctx, g, splits);
}

template int gram<float, float>(db200_context*, int, int, int, const float*, long long, const float*, long long,
                                const double*, double, double, double*, int, bool);
template int gram<double, double>(db200_context*, int, int, int, const double*, long long, const double*, long long,
                                  const double*, double, double, double*, int, bool);
template int gram<double, float>(db200_context*, int, int, int, const double*, long long, const float*, long long,
                                 const double*, double, double, double*, int, bool);

template <typename TA, typename TC>
int gemm_tall(db200_context* ctx, int n, int p, int q, const TA* A, long long lda, const double* B, int ldb,
              bool transB, double beta, TC* C, long long ldc, double alpha, int tri) {
  if (n <= 0 || q <= 0) return DB200_OK;
  DmmArgs g;
  g.m = n;
  g.q = q;
  g.p = p;
  g.A = A;
  g.lda = lda;
  g.B = B;
  g.ldb = ldb;
  g.alpha = alpha;
  g.beta = beta;
  g.C = C;
  g.ldc = ldc;
  g.tri = tri;
  return transB ? dmm_launch<TA, double, TC, false, false>(ctx, g) : dmm_launch<TA, double, TC, false, true>(ctx, g);
}

template int gemm_tall<float, double>(db200_context*, int, int, int, const float*, long long, const double*, int,
                                      bool, double, double*, long long, double, int);
template int gemm_tall<double, double>(db200_context*, int, int, int, const double*, long long, const double*, int,
                                       bool, double, double*, long long, double, int);
template int gemm_tall<double, float>(db200_context*, int, int, int, const double*, long long, const double*, int,
                                      bool, double, float*, long long, double, int);
template int gemm_tall<float, float>(db200_context*, int, int, int, const float*, long long, const double*, int,
                                     bool, double, float*, long long, double, int);

// C (p x q, upper entries only) -= P^T P' for the k rows of a factored panel, in place (the Cholesky's updates)
static int syrk_update(db200_context* ctx, int k, int p, int q, const double* P, int ldp, double* C, int ldc) {
  DmmArgs g;
  g.m = p;
  g.q = q;
  g.p = k;
  g.A = P;
  g.lda = ldp;
  g.B = P;
  g.ldb = ldp;
  g.alpha = -1.0;
  g.C = C;
  g.ldc = ldc;
  g.upper = 1;
  g.epi = DMM_ADD;
  return dmm_launch<double, double, double, true, true>(ctx, g);
}

int potrf_upper(db200_context* ctx, double* A, int lda, int l, int* d_status, int* d_bad, int nb, double* W) {
  if (nb < 1 || nb > 64 || W) nb = 64;
  // up to l = 544 (the barrier's capacity matrices, the CholeskyQR2 and Nystrom Grams) the whole factor is one
  // launch on a thread-block cluster; an explicit smaller block size keeps the multi-kernel path
  if (nb == 64) {
    const int s = potrf_cluster(ctx, A, lda, l, d_status, d_bad, W);
    if (s != DB200_ERR_UNSUPPORTED) return s;
  }
  // (k0 is a multiple of nb: 16-byte loads need an even one too)
  const bool vec = reinterpret_cast<uintptr_t>(A) % 16 == 0 && lda % 2 == 0 && nb % 2 == 0;
  DB200_CUDA(ctx, cudaFuncSetAttribute(vec ? potrf_block_kernel<true> : potrf_block_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P64Smem)));
  // the diagonal-block kernel's arrival counter starts every factorisation at zero
  DB200_CUDA(ctx, cudaMemsetAsync(ctx->d_status + 1, 0, sizeof(int), ctx->stream));
  // A trailing matrix of at least one wave of 128 x 128 upper tiles takes its update on the FP64 tensor cores
  // (dmm_kernel, alpha = -1, added in place).  While the matrix beyond the next 8 nb columns is that large, the
  // factor goes by outer panels of 8 nb columns: each nb-block of the panel is factored (potrf_block_kernel, which
  // also solves its row to the last column), the panel's own later rows are updated at once (a strip of at most
  // 7 nb rows), and the trailing matrix takes one rank-8 nb update per panel instead of eight rank-nb ones
  // (measured at n = 16384 / 32768 with nb = 64: rank-64 updates 225 ms / -, rank-256 120 / 856 ms, rank-512
  // 105 / 755 ms).
  auto big = [&](int rest) {
    const int tp = (rest + GT - 1) / GT;
    return rest > 0 && tp * (tp + 1) / 2 >= ctx->num_sms;
  };
  for (int K0 = 0; K0 < l;) {
    const int rest0 = l - K0;
    const int KB = big(rest0 - 8 * nb) ? 8 * nb : (rest0 < nb ? rest0 : nb);
    for (int k0 = K0; k0 < K0 + KB; k0 += nb) {
      const int kb = (K0 + KB - k0 < nb) ? K0 + KB - k0 : nb;
      const int rest = l - k0 - kb;
      const unsigned ctas = rest > 64 ? (unsigned)((rest + 63) / 64) : 1u;
      if (vec)
        potrf_block_kernel<true><<<ctas, P64_THREADS, sizeof(P64Smem), ctx->stream>>>(A, lda, k0, kb, l, d_status,
                                                                                      d_bad, ctx->d_status + 1, W);
      else
        potrf_block_kernel<false><<<ctas, P64_THREADS, sizeof(P64Smem), ctx->stream>>>(A, lda, k0, kb, l, d_status,
                                                                                       d_bad, ctx->d_status + 1, W);
      count_launch(ctx);
      const int pr = K0 + KB - (k0 + kb);  // rows of this panel below the block
      if (pr > 0) {
        const double* P = A + (long long)(k0 + kb) * lda + k0;
        double* C = A + (long long)(k0 + kb) * lda + k0 + kb;
        const int s2 = syrk_update(ctx, kb, pr, rest, P, lda, C, lda);
        if (s2) return s2;
      }
    }
    const int rest = l - K0 - KB;
    if (rest > 0) {
      // trailing update A22 -= A12^T A12 (upper triangle only) with the panel's KB rows
      const double* P = A + (long long)(K0 + KB) * lda + K0;
      double* C = A + (long long)(K0 + KB) * lda + K0 + KB;
      if (KB > nb || big(rest)) {
        const int s2 = syrk_update(ctx, KB, rest, rest, P, lda, C, lda);
        if (s2) return s2;
      } else {
        // the r ~ 500..2000 capacity factors of the barrier: 32 x 32 tiles, so that they spread over the GPU
        const int nt = (rest + 31) / 32;
        syrk_update_kernel<<<nt * (nt + 1) / 2, 256, 0, ctx->stream>>>(P, lda, KB, rest, C, lda, d_status);
        count_launch(ctx);
      }
    }
    K0 += KB;
  }
  zero_lower_kernel<<<grid_for((long long)l * l, 256, 1024), 256, 0, ctx->stream>>>(A, lda, l);
  count_launch(ctx);
  DB200_CUDA(ctx, cudaGetLastError());
  return DB200_OK;
}

// X = R^-1 by block doubling: the 32 x 32 diagonal blocks by substitution, then for half = 32, 64, 128, ... every pair of
// inverted blocks X11, X22 (the second one possibly shorter) becomes one with X12 = -X11 R12 X22, two batched products per
// level on the FP64 tensor cores.  The first product is kept transposed, T^T = (R12 X22)^T, in the pair's place
// below the diagonal (q x half, exactly its shape), cleared before the next level reads the blocks.
static int trinv_doubling(db200_context* ctx, const double* R, int ldr, int l, double* X, int ldx) {
  trinv_diag_kernel<<<(l + TI * TI_WARPS - 1) / (TI * TI_WARPS), 32 * TI_WARPS, 0, ctx->stream>>>(R, ldr, l, X, ldx);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  for (int h = TI; h < l; h *= 2) {
    const int pairs = (l - h + 2 * h - 1) / (2 * h);  // pairs whose second half is not empty
    const int widest = std::min(h, l - h);            // rows of the longest second half
    const long long sr = 2LL * h * (ldr + 1LL), sx = 2LL * h * (ldx + 1LL);
    DmmArgs g;
    g.bl = l;
    g.bs = h;
    g.ldc = ldx;
    g.sC = sx;
    // T^T (q x h) = X22^T R12^T
    g.m = g.p = widest;
    g.q = h;
    g.vary = 1;
    g.A = X + h * (ldx + 1LL);
    g.lda = ldx;
    g.sA = sx;
    g.B = R + (long long)h * ldr;
    g.ldb = ldr;
    g.sB = sr;
    g.C = X + h;
    int st = dmm_launch<double, double, double, true, false>(ctx, g, 1, pairs);
    if (st) return st;
    // X12 (h x q) = -X11 T
    g.m = g.p = h;
    g.q = widest;
    g.vary = 2;
    g.A = X;
    g.B = X + h;
    g.ldb = ldx;
    g.sB = sx;
    g.C = X + (long long)h * ldx;
    g.alpha = -1.0;
    if ((st = dmm_launch<double, double, double, false, false>(ctx, g, 1, pairs))) return st;
    trinv_clear_kernel<<<dim3(grid_for((long long)h * widest, 256, 128), pairs), 256, 0, ctx->stream>>>(X, ldx, l, h);
    DB200_CUDA(ctx, cudaGetLastError());
    count_launch(ctx);
  }
  return DB200_OK;
}

// X = R^-1: the inverse X0 by block doubling and one correction, X = X0 + X0 (I - R X0).  The doubling's right residual
// R X - I grows at every level by that of X11: 4 to 8 times column substitution's for factors of condition 1e4 to 1e8, and
// 2e-7 against 1e-12 for the factor of an RBF kernel of 528 sorted points + 1e-7 I (against |R| |X| 2e-10 and 2e-16).  The
// correction brings it to substitution's (2e-16; a correction of every level's X12 does no better and takes five times
// the launches).  Bound by the launches' latency and the longest tile's reduction: db200_trsm_lutn of one column takes
// 266 us at l = 528 and 341 at l = 1024, of which the correction 62 and 112.  One warp per column doing its own back
// substitution over global memory, a chain of l dependent memory round trips, took 1.01 and 3.4 ms for the inverse alone.
int trinv_upper(db200_context* ctx, const double* R, int ldr, int l, double* X, int ldx, double* X0, double* D) {
  if (l <= TI) return trinv_doubling(ctx, R, ldr, l, X, ldx);  // one block, by substitution
  int st = trinv_doubling(ctx, R, ldr, l, X0, l);
  if (st) return st;
  // D = I - R X0 and X = X0 + X0 D, zeros below the diagonal included
  DmmArgs g;
  g.m = g.q = g.p = l;
  g.tri = kUpperB;
  g.tri_a = 1;
  g.epi = DMM_FROM;
  g.A = R;
  g.lda = ldr;
  g.B = X0;
  g.ldb = l;
  g.alpha = -1.0;
  g.C = D;
  g.ldc = l;
  if ((st = dmm_launch<double, double, double, false, true>(ctx, g))) return st;
  g.A = X0;
  g.lda = l;
  g.B = D;
  g.alpha = 1.0;
  g.S = X0;
  g.lds = l;
  g.C = X;
  g.ldc = ldx;
  return dmm_launch<double, double, double, false, true>(ctx, g);
}

int copy_upper(db200_context* ctx, const double* R, int ldr, int l, double* U, int ldu) {
  copy_upper_kernel<<<grid_for((long long)l * l, 256, 1024), 256, 0, ctx->stream>>>(R, ldr, l, U, ldu);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int trsv_pair(db200_context* ctx, const double* R, int ld, int l, const double* W, double* x) {
  if (l > TV_MAX_L) return fail(ctx, DB200_ERR_UNSUPPORTED, "trsv: l > 4096");
  trsv_pair_kernel<<<1, TV_THREADS, 0, ctx->stream>>>(R, ld, l, W, x);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int symmetrize(db200_context* ctx, double* C, int ldc, int l, double shift) {
  symmetrize_kernel<<<grid_for((long long)l * l, 256, 1024), 256, 0, ctx->stream>>>(C, ldc, l, shift);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int mirror_upper(db200_context* ctx, double* C, int ldc, int l) {
  fill_upper_from_lower_kernel<<<grid_for((long long)l * l, 256, 1024), 256, 0, ctx->stream>>>(C, ldc, l);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

template <typename TS, typename TD>
int convert(db200_context* ctx, const TS* src, long long lds, TD* dst, long long ldd, int m, int n) {
  convert_kernel<TS, TD><<<grid_for((long long)m * n, 256, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(src, lds, dst,
                                                                                                     ldd, m, n);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}
template int convert<double, float>(db200_context*, const double*, long long, float*, long long, int, int);
template int convert<float, double>(db200_context*, const float*, long long, double*, long long, int, int);
template int convert<double, double>(db200_context*, const double*, long long, double*, long long, int, int);
template int convert<float, float>(db200_context*, const float*, long long, float*, long long, int, int);

int jacobi_svd_values(db200_context* ctx, double* A, int lda, int n, double* S, int* d_status) {
  jacobi_svd_kernel<<<1, 1024, 0, ctx->stream>>>(A, lda, n, 40, 1e-15, S, d_status);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int axpby_f32(db200_context* ctx, float* C, long long ldc, const double* T, long long ldt, int m, int n,
              double alpha, double beta) {
  axpby_f32_kernel<<<grid_for((long long)m * n, 256, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(C, ldc, T, ldt, m, n,
                                                                                                alpha, beta);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int sumsq_f32(db200_context* ctx, const float* A, long long lda, int m, int n, double* d_out) {
  sumsq_f32_kernel<<<grid_for((long long)m * n, 256, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(A, lda, m, n, d_out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

// The FP64 kernel block in one launch: cross terms on the FP64 tensor cores over the d features, the norms, exp and
// labels in the epilogue, K written once.  Bound by the d-long products and the exp (131072 x 1024, d = 64: 0.46 ms
// of tensor pipe, 0.17 ms of stores); clearing K, a Gram added into it and a second pass over it took 3.4 ms.
int rbf_block_f64_fused(db200_context* ctx, int m, int n, int d, const float* Xi, long long ldxi, const float* Xj,
                        long long ldxj, const double* si, const double* sj, const float* yi, const float* yj,
                        double gamma, double* K, long long ldk) {
  DmmArgs g;
  g.m = m;
  g.q = n;
  g.p = d;
  g.A = Xi;
  g.lda = ldxi;
  g.B = Xj;
  g.ldb = ldxj;
  g.C = K;
  g.ldc = ldk;
  g.epi = DMM_RBF;
  g.si = si;
  g.sj = sj;
  g.yi = yi;
  g.yj = yj;
  g.gamma = gamma;
  return dmm_launch<float, float, double, true, true>(ctx, g);
}

int rownorm_f64(db200_context* ctx, const float* X, long long ldx, int n, int d, double* s) {
  rownorm_f64_kernel<<<grid_for((long long)n * 32, 256, 16 * ctx->num_sms), 256, 0, ctx->stream>>>(X, ldx, n, d, s);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int sort_desc(db200_context* ctx, double* v, int n) {
  if (n > 8192) return fail(ctx, DB200_ERR_UNSUPPORTED, "sort_desc: n > 8192");
  sort_desc_kernel<<<1, 1024, sizeof(double) * n, ctx->stream>>>(v, n);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int trace(db200_context* ctx, const double* C, int ldc, int l, double* d_out) {
  trace_kernel<<<1, 1024, 0, ctx->stream>>>(C, ldc, l, d_out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

}  // namespace db200
