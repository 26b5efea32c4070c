// Learned Nystrom landmarks: k-NN distance features, the leverage MLP (forward, backward, Adam, all hand-written
// kernels), Gumbel top-k selection, the landmark Nystrom factor, a sampled residual estimate and ridge leverage
// scores from a low-rank factor.
//
// The reference always sketches with a Gaussian test matrix (include/dkernel.h:13-46, tests/testsvm.cpp:94-134);
// this file replaces Omega by r landmark columns of K when a model of the ridge leverage scores picks landmarks
// whose Nystrom factor meets a residual tolerance.  The factor is the column form of the Nystrom approximation,
// K ~ K(:, L) K(L, L)^-1 K(L, :), with the same y-folding as the sketch (Q = diag(y) K diag(y), dkernel.cu:125).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_bf16.h>

#include "internal.h"
#include "la64.h"

struct db200_mlp {
  int in = 0, width = 0, hidden = 0, layers = 0, nparams = 0, device = 0;
  float* master = nullptr;        // fp32 parameters
  float* grad = nullptr;          // fp32 gradient of the last call
  float* mom1 = nullptr;          // Adam first moment
  float* mom2 = nullptr;          // Adam second moment
  __nv_bfloat16* wbf = nullptr;   // bf16 copy of the parameters used by the forward and backward passes
  float* in_mean = nullptr;
  float* in_scale = nullptr;
  double* d_loss = nullptr;
  long long step = 0;
  void* act = nullptr;            // activations / backward buffers, grow-only
  size_t act_bytes = 0;
  std::vector<int> off_w, off_b, fan_in, fan_out;
};

namespace db200 {

namespace {

inline unsigned blocks_for(long long total, int threads, long long cap = 65535LL * 16) {
  long long b = (total + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

// ------------------------------------------------------------------ k-NN distance
// One thread per query point, the query in registers (DMAX >= d), reference points staged through shared memory
// 64 at a time; the k smallest squared distances are kept sorted in registers.
constexpr int KNN_THREADS = 128, KNN_TILE = 64, KNN_KMAX = 16;

template <int DMAX>
__global__ void __launch_bounds__(KNN_THREADS) knn_kernel(int n, int d, const float* __restrict__ X, int ldx, int s,
                                                          const int* __restrict__ ref, int k, float* __restrict__ out) {
  __shared__ float sR[KNN_TILE][DMAX + 1];
  __shared__ int sI[KNN_TILE];
  const int i = blockIdx.x * KNN_THREADS + threadIdx.x;
  float q[DMAX];
#pragma unroll
  for (int c = 0; c < DMAX; ++c) q[c] = (i < n && c < d) ? X[(long long)i * ldx + c] : 0.f;
  float best[KNN_KMAX];
#pragma unroll
  for (int t = 0; t < KNN_KMAX; ++t) best[t] = INFINITY;
  for (int t0 = 0; t0 < s; t0 += KNN_TILE) {
    __syncthreads();
    for (int e = threadIdx.x; e < KNN_TILE * DMAX; e += KNN_THREADS) {
      const int jj = e / DMAX, c = e % DMAX;
      const int j = t0 + jj;
      sR[jj][c] = (j < s && c < d) ? X[(long long)ref[j] * ldx + c] : 0.f;
    }
    if (threadIdx.x < KNN_TILE) sI[threadIdx.x] = (t0 + threadIdx.x < s) ? ref[t0 + threadIdx.x] : -1;
    __syncthreads();
    const int cnt = min(KNN_TILE, s - t0);
    for (int jj = 0; jj < cnt; ++jj) {
      float dist = 0.f;
#pragma unroll
      for (int c = 0; c < DMAX; ++c) {
        const float df = q[c] - sR[jj][c];
        dist = fmaf(df, df, dist);
      }
      if (sI[jj] == i) continue;  // a point is not its own neighbour
      if (dist < best[KNN_KMAX - 1]) {
        // insertion into the sorted list (only the first k entries are used)
#pragma unroll
        for (int t = KNN_KMAX - 1; t > 0; --t) {
          const bool shift = dist < best[t - 1];
          best[t] = shift ? best[t - 1] : (dist < best[t] ? dist : best[t]);
        }
        if (dist < best[0]) best[0] = dist;
      }
    }
  }
  if (i < n) {
    float v = best[0];
#pragma unroll
    for (int t = 0; t < KNN_KMAX; ++t)
      if (t == k - 1) v = best[t];
    out[i] = sqrtf(v);
  }
}

// Rows ref[j] of X (point-major) gathered into R (s x d, point-major with leading dimension d).
__global__ void gather_rows_kernel(const float* __restrict__ X, int ldx, const int* __restrict__ ref, int s, int d,
                                   float* __restrict__ R) {
  const long long total = (long long)s * d;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(e / d), c = (int)(e % d);
    R[e] = X[(long long)ref[j] * ldx + c];
  }
}

// out[i] = sqrt of the k-th smallest of the `cand` candidates part[cand i ..] (sorted lists of 8).
__global__ void knn_merge_kernel(int n, const float* __restrict__ part, int cand, int k, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float best[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) best[t] = INFINITY;
  const float4* p = reinterpret_cast<const float4*>(part + (size_t)i * cand);
#pragma unroll 2
  for (int c = 0; c < cand / 4; ++c) {
    const float4 q = p[c];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = e == 0 ? q.x : e == 1 ? q.y : e == 2 ? q.z : q.w;
#pragma unroll
      for (int t = 7; t > 0; --t) best[t] = fminf(best[t], fmaxf(best[t - 1], x));
      best[0] = fminf(best[0], x);
    }
  }
  float v = best[0];
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (t == k - 1) v = best[t];
  out[i] = sqrtf(fmaxf(v, 0.0f));
}


// F[i, :] = [x_i (d), ||x_i||, knn_i], row major n x (d + 2); one warp per point.
__global__ void features_kernel(int n, int d, const float* __restrict__ X, int ldx, const float* __restrict__ knn,
                                float* __restrict__ F) {
  const int lane = threadIdx.x % 32;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long i = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; i < n; i += warps) {
    float ss = 0.f;
    float* row = F + i * (d + 2);
    for (int c = lane; c < d; c += 32) {
      const float x = X[i * ldx + c];
      row[c] = x;
      ss = fmaf(x, x, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) {
      row[d] = sqrtf(ss);
      row[d + 1] = knn[i];
    }
  }
}

// lev_i = sum_c W(i, c)^2, W n x r column major (FP64)
__global__ void row_sumsq64_kernel(int n, int r, const double* __restrict__ W, long long ldw, double* __restrict__ lev) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int c = 0; c < r; ++c) {
      const double v = W[(long long)c * ldw + i];
      s = fma(v, v, s);
    }
    lev[i] = s;
  }
}

// ------------------------------------------------------------------ gathers
__global__ void gather_rows_f32_kernel(const float* __restrict__ X, int ldx, const int* __restrict__ idx, int r, int d,
                                       float* __restrict__ out) {
  const long long total = (long long)r * d;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(e / d), c = (int)(e % d);
    out[e] = X[(long long)idx[a] * ldx + c];
  }
}
__global__ void gather_f32_kernel(const float* __restrict__ v, const int* __restrict__ idx, int r, float* __restrict__ out) {
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < r; a += gridDim.x * blockDim.x) out[a] = v[idx[a]];
}
// out(a, b) = M(idx[a], b), M column major (ldm) with `cols` columns, out column major r x cols (ld r)
template <typename TS>
__global__ void gather_matrix_rows_kernel(const TS* __restrict__ M, long long ldm, const int* __restrict__ idx, int r,
                                          int cols, double* __restrict__ out) {
  const long long total = (long long)r * cols;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(e % r), b = (int)(e / r);
    out[e] = (double)M[(long long)b * ldm + idx[a]];
  }
}

// ------------------------------------------------------------------ Gumbel keys and radix selection
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  // splitmix64 finaliser (Vigna): a bijective avalanche mix of a 64-bit counter
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__global__ void gumbel_kernel(int n, const float* __restrict__ logits, unsigned long long seed, float* __restrict__ keys) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned long long h = mix64(seed * 0x9e3779b97f4a7c15ull + (unsigned long long)i + 1ull);
    // uniform in (0, 1) from the top 53 bits
    const double u = ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    keys[i] = logits[i] + (float)(-log(-log(u)));
  }
}
__device__ __forceinline__ unsigned int key_bits(float f) {
  const unsigned int b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);  // order preserving: larger float -> larger unsigned
}
// histogram of byte `shift` of the keys whose higher bytes equal `prefix` (under `mask`)
__global__ void radix_hist_kernel(int n, const float* __restrict__ keys, unsigned int prefix, unsigned int mask, int shift,
                                  unsigned int* __restrict__ hist) {
  __shared__ unsigned int h[256];
  for (int b = threadIdx.x; b < 256; b += blockDim.x) h[b] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned int u = key_bits(keys[i]);
    if ((u & mask) == prefix) atomicAdd(&h[(u >> shift) & 0xFFu], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < 256; b += blockDim.x)
    if (h[b]) atomicAdd(&hist[b], h[b]);
}
// indices with key > thr, and the first `ties` (by arrival) with key == thr
__global__ void radix_compact_kernel(int n, const float* __restrict__ keys, unsigned int thr, int ties,
                                     unsigned int* __restrict__ counters, int* __restrict__ idx) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned int u = key_bits(keys[i]);
    if (u > thr) {
      idx[atomicAdd(&counters[0], 1u)] = i;
    } else if (u == thr) {
      const unsigned int t = atomicAdd(&counters[1], 1u);
      if ((int)t < ties) idx[atomicAdd(&counters[0], 1u)] = i;
    }
  }
}

// ------------------------------------------------------------------ MLP
// C(i, j) = sum_k A(i, k) B(k, j) in fp32, every output one fused-multiply-add chain over ascending k (activations are
// rounded to bf16 between layers, so another order of the sums would move later layers by whole bf16 steps).
// AK / BK: k is the contiguous index (A[i * lda + k], B[j * ldb + k]), else i / j is (A[k * lda + i], B[k * ldb + j]).
//
// Bound by the FP32 pipe.  128 x 128 per CTA of 256 threads; a warp owns 64 x 32, a lane 8 x 8 as two by two 4 x 4 blocks,
// so that a k step is four conflict-free 16-byte shared loads for 32 packed multiply-adds (fma.rn.f32x2: two outputs per
// instruction, each rounded as fmaf).  Stages of 16 k are fetched into registers one stage ahead (16-byte pieces where
// the operand's rows allow it), converted to fp32 and parked [k][row] in a double buffer.  One training
// step's products over 16384 rows of the 66 -> 256 x 3 -> 1 net take 425 us (37 TFLOP/s); 64 x 64 tiles with 4 x 4 outputs
// and scalar loads took 800, 128 x 256 tiles (fewer shared loads, one CTA per SM) 455.  grid.z splits k (EPI_ATOMIC only).
enum { EPI_HIDDEN = 0, EPI_DH = 2, EPI_ATOMIC = 3 };
constexpr int MT = 128, MK = 16, MLD = MT + 4;

__device__ __forceinline__ float tof(float v) { return v; }
__device__ __forceinline__ float tof(__nv_bfloat16 v) { return __bfloat162float(v); }

// One operand's stage: entries (r0 + 0..127, k0 + 0..15), zero outside (rows, k1).  8 values per thread.
template <typename T, bool KC, bool VEC>
__device__ __forceinline__ void mlp_fetch(float (&v)[8], const T* X, long long ld, int r0, int rows, int k0, int k1) {
  const int t = threadIdx.x;
  const int r = KC ? t / 2 : (t % 16) * 8, k = KC ? (t % 2) * 8 : t / 16;  // first of 8 along the contiguous index
  const T* p = X + (KC ? (long long)(r0 + r) * ld + k0 + k : (long long)(k0 + k) * ld + r0 + r);
  const bool in = KC ? r0 + r < rows : k0 + k < k1;
  const int left = in ? (KC ? k1 - (k0 + k) : rows - (r0 + r)) : 0;
  if (VEC && left >= 8) {
    if constexpr (sizeof(T) == 2) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // bf16 is the upper half of an fp32
        v[2 * e] = __uint_as_float(w[e] << 16);
        v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
      }
    } else {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = e < left ? tof(p[e]) : 0.f;
  }
}
template <bool KC>
__device__ __forceinline__ void mlp_park(float (*s)[MLD], const float (&v)[8]) {
  const int t = threadIdx.x;
  if (KC) {
#pragma unroll
    for (int e = 0; e < 8; ++e) s[(t % 2) * 8 + e][t / 2] = v[e];
  } else {
    float4* d = reinterpret_cast<float4*>(&s[t / 16][(t % 16) * 8]);
    d[0] = make_float4(v[0], v[1], v[2], v[3]);
    d[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

template <typename TA, typename TB, bool AK, bool BK, bool VEC, int EPI>
__global__ void __launch_bounds__(256, 2) mlp_gemm_kernel(int M, int N, int K, const TA* __restrict__ A, long long lda,
                                                          const TB* __restrict__ B, long long ldb,
                                                          const float* __restrict__ bias,
                                                          const __nv_bfloat16* __restrict__ H, void* Cv, long long ldc,
                                                          int k_per_split) {
  __shared__ __align__(16) float sA[2][MK][MLD];
  __shared__ __align__(16) float sB[2][MK][MLD];
  const int i0 = blockIdx.x * MT, j0 = blockIdx.y * MT;
  const int kb = blockIdx.z * k_per_split, ke = min(K, kb + k_per_split);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ri = 64 * (warp % 2) + 4 * (lane / 4), cj = 32 * (warp / 2) + 4 * (lane % 4);  // + 32 rows, + 16 columns
  unsigned long long acc[8][4];  // rows ri + 0..3, ri + 32 + 0..3; column pairs cj + {0,1}, {2,3}, + 16 + {0,1}, {2,3}
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0ull;
  float va[8], vb[8];
  mlp_fetch<TA, AK, VEC>(va, A, lda, i0, M, kb, ke);
  mlp_fetch<TB, BK, VEC>(vb, B, ldb, j0, N, kb, ke);
  mlp_park<AK>(sA[0], va);
  mlp_park<BK>(sB[0], vb);
  __syncthreads();
  int buf = 0;
  for (int k0 = kb; k0 < ke; k0 += MK, buf ^= 1) {
    const bool more = k0 + MK < ke;
    if (more) {
      mlp_fetch<TA, AK, VEC>(va, A, lda, i0, M, k0 + MK, ke);
      mlp_fetch<TB, BK, VEC>(vb, B, ldb, j0, N, k0 + MK, ke);
    }
#pragma unroll
    for (int t = 0; t < MK; ++t) {
      const float4 a0 = *reinterpret_cast<const float4*>(&sA[buf][t][ri]);
      const float4 a1 = *reinterpret_cast<const float4*>(&sA[buf][t][ri + 32]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&sB[buf][t][cj]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&sB[buf][t][cj + 16]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const unsigned long long bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const unsigned long long aa = pack2(av[a], av[a]);
#pragma unroll
        for (int b = 0; b < 4; ++b)
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[a][b]) : "l"(aa), "l"(bv[b]));
      }
    }
    if (more) {  // the other buffer was last read one stage ago, before the barrier that ended it
      mlp_park<AK>(sA[buf ^ 1], va);
      mlp_park<BK>(sB[buf ^ 1], vb);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int i = i0 + ri + (a < 4 ? a : 28 + a);
    if (i >= M) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float2 o = unpack2(acc[a][b]);
      const int j = j0 + cj + (b < 2 ? 2 * b : 12 + 2 * b);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (j + e >= N) continue;
        const float v = e ? o.y : o.x;
        const long long at = i * ldc + j + e;
        if (EPI == EPI_HIDDEN) {
          static_cast<__nv_bfloat16*>(Cv)[at] = __float2bfloat16_rn(fmaxf(v + bias[j + e], 0.f));
        } else if (EPI == EPI_DH) {
          static_cast<float*>(Cv)[at] = (__bfloat162float(H[at]) > 0.f) ? v : 0.f;
        } else {
          atomicAdd(static_cast<float*>(Cv) + at, v);
        }
      }
    }
  }
}

// The output layer (one unit).  Forward: out_i = sum_k H(i, k) w_k + b, one chain per row, a thread per row.
template <bool VEC>
__global__ void __launch_bounds__(128) mlp_out_kernel(int m, int K, const __nv_bfloat16* __restrict__ H,
                                                      const __nv_bfloat16* __restrict__ w, const float* __restrict__ b,
                                                      float* __restrict__ out) {
  extern __shared__ float sw[];
  for (int k = threadIdx.x; k < K; k += blockDim.x) sw[k] = tof(w[k]);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const __nv_bfloat16* h = H + (long long)i * K;
  float acc = 0.f;
  int k = 0;
  if (VEC) {
#pragma unroll 4
    for (; k + 8 <= K; k += 8) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(h + k));
      const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc = fmaf(__uint_as_float(u[e] << 16), sw[k + 2 * e], acc);
        acc = fmaf(__uint_as_float(u[e] & 0xffff0000u), sw[k + 2 * e + 1], acc);
      }
    }
  }
  for (; k < K; ++k) acc = fmaf(tof(h[k]), sw[k], acc);
  out[i] = acc + *b;
}
// Backward of the output layer in one pass over H (m x K): dw_k += sum_i d_i H(i, k), db += sum_i d_i and
// dX(i, k) = d_i w_k where H(i, k) > 0.  A thread per column k, the rows split over blockIdx.y.
__global__ void __launch_bounds__(256) mlp_out_backward_kernel(int m, int K, const float* __restrict__ d,
                                                               const __nv_bfloat16* __restrict__ H,
                                                               const __nv_bfloat16* __restrict__ w, int rows,
                                                               float* __restrict__ dX, float* dw, float* db) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int r0 = blockIdx.y * rows, r1 = min(m, r0 + rows);
  if (k < K) {
    const float wk = tof(w[k]);
    float s = 0.f;
#pragma unroll 4
    for (int i = r0; i < r1; ++i) {
      const float h = tof(H[(long long)i * K + k]), di = __ldg(d + i);
      s = fmaf(di, h, s);
      dX[(long long)i * K + k] = h > 0.f ? di * wk : 0.f;
    }
    atomicAdd(dw + k, s);
  }
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    float s = 0.f;
    for (int i = r0 + threadIdx.x; i < r1; i += 32) s += d[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) atomicAdd(db, s);
  }
}

__global__ void standardize_kernel(int m, int in, const float* __restrict__ F, const float* __restrict__ mean,
                                   const float* __restrict__ scale, __nv_bfloat16* __restrict__ H0) {
  const long long total = (long long)m * in;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(e % in);
    H0[e] = __float2bfloat16_rn((F[e] - mean[c]) * scale[c]);
  }
}
// dout = (out - t) / m, loss += 0.5 (out - t)^2 / m
__global__ void mse_kernel(int m, const float* __restrict__ out, const float* __restrict__ t, float* __restrict__ dout,
                           double* loss) {
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const float r = out[i] - t[i];
    dout[i] = r / (float)m;
    s += 0.5 * (double)r * (double)r / (double)m;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x % 32 == 0) atomicAdd(loss, s);
}
// g[j] += sum_i dY[i*N + j], a thread per column, the rows split over blockIdx.y
__global__ void __launch_bounds__(256) colsum_kernel(int m, int N, int rows, const float* __restrict__ dY, float* g) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const int r1 = min(m, ((int)blockIdx.y + 1) * rows);
  float s = 0.f;
#pragma unroll 8
  for (int i = blockIdx.y * rows; i < r1; ++i) s += __ldg(dY + (long long)i * N + j);
  atomicAdd(g + j, s);
}
__global__ void adam_kernel(int np, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                            float* __restrict__ m2, __nv_bfloat16* __restrict__ wbf, float lr, float c1, float c2) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < np; e += gridDim.x * blockDim.x) {
    const float gi = g[e];
    const float a = 0.9f * m1[e] + 0.1f * gi;
    const float b = 0.999f * m2[e] + 0.001f * gi * gi;
    m1[e] = a;
    m2[e] = b;
    const float v = w[e] - lr * (a * c1) / (sqrtf(b * c2) + 1e-8f);
    w[e] = v;
    wbf[e] = __float2bfloat16_rn(v);
  }
}
__global__ void to_bf16_kernel(int np, const float* __restrict__ w, __nv_bfloat16* __restrict__ wbf) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < np; e += gridDim.x * blockDim.x) wbf[e] = __float2bfloat16_rn(w[e]);
}

template <typename TA, typename TB, bool AK, bool BK, int EPI>
int mlp_gemm(db200_context* ctx, int M, int N, int K, const TA* A, long long lda, const TB* B, long long ldb,
             const float* bias, const __nv_bfloat16* H, void* C, long long ldc, int splits = 1) {
  if (M <= 0 || N <= 0) return DB200_OK;
  int kps = (K + splits - 1) / splits;
  kps = round_up(kps < MK ? MK : kps, MK);
  splits = std::max(1, (K + kps - 1) / kps);
  const dim3 grid((M + MT - 1) / MT, (N + MT - 1) / MT, splits);
  if (grid.y > 65535 || grid.z > 65535) return fail(ctx, DB200_ERR_UNSUPPORTED, "mlp: GEMM too large");
  // 16-byte pieces: aligned bases and rows
  const bool vec = reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0 &&
                   lda * (long long)sizeof(TA) % 16 == 0 && ldb * (long long)sizeof(TB) % 16 == 0;
  if (vec)
    mlp_gemm_kernel<TA, TB, AK, BK, true, EPI><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, bias, H, C, ldc,
                                                                              kps);
  else
    mlp_gemm_kernel<TA, TB, AK, BK, false, EPI><<<grid, 256, 0, ctx->stream>>>(M, N, K, A, lda, B, ldb, bias, H, C, ldc,
                                                                               kps);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

// activation buffers of one forward/backward over m rows
struct MlpActs {
  __nv_bfloat16* h[8];  // h[0] = standardised input (m x in), h[l] = layer l output (m x width), l = 1..hidden
  float* out;           // m
  float* dy0;           // m x max(width, 1)
  float* dy1;
};

int mlp_acts(db200_context* ctx, db200_mlp* net, int m, MlpActs* A) {
  const size_t hb = align_up((size_t)m * std::max(net->in, net->width) * 2, 256);
  const size_t need = (size_t)(net->hidden + 1) * hb + align_up((size_t)m * 4, 256) +
                      2 * align_up((size_t)m * net->width * 4, 256) + 1024;
  if (need > net->act_bytes) {
    DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (net->act) cudaFree(net->act);
    net->act = nullptr;
    net->act_bytes = 0;
    DB200_CUDA(ctx, cudaMalloc(&net->act, need));
    net->act_bytes = need;
  }
  Carve cv{static_cast<char*>(net->act)};
  for (int l = 0; l <= net->hidden; ++l) A->h[l] = reinterpret_cast<__nv_bfloat16*>(cv.take<char>(hb));
  A->out = cv.take<float>(m);
  A->dy0 = cv.take<float>((size_t)m * net->width);
  A->dy1 = cv.take<float>((size_t)m * net->width);
  return DB200_OK;
}

int mlp_forward_impl(db200_context* ctx, db200_mlp* net, int m, const float* F, MlpActs& A) {
  standardize_kernel<<<blocks_for((long long)m * net->in, 256), 256, 0, ctx->stream>>>(m, net->in, F, net->in_mean,
                                                                                         net->in_scale, A.h[0]);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  int st;
  for (int l = 0; l < net->layers; ++l) {
    const int K = net->fan_in[l], N = net->fan_out[l];
    const __nv_bfloat16* W = net->wbf + net->off_w[l];
    const float* b = net->master + net->off_b[l];
    if (l < net->hidden) {
      st = mlp_gemm<__nv_bfloat16, __nv_bfloat16, true, true, EPI_HIDDEN>(ctx, m, N, K, A.h[l], K, W, K, b, nullptr,
                                                                         A.h[l + 1], N);
    } else {
      const bool vec = K % 8 == 0;  // (A.h is 256-byte aligned)
      if (vec)
        mlp_out_kernel<true><<<(m + 127) / 128, 128, sizeof(float) * K, ctx->stream>>>(m, K, A.h[l], W, b, A.out);
      else
        mlp_out_kernel<false><<<(m + 127) / 128, 128, sizeof(float) * K, ctx->stream>>>(m, K, A.h[l], W, b, A.out);
      DB200_CUDA(ctx, cudaGetLastError());
      count_launch(ctx);
      st = DB200_OK;
    }
    if (st) return st;
  }
  return DB200_OK;
}

// gradient of 0.5 mean (out - t)^2 into net->grad; loss into net->d_loss
int mlp_backward_impl(db200_context* ctx, db200_mlp* net, int m, const float* target, MlpActs& A) {
  DB200_CUDA(ctx, cudaMemsetAsync(net->grad, 0, sizeof(float) * net->nparams, ctx->stream));
  DB200_CUDA(ctx, cudaMemsetAsync(net->d_loss, 0, sizeof(double), ctx->stream));
  mse_kernel<<<blocks_for(m, 256, 1024), 256, 0, ctx->stream>>>(m, A.out, target, A.dy0, net->d_loss);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  float* dY = A.dy0;  // gradient at the output of layer l (m x fan_out[l])
  float* dX = A.dy1;
  // rows of one split of the sums over m: enough CTAs for two per SM, at least 64 rows each
  auto split_rows = [&](long long tiles) -> int {
    const long long want = std::max(1LL, 2LL * ctx->num_sms / tiles);
    return (int)std::max(64LL, (m + want - 1) / want);
  };
  int st;
  for (int l = net->layers - 1; l >= 0; --l) {
    const int K = net->fan_in[l], N = net->fan_out[l];
    if (l == net->hidden) {  // one unit: its weights' and bias's gradient and dH_{l-1} in one pass
      const int rows = split_rows((K + 255) / 256);
      mlp_out_backward_kernel<<<dim3((K + 255) / 256, (m + rows - 1) / rows), 256, 0, ctx->stream>>>(
          m, K, dY, A.h[l], net->wbf + net->off_w[l], rows, dX, net->grad + net->off_w[l], net->grad + net->off_b[l]);
      DB200_CUDA(ctx, cudaGetLastError());
      count_launch(ctx);
      std::swap(dY, dX);
      continue;
    }
    // dW_l (N x K) = dY^T H_l  (sum over the m rows, split with atomics)
    const int wrows = split_rows((long long)((N + MT - 1) / MT) * ((K + MT - 1) / MT));
    if ((st = mlp_gemm<float, __nv_bfloat16, false, false, EPI_ATOMIC>(ctx, N, K, m, dY, N, A.h[l], K, nullptr, nullptr,
                                                                       net->grad + net->off_w[l], K,
                                                                       (m + wrows - 1) / wrows)))
      return st;
    const int crows = split_rows((N + 255) / 256);
    colsum_kernel<<<dim3((N + 255) / 256, (m + crows - 1) / crows), 256, 0, ctx->stream>>>(m, N, crows, dY,
                                                                                         net->grad + net->off_b[l]);
    DB200_CUDA(ctx, cudaGetLastError());
    count_launch(ctx);
    if (l > 0) {
      // dH_{l-1} (m x K) = (dY W_l) masked by ReLU'(H_{l-1})
      if ((st = mlp_gemm<float, __nv_bfloat16, true, false, EPI_DH>(ctx, m, K, N, dY, N, net->wbf + net->off_w[l], K,
                                                                   nullptr, A.h[l], dX, K)))
        return st;
      std::swap(dY, dX);
    }
  }
  return DB200_OK;
}

// Uniform sample of s distinct indices of [0, n) (partial Fisher-Yates, seeded), sorted.
std::vector<int> sample_indices(int n, int s, unsigned long long seed) {
  s = std::min(s, n);
  std::vector<int> p(n);
  for (int i = 0; i < n; ++i) p[i] = i;
  std::mt19937_64 g(seed);
  for (int i = 0; i < s; ++i) {
    std::uniform_int_distribution<int> u(i, n - 1);
    std::swap(p[i], p[u(g)]);
  }
  p.resize(s);
  std::sort(p.begin(), p.end());
  return p;
}

struct LandTimer {
  cudaStream_t s;
  cudaEvent_t a = nullptr, b = nullptr;
  explicit LandTimer(cudaStream_t st) : s(st) {
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a, s);
  }
  double stop() {
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
  }
  ~LandTimer() {
    cudaEventDestroy(a);
    cudaEventDestroy(b);
  }
};

}  // namespace

// ------------------------------------------------------------------ internal entry points (shared with C ABI)
int knn_distance(db200_context* ctx, int n, int d, const float* X, int ldx, int s, const int* ref, int k, float* out) {
  if (k <= 8 && d <= 128) {
    // On the tensor cores: squared distances |x_i|^2 + |x_j|^2 - 2 x_i.x_j from the tile engine's split-fp16
    // distance GEMM (22 significant bits per coordinate), each row's 8 smallest per column quarter kept in
    // registers (RBF_MODE_KNN), then the quarters merged.  The reference points are gathered and packed as the
    // second point set; their indices skip each point's own distance.
    const int dp = feature_pad(d), npad = point_pad(n), spad = point_pad(s);
    // ranges of the reference points, so that the query blocks fill the GPU: a list of 8 per quarter and range
    const int split = tile_split(ctx, npad / 256, spad / 128, 1, 2, 2), ranges = (spad / 128 + split - 1) / split;
    const size_t bytes = 4096 + (size_t)s * d * 4 + (size_t)npad * 2 * dp * 2 + packed_norm_floats(npad) * 4 +
                         (size_t)spad * 2 * dp * 2 + packed_norm_floats(spad) * 4 + (size_t)n * 32 * ranges * 4 + 8 * 256;
    char* ws = static_cast<char*>(workspace(ctx, bytes));
    if (!ws) return DB200_ERR_NOMEM;
    Carve cv{ws};
    float* R = cv.take<float>((size_t)s * d);
    void* xq = cv.take<uint16_t>((size_t)npad * 2 * dp);
    float* nq = cv.take<float>(packed_norm_floats(npad));
    void* xr = cv.take<uint16_t>((size_t)spad * 2 * dp);
    float* nr = cv.take<float>(packed_norm_floats(spad));
    float* part = cv.take<float>((size_t)n * 32 * ranges);
    gather_rows_kernel<<<blocks_for((long long)s * d, 256, 65535LL * 8), 256, 0, ctx->stream>>>(X, ldx, ref, s, d, R);
    DB200_CUDA(ctx, cudaGetLastError());
    count_launch(ctx);
    int st = pack_points(ctx, X, ldx, DB200_POINT_MAJOR, n, d, dp, npad, xq, nq);
    if (!st) st = pack_points(ctx, R, d, DB200_POINT_MAJOR, s, d, dp, spad, xr, nr);
    if (st) return st;
    TileJob J;
    J.pi.xp = xq;
    J.pi.norms = nq;
    J.pi.n = n;
    J.pi.npad = npad;
    J.pi.dp = dp;
    J.pj.xp = xr;
    J.pj.norms = nr;
    J.pj.n = s;
    J.pj.npad = spad;
    J.pj.dp = dp;
    J.yj = reinterpret_cast<const float*>(ref);  // the reference points' indices (RBF_MODE_KNN)
    J.gamma = 1.0f;
    J.out = part;
    J.ldo = 32;
    J.split_tiles = split;
    TilePlan T;
    if ((st = prepare_rbf_tiles(ctx, RBF_MODE_KNN, &J, 1, nullptr, 0, &T))) return st;
    if ((st = launch_rbf_plan(ctx, T))) return st;
    knn_merge_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(n, part, 32 * ranges, k, out);
    DB200_CUDA(ctx, cudaGetLastError());
    count_launch(ctx);
    return DB200_OK;
  }
  // k > 8: one thread per query on the FP32 pipes
  const unsigned grid = (unsigned)((n + KNN_THREADS - 1) / KNN_THREADS);
  if (d <= 32)
    knn_kernel<32><<<grid, KNN_THREADS, 0, ctx->stream>>>(n, d, X, ldx, s, ref, k, out);
  else if (d <= 64)
    knn_kernel<64><<<grid, KNN_THREADS, 0, ctx->stream>>>(n, d, X, ldx, s, ref, k, out);
  else
    knn_kernel<128><<<grid, KNN_THREADS, 0, ctx->stream>>>(n, d, X, ldx, s, ref, k, out);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

}  // namespace db200

using namespace db200;

extern "C" {

int db200_knn_distance(db200_context* ctx, int n, int d, const float* X, int ldx, int s, const int* ref_idx, int k,
                       float* out) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 0 || d < 1 || d > 128 || ldx < d || s < 1 || k < 1 || k > KNN_KMAX || k > s || !X || !ref_idx || !out)
    return fail(ctx, DB200_ERR_INVALID, "knn_distance: bad arguments (d <= 128, 1 <= k <= min(16, s))");
  if (n == 0) return DB200_OK;
  return knn_distance(ctx, n, d, X, ldx, s, ref_idx, k, out);
}

int db200_leverage_features(db200_context* ctx, int n, int d, const float* X, int ldx, const float* knn, float* F) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 0 || d < 1 || ldx < d || !X || !knn || !F) return fail(ctx, DB200_ERR_INVALID, "leverage_features: bad arguments");
  if (n == 0) return DB200_OK;
  features_kernel<<<blocks_for((long long)n * 32, 256, 65535LL * 8), 256, 0, ctx->stream>>>(n, d, X, ldx, knn, F);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int db200_ridge_leverage(db200_context* ctx, int n, int r, const double* Z, int ldz, double lambda, double* lev) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 1 || r < 1 || ldz < n || !Z || !lev || !(lambda > 0)) return fail(ctx, DB200_ERR_INVALID, "ridge_leverage: bad arguments");
  const size_t rr = (size_t)r * r;
  const size_t bytes = 1024 + 4 * align_up(rr * 8, 256) + align_up((size_t)n * r * 8, 256);
  char* base = static_cast<char*>(slot_buffer(ctx, SLOT_SPARE, bytes));
  if (!base) return DB200_ERR_NOMEM;
  Carve cv{base};
  int* d_pair = cv.take<int>(4);
  double* G = cv.take<double>(rr);
  double* Xi = cv.take<double>(rr);
  double* X0 = cv.take<double>(rr);
  double* D = cv.take<double>(rr);
  double* W = cv.take<double>((size_t)n * r);
  // (Z^T Z + lambda I) = R^T R;  lev_i = ||z_i^T R^-1||^2
  int st = gram<double, double>(ctx, n, r, r, Z, ldz, Z, ldz, nullptr, 1.0, 0.0, G, r, true);
  if (!st) st = mirror_upper(ctx, G, r, r);
  if (!st) st = symmetrize(ctx, G, r, r, lambda);
  if (st) return st;
  DB200_CUDA(ctx, cudaMemsetAsync(d_pair, 0, 2 * sizeof(int), ctx->stream));
  if ((st = potrf_upper(ctx, G, r, r, d_pair, d_pair + 1))) return st;
  int hs[2] = {0, 0};
  DB200_CUDA(ctx, cudaMemcpyAsync(hs, d_pair, 2 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (hs[0]) return fail(ctx, DB200_ERR_NOT_SPD, "ridge_leverage: Z^T Z + lambda I not positive definite");
  if ((st = trinv_upper(ctx, G, r, r, Xi, r, X0, D))) return st;
  if ((st = gemm_tall<double, double>(ctx, n, r, r, Z, ldz, Xi, r, false, 0.0, W, n, 1.0, kUpperB))) return st;
  row_sumsq64_kernel<<<blocks_for(n, 256, 4096), 256, 0, ctx->stream>>>(n, r, W, n, lev);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return db200_synchronize(ctx);
}

// ------------------------------------------------------------------ MLP C ABI
int db200_mlp_create(db200_context* ctx, int in_dim, int width, int hidden, unsigned long long seed, db200_mlp** out) {
  if (!ctx || !out) return DB200_ERR_INVALID;
  *out = nullptr;
  if (in_dim < 1 || width < 1 || hidden < 1 || hidden > 7 || in_dim > 4096 || width > 4096)
    return fail(ctx, DB200_ERR_INVALID, "mlp_create: 1 <= hidden <= 7, dims <= 4096");
  db200_mlp* net = new db200_mlp();
  net->in = in_dim;
  net->width = width;
  net->hidden = hidden;
  net->layers = hidden + 1;
  net->device = ctx->device;
  int off = 0;
  for (int l = 0; l < net->layers; ++l) {
    const int fi = (l == 0) ? in_dim : width, fo = (l == hidden) ? 1 : width;
    net->fan_in.push_back(fi);
    net->fan_out.push_back(fo);
    net->off_w.push_back(off);
    off += fi * fo;
    net->off_b.push_back(off);
    off += fo;
  }
  net->nparams = off;
  // He-uniform weights, zero biases (host RNG, seeded)
  std::vector<float> w(off, 0.f);
  std::mt19937_64 g(seed);
  for (int l = 0; l < net->layers; ++l) {
    const float lim = std::sqrt(6.0f / (float)net->fan_in[l]) * (l == hidden ? 0.5f : 1.0f);
    std::uniform_real_distribution<float> u(-lim, lim);
    for (int e = 0; e < net->fan_in[l] * net->fan_out[l]; ++e) w[net->off_w[l] + e] = u(g);
  }
  std::vector<float> mean(in_dim, 0.f), scale(in_dim, 1.f);
  cudaError_t e = cudaSuccess;
  auto alloc = [&](void** p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b);
  };
  alloc((void**)&net->master, sizeof(float) * off);
  alloc((void**)&net->grad, sizeof(float) * off);
  alloc((void**)&net->mom1, sizeof(float) * off);
  alloc((void**)&net->mom2, sizeof(float) * off);
  alloc((void**)&net->wbf, sizeof(__nv_bfloat16) * off);
  alloc((void**)&net->in_mean, sizeof(float) * in_dim);
  alloc((void**)&net->in_scale, sizeof(float) * in_dim);
  alloc((void**)&net->d_loss, sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(net->master, w.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(net->mom1, 0, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMemset(net->mom2, 0, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMemcpy(net->in_mean, mean.data(), sizeof(float) * in_dim, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(net->in_scale, scale.data(), sizeof(float) * in_dim, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    db200_mlp_destroy(net);
    return cuda_fail(ctx, e, "mlp_create");
  }
  to_bf16_kernel<<<blocks_for(off, 256, 4096), 256, 0, ctx->stream>>>(off, net->master, net->wbf);
  count_launch(ctx);
  DB200_CUDA(ctx, cudaGetLastError());
  *out = net;
  return db200_synchronize(ctx);
}

void db200_mlp_destroy(db200_mlp* net) {
  if (!net) return;
  cudaSetDevice(net->device);
  cudaDeviceSynchronize();
  for (void* p : {(void*)net->master, (void*)net->grad, (void*)net->mom1, (void*)net->mom2, (void*)net->wbf,
                  (void*)net->in_mean, (void*)net->in_scale, (void*)net->d_loss, net->act})
    if (p) cudaFree(p);
  delete net;
}

int db200_mlp_param_count(const db200_mlp* net) { return net ? net->nparams : 0; }

int db200_mlp_get_params(db200_context* ctx, const db200_mlp* net, float* host) {
  if (!ctx || !net || !host) return DB200_ERR_INVALID;
  DB200_CUDA(ctx, cudaMemcpyAsync(host, net->master, sizeof(float) * net->nparams, cudaMemcpyDeviceToHost, ctx->stream));
  return db200_synchronize(ctx);
}

int db200_mlp_set_params(db200_context* ctx, db200_mlp* net, const float* host) {
  if (!ctx || !net || !host) return DB200_ERR_INVALID;
  DB200_CUDA(ctx, cudaMemcpyAsync(net->master, host, sizeof(float) * net->nparams, cudaMemcpyHostToDevice, ctx->stream));
  DB200_CUDA(ctx, cudaMemsetAsync(net->mom1, 0, sizeof(float) * net->nparams, ctx->stream));
  DB200_CUDA(ctx, cudaMemsetAsync(net->mom2, 0, sizeof(float) * net->nparams, ctx->stream));
  net->step = 0;
  to_bf16_kernel<<<blocks_for(net->nparams, 256, 4096), 256, 0, ctx->stream>>>(net->nparams, net->master, net->wbf);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return db200_synchronize(ctx);
}

int db200_mlp_set_input_scaling(db200_context* ctx, db200_mlp* net, const float* mean, const float* scale) {
  if (!ctx || !net || !mean || !scale) return DB200_ERR_INVALID;
  DB200_CUDA(ctx, cudaMemcpyAsync(net->in_mean, mean, sizeof(float) * net->in, cudaMemcpyHostToDevice, ctx->stream));
  DB200_CUDA(ctx, cudaMemcpyAsync(net->in_scale, scale, sizeof(float) * net->in, cudaMemcpyHostToDevice, ctx->stream));
  return db200_synchronize(ctx);
}

int db200_mlp_forward(db200_context* ctx, const db200_mlp* cnet, int m, const float* F, float* out) {
  if (!ctx || !cnet) return DB200_ERR_INVALID;
  if (m < 0 || !F || !out) return fail(ctx, DB200_ERR_INVALID, "mlp_forward: bad arguments");
  if (m == 0) return DB200_OK;
  db200_mlp* net = const_cast<db200_mlp*>(cnet);  // only the grow-only activation buffer changes
  // large m: in chunks so the activations stay bounded
  const int chunk = 1 << 18;
  for (int r0 = 0; r0 < m; r0 += chunk) {
    const int mb = std::min(chunk, m - r0);
    MlpActs A;
    int st = mlp_acts(ctx, net, mb, &A);
    if (!st) st = mlp_forward_impl(ctx, net, mb, F + (size_t)r0 * net->in, A);
    if (st) return st;
    DB200_CUDA(ctx, cudaMemcpyAsync(out + r0, A.out, sizeof(float) * mb, cudaMemcpyDeviceToDevice, ctx->stream));
  }
  return DB200_OK;
}

int db200_mlp_gradients(db200_context* ctx, db200_mlp* net, int m, const float* F, const float* target, float* loss,
                        float* grads) {
  if (!ctx || !net) return DB200_ERR_INVALID;
  if (m < 1 || !F || !target) return fail(ctx, DB200_ERR_INVALID, "mlp_gradients: bad arguments");
  MlpActs A;
  int st = mlp_acts(ctx, net, m, &A);
  if (!st) st = mlp_forward_impl(ctx, net, m, F, A);
  if (!st) st = mlp_backward_impl(ctx, net, m, target, A);
  if (st) return st;
  if (grads)
    DB200_CUDA(ctx, cudaMemcpyAsync(grads, net->grad, sizeof(float) * net->nparams, cudaMemcpyDeviceToDevice, ctx->stream));
  double l = 0;
  DB200_CUDA(ctx, cudaMemcpyAsync(&l, net->d_loss, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  st = db200_synchronize(ctx);
  if (loss) *loss = (float)l;
  return st;
}

int db200_mlp_adam_step(db200_context* ctx, db200_mlp* net, int m, const float* F, const float* target, float lr,
                        float* loss) {
  if (!ctx || !net) return DB200_ERR_INVALID;
  if (m < 1 || !F || !target || !(lr > 0)) return fail(ctx, DB200_ERR_INVALID, "mlp_adam_step: bad arguments");
  MlpActs A;
  int st = mlp_acts(ctx, net, m, &A);
  if (!st) st = mlp_forward_impl(ctx, net, m, F, A);
  if (!st) st = mlp_backward_impl(ctx, net, m, target, A);
  if (st) return st;
  net->step += 1;
  const float c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)net->step)));
  const float c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)net->step)));
  adam_kernel<<<blocks_for(net->nparams, 256, 4096), 256, 0, ctx->stream>>>(net->nparams, net->master, net->grad,
                                                                            net->mom1, net->mom2, net->wbf, lr, c1, c2);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  if (loss) {
    double l = 0;
    DB200_CUDA(ctx, cudaMemcpyAsync(&l, net->d_loss, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    st = db200_synchronize(ctx);
    *loss = (float)l;
    return st;
  }
  return DB200_OK;
}

// ------------------------------------------------------------------ selection
int db200_gumbel_keys(db200_context* ctx, int n, const float* logits, unsigned long long seed, float* keys) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 0 || !logits || !keys) return fail(ctx, DB200_ERR_INVALID, "gumbel_keys: bad arguments");
  if (n == 0) return DB200_OK;
  gumbel_kernel<<<blocks_for(n, 256, 8192), 256, 0, ctx->stream>>>(n, logits, seed, keys);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

int db200_select_topk(db200_context* ctx, int n, const float* keys, int k, int* idx) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 1 || k < 1 || k > n || !keys || !idx) return fail(ctx, DB200_ERR_INVALID, "select_topk: bad arguments");
  unsigned int* buf = static_cast<unsigned int*>(io_buffer(ctx, 4096));
  if (!buf) return DB200_ERR_NOMEM;
  unsigned int prefix = 0, mask = 0;
  int need = k;  // how many still to take at or below the current prefix
  std::vector<unsigned int> h(256);
  const unsigned grid = blocks_for(n, 256, 1024);
  for (int shift = 24; shift >= 0; shift -= 8) {
    DB200_CUDA(ctx, cudaMemsetAsync(buf, 0, 256 * sizeof(unsigned int), ctx->stream));
    radix_hist_kernel<<<grid, 256, 0, ctx->stream>>>(n, keys, prefix, mask, shift, buf);
    DB200_CUDA(ctx, cudaGetLastError());
    count_launch(ctx);
    DB200_CUDA(ctx, cudaMemcpyAsync(h.data(), buf, 256 * sizeof(unsigned int), cudaMemcpyDeviceToHost, ctx->stream));
    DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    // walk buckets from the top until `need` is covered
    int b = 255;
    for (; b > 0; --b) {
      if ((int)h[b] >= need) break;
      need -= (int)h[b];
    }
    prefix |= (unsigned int)b << shift;
    mask |= 0xFFu << shift;
  }
  // prefix is the k-th largest key; take every key above it and `need` of the keys equal to it
  DB200_CUDA(ctx, cudaMemsetAsync(buf, 0, 2 * sizeof(unsigned int), ctx->stream));
  radix_compact_kernel<<<grid, 256, 0, ctx->stream>>>(n, keys, prefix, need, buf, idx);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  // sorted indices make the landmark order (and so the factor) independent of atomic arrival order
  std::vector<int> hi(k);
  DB200_CUDA(ctx, cudaMemcpyAsync(hi.data(), idx, sizeof(int) * k, cudaMemcpyDeviceToHost, ctx->stream));
  DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::sort(hi.begin(), hi.end());
  DB200_CUDA(ctx, cudaMemcpyAsync(idx, hi.data(), sizeof(int) * k, cudaMemcpyHostToDevice, ctx->stream));
  return db200_synchronize(ctx);
}

// ------------------------------------------------------------------ landmark factor and residual
}  // extern "C"

// Nystrom factor on landmarks idx; TC = float: C from the tcgen05 tile engine (KBLOCK mode, fp32), TC = double: C
// from the FP64 kernel block (FP64 tensor-core Gram, FP64 exp), the comparator.
template <typename TC>
static int landmark_factor_impl(db200_context* ctx, int n, int d, const float* X, int ldx, const float* y,
                                float gamma, int r, const int* idx, double* Z, int ldz, double* nu_out) {
  const size_t rr = (size_t)r * r;
  const size_t bytes = 4096 + align_up((size_t)n * r * sizeof(TC), 256) + 4 * align_up(rr * 8, 256) +
                       align_up((size_t)r * d * 4, 256) + align_up((size_t)r * 4, 256);
  char* base = static_cast<char*>(slot_buffer(ctx, SLOT_PIPE, bytes));
  if (!base) return DB200_ERR_NOMEM;
  Carve cv{base};
  int* d_pair = cv.take<int>(4);
  double* d_scalar = cv.take<double>(4);
  TC* Cm = cv.take<TC>((size_t)n * r);
  double* W = cv.take<double>(rr);
  double* R = cv.take<double>(rr);
  double* Xinv = cv.take<double>(rr);
  double* D = cv.take<double>(rr);
  float* XL = cv.take<float>((size_t)r * d);
  float* yL = cv.take<float>(r);
  gather_rows_f32_kernel<<<blocks_for((long long)r * d, 256, 4096), 256, 0, ctx->stream>>>(X, ldx, idx, r, d, XL);
  gather_f32_kernel<<<blocks_for(r, 256, 1024), 256, 0, ctx->stream>>>(y, idx, r, yL);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, 2);
  // C = diag(y) K(:, L) diag(y_L)
  int st;
  if constexpr (sizeof(TC) == 4)
    st = db200_rbf_block(ctx, n, r, d, X, ldx, XL, d, DB200_POINT_MAJOR, y, yL, Cm, n, gamma);
  else
    st = db200_rbf_block_f64(ctx, n, r, d, X, ldx, XL, d, y, yL, Cm, n, (double)gamma);
  if (st) return st;
  gather_matrix_rows_kernel<TC><<<blocks_for((long long)rr, 256, 4096), 256, 0, ctx->stream>>>(Cm, n, idx, r, r, W);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  if ((st = symmetrize(ctx, W, r, r, 0.0))) return st;
  if ((st = trace(ctx, W, r, r, d_scalar))) return st;
  double tr = 0;
  DB200_CUDA(ctx, cudaMemcpyAsync(&tr, d_scalar, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double nu = 1e-7 * std::max(tr, 1e-300) / r;
  bool ok = false;
  for (int tries = 0; tries < 12 && !ok; ++tries) {
    DB200_CUDA(ctx, cudaMemcpyAsync(R, W, sizeof(double) * rr, cudaMemcpyDeviceToDevice, ctx->stream));
    if ((st = symmetrize(ctx, R, r, r, nu))) return st;
    DB200_CUDA(ctx, cudaMemsetAsync(d_pair, 0, 2 * sizeof(int), ctx->stream));
    if ((st = potrf_upper(ctx, R, r, r, d_pair, d_pair + 1))) return st;
    int hs[2] = {0, 0};
    DB200_CUDA(ctx, cudaMemcpyAsync(hs, d_pair, 2 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    DB200_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (hs[0] == 0) ok = true;
    else nu *= 10.0;
  }
  if (!ok) return fail(ctx, DB200_ERR_NOT_SPD, "landmark_factor: K(L, L) + nu I not positive definite after 12 shifts");
  // Z = C R^-1
  if ((st = trinv_upper(ctx, R, r, r, Xinv, r, W, D))) return st;
  if ((st = gemm_tall<TC, double>(ctx, n, r, r, Cm, n, Xinv, r, false, 0.0, Z, ldz, 1.0, kUpperB))) return st;
  if (nu_out) *nu_out = nu;
  return db200_synchronize(ctx);
}

extern "C" {

int db200_landmark_factor(db200_context* ctx, int n, int d, const float* X, int ldx, const float* y, float gamma, int r,
                          const int* idx, double* Z, int ldz, double* nu_out) {
  return db200_landmark_factor_ex(ctx, n, d, X, ldx, y, gamma, r, idx, Z, ldz, nu_out, DB200_MIXED);
}

int db200_landmark_factor_ex(db200_context* ctx, int n, int d, const float* X, int ldx, const float* y, float gamma,
                             int r, const int* idx, double* Z, int ldz, double* nu_out, int precision) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 1 || d < 1 || d > 128 || ldx < d || r < 1 || r > n || !X || !y || !idx || !Z || ldz < n ||
      (precision != DB200_MIXED && precision != DB200_FP64 && precision != DB200_MIXED_FAST))
    return fail(ctx, DB200_ERR_INVALID, "landmark_factor: bad arguments");
  return precision == DB200_FP64 ? landmark_factor_impl<double>(ctx, n, d, X, ldx, y, gamma, r, idx, Z, ldz, nu_out)
                                 : landmark_factor_impl<float>(ctx, n, d, X, ldx, y, gamma, r, idx, Z, ldz, nu_out);
}

int db200_residual_estimate(db200_context* ctx, int n, int d, const float* X, int ldx, const float* y, float gamma,
                            int r, const double* Z, int ldz, int s, const int* sample_idx, double* est) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 1 || d < 1 || d > 128 || ldx < d || r < 1 || s < 1 || s > n || !X || !y || !Z || ldz < n || !sample_idx ||
      !est)
    return fail(ctx, DB200_ERR_INVALID, "residual_estimate: bad arguments");
  const size_t bytes = 4096 + align_up((size_t)n * s * 4, 256) + align_up((size_t)n * s * 8, 256) +
                       align_up((size_t)s * r * 8, 256) + align_up((size_t)s * d * 4, 256) + align_up((size_t)s * 4, 256);
  char* base = static_cast<char*>(slot_buffer(ctx, SLOT_SPARE, bytes));
  if (!base) return DB200_ERR_NOMEM;
  Carve cv{base};
  double* sums = cv.take<double>(4);
  float* Ks = cv.take<float>((size_t)n * s);
  double* T = cv.take<double>((size_t)n * s);
  double* Zs = cv.take<double>((size_t)s * r);
  float* Xs = cv.take<float>((size_t)s * d);
  float* ys = cv.take<float>(s);
  gather_rows_f32_kernel<<<blocks_for((long long)s * d, 256, 4096), 256, 0, ctx->stream>>>(X, ldx, sample_idx, s, d, Xs);
  gather_f32_kernel<<<blocks_for(s, 256, 1024), 256, 0, ctx->stream>>>(y, sample_idx, s, ys);
  gather_matrix_rows_kernel<double><<<blocks_for((long long)s * r, 256, 4096), 256, 0, ctx->stream>>>(Z, ldz, sample_idx,
                                                                                                     s, r, Zs);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, 3);
  int st = db200_rbf_block(ctx, n, s, d, X, ldx, Xs, d, DB200_POINT_MAJOR, y, ys, Ks, n, gamma);
  if (st) return st;
  // T = Z Z(S, :)^T (n x s)
  if ((st = gemm_tall<double, double>(ctx, n, r, s, Z, ldz, Zs, s, true, 0.0, T, n))) return st;
  DB200_CUDA(ctx, cudaMemsetAsync(sums, 0, 2 * sizeof(double), ctx->stream));
  if ((st = sumsq_f32(ctx, Ks, n, n, s, sums))) return st;
  if ((st = axpby_f32(ctx, Ks, n, T, n, n, s, -1.0, 1.0))) return st;
  if ((st = sumsq_f32(ctx, Ks, n, n, s, sums + 1))) return st;
  double hs[2] = {0, 0};
  DB200_CUDA(ctx, cudaMemcpyAsync(hs, sums, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  st = db200_synchronize(ctx);
  if (st) return st;
  *est = (hs[0] > 0) ? std::sqrt(hs[1] / hs[0]) : 0.0;
  return DB200_OK;
}

// ------------------------------------------------------------------ the learned-landmark solve
// Landmark selection of the learned solve: k-NN features over sk reference points -> MLP log-leverage -> Gumbel
// keys -> top r.  Scratch F, knn, logits, keys, ref come from the caller's carve; idx receives r device indices.
static int select_landmarks_impl(db200_context* ctx, int n, int d, int r, const float* X, int ldx, const db200_mlp* net,
                                 unsigned long long seed, int sk, float* F, float* knn, float* logits, float* keys,
                                 int* ref, int* idx, db200_landmark_report* L) {
  const std::vector<int> h_ref = sample_indices(n, sk, seed ^ 0x6b6e6eull);
  DB200_CUDA(ctx, cudaMemcpyAsync(ref, h_ref.data(), sizeof(int) * sk, cudaMemcpyHostToDevice, ctx->stream));
  int st;
  {
    LandTimer t(ctx->stream);
    if ((st = knn_distance(ctx, n, d, X, ldx, sk, ref, 8, knn))) return st;
    if ((st = db200_leverage_features(ctx, n, d, X, ldx, knn, F))) return st;
    L->ms_features = t.stop();
  }
  {
    LandTimer t(ctx->stream);
    if ((st = db200_mlp_forward(ctx, net, n, F, logits))) return st;
    L->ms_predict = t.stop();
  }
  {
    LandTimer t(ctx->stream);
    if ((st = db200_gumbel_keys(ctx, n, logits, seed, keys))) return st;
    if ((st = db200_select_topk(ctx, n, keys, r, idx))) return st;
    L->ms_select = t.stop();
  }
  return DB200_OK;
}

int db200_select_landmarks(db200_context* ctx, int n, int d, int r, const float* X, int ldx, const db200_mlp* net,
                           unsigned long long seed, int s_knn, int* idx) {
  if (!ctx) return DB200_ERR_INVALID;
  if (n < 2 || d < 1 || d > 128 || ldx < d || r < 1 || r > n || !X || !net || net->in != d + 2 || s_knn < 9 || !idx)
    return fail(ctx, DB200_ERR_INVALID, "select_landmarks: bad arguments (model input must be d + 2)");
  const int sk = std::min(s_knn, n);
  const size_t bytes = 4096 + align_up((size_t)n * (d + 2) * 4, 256) + 3 * align_up((size_t)n * 4, 256) +
                       align_up((size_t)sk * 4, 256);
  char* base = static_cast<char*>(slot_buffer(ctx, SLOT_LAND, bytes));
  if (!base) return DB200_ERR_NOMEM;
  Carve cv{base};
  float* F = cv.take<float>((size_t)n * (d + 2));
  float* knn = cv.take<float>(n);
  float* logits = cv.take<float>(n);
  float* keys = cv.take<float>(n);
  int* ref = cv.take<int>(sk);
  db200_landmark_report L;
  std::memset(&L, 0, sizeof(L));
  int st = select_landmarks_impl(ctx, n, d, r, X, ldx, net, seed, sk, F, knn, logits, keys, ref, idx, &L);
  if (st) return st;
  return db200_synchronize(ctx);
}

int db200_svm_solve_landmarks(db200_context* ctx, int n, int d, int r, const float* X, int ldx, const float* y,
                              float gamma, double C, const db200_mlp* net, unsigned long long seed, int s_knn,
                              int s_res, double tol, const float* Omega, int ldo, int l_fb, int q,
                              const db200_barrier_params* params, double* a, double* Z, int ldz, db200_svm_report* rep,
                              db200_landmark_report* lrep) {
  if (!ctx) return DB200_ERR_INVALID;
  if (sharded(ctx))
    return fail(ctx, DB200_ERR_UNSUPPORTED, "svm_solve_landmarks: not row-sharded (detach the collective first)");
  if (n < 2 || d < 1 || d > 128 || ldx < d || r < 1 || r > n || !X || !y || !net || net->in != d + 2 || s_knn < 9 ||
      s_res < 1 || !a || !Z || ldz < n || (Omega && (ldo < n || l_fb < 1 || l_fb > n)) || q < 0)
    return fail(ctx, DB200_ERR_INVALID, "svm_solve_landmarks: bad arguments (model input must be d + 2)");
  db200_landmark_report L;
  std::memset(&L, 0, sizeof(L));
  db200_svm_report R;
  std::memset(&R, 0, sizeof(R));
  LandTimer total(ctx->stream);
  const int sk = std::min(s_knn, n), sr = std::min(s_res, n);
  const size_t bytes = 4096 + align_up((size_t)n * (d + 2) * 4, 256) + 3 * align_up((size_t)n * 4, 256) +
                       align_up((size_t)r * 4, 256) + align_up((size_t)sk * 4, 256) + align_up((size_t)sr * 4, 256);
  char* base = static_cast<char*>(slot_buffer(ctx, SLOT_LAND, bytes));
  if (!base) return DB200_ERR_NOMEM;
  Carve cv{base};
  float* F = cv.take<float>((size_t)n * (d + 2));
  float* knn = cv.take<float>(n);
  float* logits = cv.take<float>(n);
  float* keys = cv.take<float>(n);
  int* idx = cv.take<int>(r);
  int* ref = cv.take<int>(sk);
  int* res = cv.take<int>(sr);
  const std::vector<int> h_res = sample_indices(n, sr, seed ^ 0x726573ull);
  DB200_CUDA(ctx, cudaMemcpyAsync(res, h_res.data(), sizeof(int) * sr, cudaMemcpyHostToDevice, ctx->stream));
  int st = select_landmarks_impl(ctx, n, d, r, X, ldx, net, seed, sk, F, knn, logits, keys, ref, idx, &L);
  if (st) return st;
  {
    LandTimer t(ctx->stream);
    double nu = 0;
    // The landmark columns C = K(:, L) cost n r d, a fraction r / n of one Gaussian kernel pass: the parity-grade
    // mixed form (and the FP64 one) takes them in FP64, whose factor then matches the FP64 Nystrom factor on the
    // same landmarks to round-off; the fast mixed form takes the tile engine's fp32 block (~1e-6 from FP64 in f).
    db200_barrier_params Pf;
    if (params) Pf = *params;
    else db200_barrier_defaults(&Pf);
    const int cprec = (Pf.precision == DB200_MIXED_FAST) ? DB200_MIXED_FAST : DB200_FP64;
    if ((st = db200_landmark_factor_ex(ctx, n, d, X, ldx, y, gamma, r, idx, Z, ldz, &nu, cprec))) return st;
    R.nu = nu;
    L.ms_factor = t.stop();
  }
  {
    LandTimer t(ctx->stream);
    if ((st = db200_residual_estimate(ctx, n, d, X, ldx, y, gamma, r, Z, ldz, sr, res, &L.residual_est))) return st;
    L.ms_residual = t.stop();
  }
  int rank = r;
  if (!(L.residual_est <= tol) && Omega) {
    // fall back to the Gaussian sketch
    LandTimer t(ctx->stream);
    L.used_fallback = 1;
    db200_barrier_params P;
    if (params) P = *params;
    else db200_barrier_defaults(&P);
    if ((st = db200_lowrank(ctx, n, d, l_fb, q, X, ldx, y, Omega, ldo, gamma, P.precision, Z, ldz, &R))) return st;
    rank = l_fb;
    if ((st = db200_residual_estimate(ctx, n, d, X, ldx, y, gamma, rank, Z, ldz, sr, res, &L.residual_fallback)))
      return st;
    L.ms_fallback = t.stop();
  }
  L.rank = rank;
  const double nu_keep = R.nu;
  st = db200_svm_barrier(ctx, n, rank, Z, ldz, y, C, params, a, &R);
  if (st && st != DB200_ERR_MAXITER) return st;
  if (!L.used_fallback) R.nu = nu_keep;
  R.ms_total = total.stop();
  if (rep) *rep = R;
  if (lrep) *lrep = L;
  return st;
}

}  // extern "C"
