// Cholesky of a small SPD matrix in one launch on a thread-block cluster: the r x r capacity matrices of the
// barrier's Newton steps and the l x l Grams of CholeskyQR2 and the Nystrom core (l <= 544).
//
// The blocked right-looking algorithm of include/lapack_like.h:10-57 (potrf of the diagonal block, trsm of its
// block row, syrk of the trailing matrix) in 64-column steps on the nc CTAs of one cluster.  One step:
//   1. every CTA reads the 64 x 64 diagonal block and factors it itself (p64_run: the same inputs and instructions
//      give every CTA the same R11, so nothing is broadcast and a failing pivot stops every CTA at the same step),
//      its other four warps solving up to four of the block row's 16-column groups at the same time;
//   2. cluster barrier (the block row is complete, the diagonal block has been read); one CTA writes R11;
//   3. the trailing matrix is updated in 16 x 16 tiles, one warp each, fragments read straight from the block row
//      (k contiguous, so a fragment is a 16-byte load); cluster barrier.
// The matrix stays in L2 (2.2 MB at l = 528), which all CTAs reach at full rate: 52 us at l = 138, 219 us at l = 528 (and
// 3 and 10 us less since a short last block stops at its last 16 columns).
// The form that kept the triangle in the CTAs' shared memory (67 and 372 us) spent a quarter of its time on the
// all-to-all copy of the block row through distributed shared memory (~170 bytes per cycle for 13 CTAs), and the rest
// about equally on its one-warp 32-pivot chains, its substitution and its update over column-cyclic slots.
#include <algorithm>
#include <mutex>

#include "internal.h"
#include "la64.h"
#include "potrf64.cuh"
#include "ptx.cuh"

namespace db200 {

namespace {

constexpr int PC_MAX_L = 544;   // beyond, the launches of the blocked path spread over all SMs
constexpr int PC_MAX_NC = 16;
static_assert(4 * 8 * 16 >= PC_MAX_L - P64_NB, "the four solving warps of 8 CTAs cover the block row");

// C(i, j) -= sum_k R(k, i) R(k, j) for the 16 x 16 tile with rows i0.. and columns j0.. (entries i <= j < l), R's 64
// rows at P (column c at P + c * lda).
template <bool VEC>
__device__ __forceinline__ void pc_update_tile(const double* P, double* C, long long lda, int i0, int j0, int l) {
  const int lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
  double acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
  const int ja = min(j0 + g, l - 1), jb = min(j0 + g + 8, l - 1);  // columns past l repeat the last: not stored
  const int ia = min(i0 + g, l - 1), ib = min(i0 + g + 8, l - 1);
  const double* cja = P + ja * lda + 2 * t;
  const double* cjb = P + jb * lda + 2 * t;
  const double* cia = P + ia * lda + 2 * t;
  const double* cib = P + ib * lda + 2 * t;
  auto ld2 = [](const double* q) -> double2 {
    if (VEC) return __ldcg(reinterpret_cast<const double2*>(q));
    return make_double2(__ldcg(q), __ldcg(q + 1));
  };
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // 32 k at a time: 16 loads in flight
    double2 a0[4], a1[4], b0[4], b1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int o = 32 * h + 8 * k;
      a0[k] = ld2(cja + o);
      a1[k] = ld2(cjb + o);
      b0[k] = ld2(cia + o);
      b1[k] = ld2(cib + o);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double af[4] = {a0[k].x, a1[k].x, a0[k].y, a1[k].y};
      const double f0[2] = {b0[k].x, b0[k].y}, f1[2] = {b1[k].x, b1[k].y};
      p64_mma(acc[0], af, f0);
      p64_mma(acc[1], af, f1);
    }
  }
  // acc[n][0, 1]: column j0 + g, rows i0 + 8 n + 2 t + 0, 1; acc[n][2, 3]: column j0 + g + 8
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = j0 + g + 8 * (e >> 1), i = i0 + 8 * n + 2 * t + (e & 1);
      if (j < l && i <= j) {
        double* c = C + j * lda + i;
        *c = __ldcg(c) - acc[n][e];
      }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(P64_THREADS, 1) potrf_cluster_kernel(double* A, int lda, int l, int* status,
                                                                       int* bad, double* W) {
  extern __shared__ __align__(16) unsigned char raw[];
  P64Smem& S = *reinterpret_cast<P64Smem*>(raw);
  const int nc = (int)cluster_nctarank(), c = (int)cluster_ctarank();
  const int tid = threadIdx.x, warp = tid / 32;
  if (*(volatile int*)status) return;  // an earlier factorisation on this status word failed (same in every CTA)
  double acc[8][4];
  for (int c0 = 0, step = 0; c0 < l; c0 += P64_NB, ++step) {
    const int kb = min(P64_NB, l - c0), r0 = c0 + kb;
    const int ng = (l - r0 + 15) / 16;  // 16-column groups of the block row
    int group = warp, col = c0 + 16 * warp, cl = r0;
    if (warp >= 4) {
      const int gi = c + nc * (warp - 4);
      group = gi < ng ? 4 + gi : -1;
      col = r0 + 16 * gi;
      cl = l;
    }
    if (group >= 0) p64_load<VEC>(acc, A, lda, c0, kb, col, cl, warp < 4 ? warp : -1);
    if (!p64_run(S, acc, group, kb)) {
      if (c == 0 && tid == 0 && atomicCAS(status, 0, DB200_ERR_NOT_SPD) == 0) *bad = (c0 + S.fail - 1) / 32 * 32;
      return;
    }
    if (group >= 4) p64_store<VEC>(acc, A, lda, c0, kb, col, cl);
    cluster_sync_all();  // the block row is complete; every CTA has read the diagonal block
    if (step % nc == c) {
      if (W) p64_store_inverses(S, W + (long long)c0 * 16, kb);
      for (int e = tid; e < kb * P64_NB; e += P64_THREADS) {
        const int i = e % P64_NB, j = e / P64_NB;
        if (i <= j) A[(long long)(c0 + j) * lda + c0 + i] = S.R[j * P64_RLD + i];
      }
    }
    if (r0 >= l) break;
    // trailing tiles (I <= J), tile number J (J + 1) / 2 + I
    const int tiles = ng * (ng + 1) / 2;
    for (int e = c + nc * warp; e < tiles; e += nc * (P64_THREADS / 32)) {
      int J = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
      while (J * (J + 1) / 2 > e) --J;
      while ((J + 1) * (J + 2) / 2 <= e) ++J;
      const int I = e - J * (J + 1) / 2;
      pc_update_tile<VEC>(A + c0, A, lda, r0 + 16 * I, r0 + 16 * J, l);
    }
    cluster_sync_all();
  }
  for (int j = c + nc * warp; j < l; j += nc * (P64_THREADS / 32))
    for (int i = j + 1 + tid % 32; i < l; i += 32) A[(long long)j * lda + i] = 0.0;
}

cudaLaunchConfig_t pc_config(cudaLaunchAttribute* attr, int nc, cudaStream_t st) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nc);
  cfg.blockDim = dim3(P64_THREADS);
  cfg.dynamicSmemBytes = sizeof(P64Smem);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Largest cluster the device can hold (0: none), probed once per device.
int pc_nc_max(int device) {
  static std::mutex mu;
  static int cached[64];
  static bool done[64] = {};
  if (device < 0 || device >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (done[device]) return cached[device];
  int best = PC_MAX_NC;
  for (auto k : {potrf_cluster_kernel<true>, potrf_cluster_kernel<false>}) {
    int nc = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P64Smem)) == cudaSuccess) {
      const bool wide = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
      for (nc = wide ? PC_MAX_NC : 8; nc >= 1; --nc) {
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = pc_config(attr, nc, nullptr);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters >= 1) break;
      }
    }
    best = std::min(best, nc);
  }
  cudaGetLastError();
  cached[device] = best;
  done[device] = true;
  return best;
}

}  // namespace

void potrf_cluster_init(db200_context* ctx) { ctx->potrf_nc_max = pc_nc_max(ctx->device); }

// A CTA per 32 columns: the solving warps then cover the block row and a warp has at most four update tiles a step.
int potrf_cluster_size(const db200_context* ctx, int l) {
  if (l < 1 || l > PC_MAX_L) return 0;
  const int nc = std::min((l + 31) / 32, ctx->potrf_nc_max);
  return 64 * nc >= l - P64_NB ? nc : 0;
}

int potrf_cluster(db200_context* ctx, double* A, int lda, int l, int* d_status, int* d_bad, double* W) {
  const int nc = potrf_cluster_size(ctx, l);
  if (nc < 1) return DB200_ERR_UNSUPPORTED;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = pc_config(attr, nc, ctx->stream);
  const bool vec = reinterpret_cast<uintptr_t>(A) % 16 == 0 && lda % 2 == 0;
  DB200_CUDA(ctx, vec ? cudaLaunchKernelEx(&cfg, potrf_cluster_kernel<true>, A, lda, l, d_status, d_bad, W)
                      : cudaLaunchKernelEx(&cfg, potrf_cluster_kernel<false>, A, lda, l, d_status, d_bad, W));
  count_launch(ctx);
  return DB200_OK;
}

}  // namespace db200
