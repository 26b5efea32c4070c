// FP64 matrix products on the FP64 tensor cores (mma.sync.m16n8k8.f64): one pipelined kernel for the tall-skinny
// Gram, the tall GEMM, the block products of the triangular inverse and the FP64 kernel block.
//
//   C(m x q) = alpha * op(A) op(B) + ...,  reduction over p; op(A)(i, k) and op(B)(k, j) each stored with k contiguous
//   (AK / BK: element (i, k) at A[i * lda + k], (k, j) at B[j * ldb + k]) or with i / j contiguous (A[k * lda + i],
//   B[k * ldb + j]).
//
// What bounds it: the FP64 tensor pipe (64 FMA per cycle and SM; 37 TFLOP/s measured with 4 or more warps per SM).
// A CTA of 8 warps owns 128 x 8 NT of C, each warp a strip of 16 rows x 8 NT columns (NT <= 11: 88 accumulator
// registers, so two CTAs share an SM and one computes while the other waits at its barrier or stores).  Stages of 32
// k are copied by cp.async (16-byte pieces, or single elements when a base or leading dimension is not 16-byte
// aligned; out-of-range parts are zero-filled by the copy), two of them: a stage's products outlast its copy's
// latency many times over.  A k-contiguous operand is kept as four panels [column][8 k], so that a fragment is one
// conflict-free 16-byte load of k = 2t, 2t + 1 (lane t of its group; the pairing of k inside the instruction is free
// as long as both operands agree); the other form is kept [k][row], rows padded so that the same fragment is two
// conflict-free loads.
//
// The width 8 NT is chosen per launch so that q is covered with little padding (128-wide tiles pad q = 528 to 640) and
// its triangles are followed closely: strips outside C, and with `upper` strips below the diagonal, issue nothing, and
// with `tri` the zero part of a triangular op(B) is not visited.  Measured on a B200: Gram of 131072 x 528 (upper)
// 1.47 ms, tall product with a triangular 528 x 528 factor 1.45 ms, with a 1024 x 1024 one 4.7 ms; the kernels before
// (128 x 128 tiles, one CTA per SM, the triangle's zeros multiplied) took 2.18, 3.5 and 10.8 ms.  What is left to the
// pipe's rate: the strips that the triangles leave idle beside busy ones, and each CTA's first copy and last stores.
#pragma once
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "internal.h"
#include "la64.h"

namespace db200 {

constexpr int DMM_THREADS = 256;
constexpr int DMM_BM = 128;     // rows of C per CTA (8 warps x 16)
constexpr int DMM_KS = 32;      // k per stage
constexpr int DMM_STAGES = 2;
static_assert(DMM_BM % DMM_KS == 0, "tri_a starts a tile's reduction at its first row");

enum DmmEpi { DMM_STORE = 0, DMM_ADD = 1, DMM_ATOMIC = 2, DMM_RBF = 3, DMM_FROM = 4 };

struct DmmArgs {
  int m = 0, q = 0, p = 0;
  const void* A = nullptr;
  long long lda = 0;
  const void* B = nullptr;
  long long ldb = 0;
  const double* w = nullptr;  // weights of the reduction index (null: ones)
  double alpha = 1.0, beta = 0.0;
  void* C = nullptr;
  long long ldc = 0;
  int nq = 1;                 // column tiles (blockIdx.x = row tile * nq + column tile, last column tile first)
  int kps = 0;                // reduction length of one split (grid.y), a multiple of DMM_KS
  int upper = 0;              // only C(i, j) with i <= j
  int tri = kFullB;            // kUpperB: op(B)(k, j) = 0 for k > j; kLowerB: for k < j
  int tri_a = 0;               // op(A)(i, k) = 0 for k < i
  int epi = DMM_STORE;
  // batches along grid.z (the block pairs of a triangular inverse of order bl, halves of bs): the z-th pair's second
  // half has min(bs, bl - (2 z + 1) bs) rows, which replaces m and p (vary = 1) or q (vary = 2)
  long long sA = 0, sB = 0, sC = 0;
  int vary = 0, bl = 0, bs = 0;
  // DMM_FROM: C = S + alpha op(A) op(B), S FP64 (null: the identity)
  const double* S = nullptr;
  long long lds = 0;
  // DMM_RBF: C(i, j) = yi_i yj_j exp(-gamma max(si_i + sj_j - 2 G, 0))
  const double* si = nullptr;
  const double* sj = nullptr;
  const float* yi = nullptr;
  const float* yj = nullptr;
  double gamma = 0.0;
};

__device__ __forceinline__ void dmm_mma(double* d, const double* a, const double* b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// cp.async of SIZE bytes (4, 8 or 16) of which the first `bytes` are read and the rest zero-filled
template <int SIZE>
__device__ __forceinline__ void dmm_cp(void* smem, const void* gmem, int bytes) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  if constexpr (SIZE == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(SIZE), "r"(bytes)
                 : "memory");
}

// One operand's stage: NC columns (rows of op(A), columns of op(B)) x DMM_KS k.
template <typename T, bool KC, int NC, bool VEC>
struct DmmTile {
  static constexpr int LD = KC ? 8 : NC + 4;  // k-contiguous: panels [NC][8]; else [DMM_KS][NC + 4]
  static constexpr int ELEMS = KC ? DMM_KS * NC : DMM_KS * LD;
  static constexpr int E = VEC ? 16 / (int)sizeof(T) : 1;  // elements per copy

  // columns c0 .. c0 + NC - 1 (those below cl exist), k from kb (those below ke exist)
  static __device__ __forceinline__ void load(T* s, const T* X, long long ld, int c0, int cl, int kb, int ke) {
    constexpr int PER = (KC ? DMM_KS : NC) / E, TOTAL = NC * DMM_KS / E;
    if constexpr (VEC && DMM_THREADS % PER == 0) {
      // whole stages: a thread's copies are one address and a fixed step apart (the general form's bounds and index
      // arithmetic took an eighth of the Gram's time)
      if (c0 + NC <= cl && kb + DMM_KS <= ke) {
        constexpr int STEP = DMM_THREADS / PER;
        const int a = threadIdx.x / PER, b = (threadIdx.x % PER) * E;
        const T* src = X + (KC ? (long long)(c0 + a) * ld + kb + b : (long long)(kb + a) * ld + c0 + b);
        T* dst = KC ? s + (b >> 3) * (NC * 8) + a * 8 + (b & 7) : s + a * LD + b;
#pragma unroll
        for (int u = 0; u < (TOTAL + DMM_THREADS - 1) / DMM_THREADS; ++u)
          if (TOTAL % DMM_THREADS == 0 || u * DMM_THREADS + (int)threadIdx.x < TOTAL)
            dmm_cp<16>(dst + u * STEP * (KC ? 8 : LD), src + u * STEP * ld, 16);
        return;
      }
    }
#pragma unroll
    for (int e0 = 0; e0 < TOTAL; e0 += DMM_THREADS) {
      const int e = e0 + threadIdx.x;
      if (TOTAL % DMM_THREADS != 0 && e >= TOTAL) break;
      const int a = e / PER, b = (e % PER) * E;
      const int c = KC ? a : b, kk = KC ? b : a;
      const int k = kb + kk;
      const int left = KC ? ke - k : cl - (c0 + c);  // elements left along the contiguous index
      const bool in = KC ? c0 + c < cl : k < ke;
      const int valid = (in && left > 0) ? (left < E ? left : E) : 0;
      const T* src = valid ? X + (KC ? (long long)(c0 + c) * ld + k : (long long)k * ld + c0 + c) : X;
      T* dst = KC ? s + (kk >> 3) * (NC * 8) + c * 8 + (kk & 7) : s + kk * LD + c;
      dmm_cp<VEC ? 16 : (int)sizeof(T)>(dst, src, valid * (int)sizeof(T));
    }
  }
  // entries k = 8 h + 2 t and + 1 of column c; SPLIT: k = 8 h + t and + 4 (k-contiguous only)
  template <bool SPLIT>
  static __device__ __forceinline__ void frag(const T* s, int c, int h, int t, double& v0, double& v1) {
    if constexpr (SPLIT) {
      static_assert(KC, "split fragments are read from k-contiguous panels");
      const T* q = s + h * (NC * 8) + c * 8 + t;
      v0 = (double)q[0];
      v1 = (double)q[4];
      return;
    }
    if constexpr (KC) {
      const T* q = s + h * (NC * 8) + c * 8 + 2 * t;
      if constexpr (sizeof(T) == 8) {
        const double2 v = *reinterpret_cast<const double2*>(q);
        v0 = v.x;
        v1 = v.y;
      } else {
        const float2 v = *reinterpret_cast<const float2*>(q);
        v0 = (double)v.x;
        v1 = (double)v.y;
      }
    } else {
      const T* q = s + (8 * h + 2 * t) * LD + c;
      v0 = (double)q[0];
      v1 = (double)q[LD];
    }
  }
};

template <typename TA, typename TB, bool AK, bool BK, int NT, bool VEC>
constexpr size_t dmm_smem() {
  const size_t a = (size_t)DmmTile<TA, AK, DMM_BM, VEC>::ELEMS * sizeof(TA);
  const size_t b = (size_t)DmmTile<TB, BK, 8 * NT, VEC>::ELEMS * sizeof(TB);
  return DMM_STAGES * (((a + 15) / 16 + (b + 15) / 16) * 16);
}

template <typename TA, typename TB, typename TC, bool AK, bool BK, int NT, bool VEC>
__global__ void __launch_bounds__(DMM_THREADS, 2) dmm_kernel(const DmmArgs g) {
  constexpr int BN = 8 * NT;
  // float operands (the kernel block's points): k in the instruction's own order, so that a cross term rounds as a
  // sequential product does (the distance cancels its leading digits)
  constexpr bool SPLIT = sizeof(TA) == 4 && sizeof(TB) == 4;
  using TileA = DmmTile<TA, AK, DMM_BM, VEC>;
  using TileB = DmmTile<TB, BK, BN, VEC>;
  constexpr size_t A_BYTES = (TileA::ELEMS * sizeof(TA) + 15) / 16 * 16;
  constexpr size_t STAGE = A_BYTES + (TileB::ELEMS * sizeof(TB) + 15) / 16 * 16;
  extern __shared__ __align__(16) unsigned char dsm[];

  int m = g.m, q = g.q, p = g.p;
  if (g.vary) {
    const int half = min(g.bs, g.bl - (2 * (int)blockIdx.z + 1) * g.bs);
    if (g.vary == 1) m = p = half;
    else q = half;
  }
  const int it = blockIdx.x / g.nq, jt = g.nq - 1 - (int)blockIdx.x % g.nq;
  const int i0 = it * DMM_BM, j0 = jt * BN;
  if (i0 >= m || j0 >= q || (g.upper && i0 > j0 + BN - 1)) return;
  const TA* A = static_cast<const TA*>(g.A) + blockIdx.z * g.sA;
  const TB* B = static_cast<const TB*>(g.B) + blockIdx.z * g.sB;
  TC* C = static_cast<TC*>(g.C) + blockIdx.z * g.sC;
  int kb = blockIdx.y * g.kps, ke = min(p, kb + g.kps);
  if (g.tri == kUpperB) ke = min(ke, j0 + BN);
  if (g.tri == kLowerB) kb = max(kb, j0 / DMM_KS * DMM_KS);
  if (g.tri_a) kb = max(kb, i0);
  const int nst = ke > kb ? (ke - kb + DMM_KS - 1) / DMM_KS : 0;

  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int fr = lane / 4, fk = lane % 4;
  // This warp's strip: turned by the tile and split, since the strips that `upper` or the end of C leave idle are always
  // the same of a tile, and warps 0, 4 / 1, 5 / ... share an SM sub-partition's tensor pipe.
  const int strip = (warp + blockIdx.x + blockIdx.y) % 8;
  const int ir = i0 + 16 * strip;
  const bool active = ir < m && !(g.upper && ir > j0 + BN - 1);

  auto issue = [&](int st) {
    unsigned char* s = dsm + (size_t)(st % DMM_STAGES) * STAGE;
    const int k = kb + st * DMM_KS;
    TileA::load(reinterpret_cast<TA*>(s), A, g.lda, i0, m, k, ke);
    TileB::load(reinterpret_cast<TB*>(s + A_BYTES), B, g.ldb, j0, q, k, ke);
  };
  double acc[NT][4];
#pragma unroll
  for (int b = 0; b < NT; ++b)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[b][e] = 0.0;
#pragma unroll
  for (int st = 0; st < DMM_STAGES - 1; ++st) {
    if (st < nst) issue(st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int st = 0; st < nst; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DMM_STAGES - 2) : "memory");
    __syncthreads();  // stage st is visible to all; every read of stage st - 1, whose buffer is refilled now, is done
    if (st + DMM_STAGES - 1 < nst) issue(st + DMM_STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (!active) continue;
    const unsigned char* s = dsm + (size_t)(st % DMM_STAGES) * STAGE;
    const TA* sA = reinterpret_cast<const TA*>(s);
    const TB* sB = reinterpret_cast<const TB*>(s + A_BYTES);
#pragma unroll
    for (int h = 0; h < DMM_KS / 8; ++h) {
      double af[4];
      TileA::template frag<SPLIT>(sA, 16 * strip + fr, h, fk, af[0], af[2]);
      TileA::template frag<SPLIT>(sA, 16 * strip + fr + 8, h, fk, af[1], af[3]);
      if (g.w) {
        const int k = kb + st * DMM_KS + 8 * h + (SPLIT ? fk : 2 * fk), k1 = k + (SPLIT ? 4 : 1);
        const double w0 = k < ke ? __ldg(g.w + k) : 0.0, w1 = k1 < ke ? __ldg(g.w + k1) : 0.0;
        af[0] *= w0;
        af[1] *= w0;
        af[2] *= w1;
        af[3] *= w1;
      }
#pragma unroll
      for (int b = 0; b < NT; ++b) {
        double bf[2];
        TileB::template frag<SPLIT>(sB, 8 * b + fr, h, fk, bf[0], bf[1]);
        dmm_mma(acc[b], af, bf);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!active) return;
  // acc[b][0, 1]: row ir + fr, columns j0 + 8 b + 2 fk + 0, 1; acc[b][2, 3]: row + 8
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = ir + fr + 8 * h;
    if (i >= m) continue;
    double si = 0.0, yi = 1.0;
    if (g.epi == DMM_RBF) {
      si = g.si[i];
      yi = g.yi ? (double)g.yi[i] : 1.0;
    }
#pragma unroll
    for (int b = 0; b < NT; ++b) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = j0 + 8 * b + 2 * fk + e;
        if (j >= q || (g.upper && i > j)) continue;
        TC* dst = C + (long long)j * g.ldc + i;
        const double v = acc[b][2 * h + e];
        if (g.epi == DMM_RBF) {
          double x = exp(-g.gamma * fmax(si + g.sj[j] - 2.0 * v, 0.0)) * yi;
          if (g.yj) x *= (double)g.yj[j];
          *dst = (TC)x;
        } else if (g.epi == DMM_ATOMIC) {
          if constexpr (sizeof(TC) == 8) atomicAdd(dst, (TC)(g.alpha * v));
        } else if (g.epi == DMM_ADD) {
          *dst = (TC)((double)*dst + g.alpha * v);
        } else if (g.epi == DMM_FROM) {
          const double s = g.S ? g.S[(long long)j * g.lds + i] : (i == j ? 1.0 : 0.0);
          *dst = (TC)(s + g.alpha * v);
        } else {
          double x = g.alpha * v;
          if (g.beta != 0.0) x += g.beta * (double)*dst;
          *dst = (TC)x;
        }
      }
    }
  }
}

template <typename TA, typename TB, typename TC, bool AK, bool BK, int NT, bool VEC>
int dmm_launch_one(db200_context* ctx, const DmmArgs& g, dim3 grid) {
  constexpr size_t smem = dmm_smem<TA, TB, AK, BK, NT, VEC>();
  auto k = dmm_kernel<TA, TB, TC, AK, BK, NT, VEC>;
  DB200_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<grid, DMM_THREADS, smem, ctx->stream>>>(g);
  DB200_CUDA(ctx, cudaGetLastError());
  count_launch(ctx);
  return DB200_OK;
}

// Column-tile widths (in units of 8 columns): all of them for aligned FP64 operands, the path of every factor;
// three of them for the rest.
constexpr int DMM_NT[] = {4, 6, 8, 9, 11};
template <typename TA, typename TB, bool VEC>
constexpr bool dmm_offers(int nt) {
  return (VEC && sizeof(TA) == 8 && sizeof(TB) == 8) || nt == 4 || nt == 8 || nt == 11;
}

// Work of one launch with tiles of 8 nt columns: columns issued per strip of 16 rows, 8 more per tile and strip for
// the copies, A fragments and barriers, strips and k outside the triangles left out.  Measured at 131072 x 528 x 528:
// triangular product 1.45, 1.63 and 1.58 ms with tiles of 48, 64 and 88 columns, upper Gram 1.47, 1.61 and 1.57 ms.
inline double dmm_cost(int m, int q, int p, int nt, bool upper, int tri) {
  const int bn = 8 * nt;
  double cost = 0.0;
  for (int j0 = 0; j0 < q; j0 += bn) {
    const double rows = upper ? std::min(m, (j0 + bn + 15) / 16 * 16) : m;
    const double k = tri == kUpperB ? std::min(p, j0 + bn) : tri == kLowerB ? std::max(0, p - j0) : p;
    cost += rows * k * (bn + 8);
  }
  return cost;
}

template <typename TA, typename TB, typename TC, bool AK, bool BK, bool VEC>
int dmm_dispatch(db200_context* ctx, DmmArgs g, int splits, int batch) {
  const int mt = (g.m + DMM_BM - 1) / DMM_BM;
  int nt = 0;
  double best = 0.0;
  for (int c : DMM_NT) {
    if (!dmm_offers<TA, TB, VEC>(c)) continue;
    const long long ctas = (long long)mt * ((g.q + 8 * c - 1) / (8 * c)) * splits * batch;
    // with fewer CTAs than two per SM the time is that of one tile, whose width counts
    const double fill = std::max(1.0, 2.0 * ctx->num_sms / (double)ctas);
    const double cost = dmm_cost(g.m, g.q, g.p, c, g.upper != 0, g.tri) * fill;
    if (nt == 0 || cost < best) {
      best = cost;
      nt = c;
    }
  }
  g.nq = (g.q + 8 * nt - 1) / (8 * nt);
  if (g.kps <= 0) g.kps = round_up(std::max(g.p, 1), DMM_KS);
  if ((long long)mt * g.nq > 0x7fffffffLL || splits > 65535 || batch > 65535)
    return fail(ctx, DB200_ERR_UNSUPPORTED, "FP64 product: too many tiles");
  const dim3 grid((unsigned)(mt * g.nq), (unsigned)splits, (unsigned)batch);
  if constexpr (dmm_offers<TA, TB, VEC>(6))
    if (nt == 6) return dmm_launch_one<TA, TB, TC, AK, BK, 6, VEC>(ctx, g, grid);
  if constexpr (dmm_offers<TA, TB, VEC>(9))
    if (nt == 9) return dmm_launch_one<TA, TB, TC, AK, BK, 9, VEC>(ctx, g, grid);
  if (nt == 4) return dmm_launch_one<TA, TB, TC, AK, BK, 4, VEC>(ctx, g, grid);
  if (nt == 8) return dmm_launch_one<TA, TB, TC, AK, BK, 8, VEC>(ctx, g, grid);
  return dmm_launch_one<TA, TB, TC, AK, BK, 11, VEC>(ctx, g, grid);
}

// Launch with the cheapest offered width.  `splits` (grid.y, with DMM_ATOMIC when above 1) cuts the reduction into
// g.kps-long parts; batch: grid.z.
template <typename TA, typename TB, typename TC, bool AK, bool BK>
int dmm_launch(db200_context* ctx, const DmmArgs& g, int splits = 1, int batch = 1) {
  const bool vec = reinterpret_cast<uintptr_t>(g.A) % 16 == 0 && reinterpret_cast<uintptr_t>(g.B) % 16 == 0 &&
                   g.lda * (long long)sizeof(TA) % 16 == 0 && g.ldb * (long long)sizeof(TB) % 16 == 0 &&
                   g.sA * (long long)sizeof(TA) % 16 == 0 && g.sB * (long long)sizeof(TB) % 16 == 0;
  return vec ? dmm_dispatch<TA, TB, TC, AK, BK, true>(ctx, g, splits, batch)
             : dmm_dispatch<TA, TB, TC, AK, BK, false>(ctx, g, splits, batch);
}

}  // namespace db200
