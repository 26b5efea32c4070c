// Cholesky of a diagonal block of up to 64 columns together with the solve of its block row, by the warps of one CTA
// (256 threads): the building block of the one-launch factor (potrf_cluster.cu) and of the blocked one (la64.cu).
//
// Every warp holds 16 columns x 64 rows as mma.sync.m16n8k8.f64 accumulators of the transposed tile (column g of the
// group, rows 8 b + 2 t and + 1 in d0, d1; column g + 8 in d2, d3), which are at once the A fragments of a product
// over those rows (the pairing k = 2t, 2t + 1 inside the instruction is free).  Warps 0..3 hold the block's own column
// groups, the others column groups of the block row.  In up to four steps p of 16 rows:
//   warp p factors its 16 x 16 diagonal block (factor16, whose elimination keeps the factor's backward error at a few u):
//     one warp, lane = column, with the 16 columns of the identity in the other half-warp, so it also leaves W = R_pp^-T;
//   every later group solves its rows p, X = W B, then X += W (B - R_pp^T X): the correction makes the solve as
//     backward stable as substitution, whose 16 dependent steps it replaces by three 16 x 16 products;
//   every later group subtracts R_pr^T X_p from its rows r > p.
// What bounds it is the chain of 64 pivots, taken two at a time (a shuffle, a reciprocal, the reduced row through shared
// memory and some products per pair): 23.6 k cycles for a full block with 64 columns of its block row, of which the four
// 16 x 16 factors take 16 k.  One 64-column step of the blocked factor takes 21.5 us; with a barrier, a division and a
// strip update per pivot, and the block row solved by 64 dependent shuffle steps, it took 38.8 us.  A block of fewer
// columns stops at its last 16.
#pragma once
#include <cstdint>

namespace db200 {

constexpr int P64_THREADS = 256;
constexpr int P64_NB = 64;     // columns per step
constexpr int P64_RLD = 72;    // leading dimension of the block, column major (= 8 mod 16: conflict-free fragments)
constexpr int P64_WLD = 24;    // of W, row major
constexpr int P64_DLD = 18;    // of the staged 16 x 16 block, column major

struct P64Smem {
  double R[P64_NB * P64_RLD];        // R(i, j) at j * P64_RLD + i, zeros below the diagonal of each 16 x 16 block
  double W[4][16 * P64_WLD];         // R_pp^-T(i, j) at i * P64_WLD + j
  double D[16 * P64_DLD];
  double row[4 * 16];
  double rs[16];
  int fail;                          // 1 + first column of the 16-column block whose pivot is not positive
  int flag;
};

__device__ __forceinline__ void p64_mma(double* d, const double* a, const double* b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// d += sign * (tile a as A fragment) * B, B's entries k = 2t, 2t + 1 of column g at bp (contiguous)
__device__ __forceinline__ void p64_mma_tile(double* d, const double* a, double sign, const double* bp) {
  const double af[4] = {sign * a[0], sign * a[2], sign * a[1], sign * a[3]};
  const double2 b = *reinterpret_cast<const double2*>(bp);
  const double bf[2] = {b.x, b.y};
  p64_mma(d, af, bf);
}

// Factor of the staged 16 x 16 block D (upper entries) by one warp: R into Rb (column major, ld P64_RLD, zeros below
// the diagonal), W = R^-T; returns false on a non-positive or NaN pivot (the same answer in every lane).  Rows are
// eliminated unscaled and divided by the square roots of their pivots at the end, two at a time: with the 2 x 2
// pivot [p q; q r], det = p r - q^2 and the second row reduced by the first, u = a_i+1 - (q / p) a_i, the rows below lose
// a_im a_i / p + u_m u (p / det), so that one reciprocal's latency (1 / p and 1 / det are independent) sits on the chain
// per two columns; the second pivot is det / p.  Applying [p q; q r]^-1 to the unreduced rows instead is shorter by a
// shared-memory round trip, but its errors grow by 1 / (1 - rho^2) for columns i, i + 1 of correlation rho, where
// eliminating one row at a time (and this form) leaves a few u |A| whatever the matrix.
// The block is first scaled symmetrically by powers of two to diagonal entries in [1, 4), exactly, so that det neither
// overflows nor underflows for any range of the entries, and R and W are scaled back at the end.
static __device__ __noinline__ bool p64_factor16(P64Smem& S, double* Rb, double* Wb) {
  const int lane = threadIdx.x % 32, j = lane & 15;
  const bool unit = lane >= 16;  // a column of the identity
  const int k2 = (((__double2hiint(S.D[j * P64_DLD + j]) >> 20) & 0x7ff) - 1023) >> 1;
  const double s = __hiloint2double((1023 - k2) << 20, 0), s_inv = __hiloint2double((1023 + k2) << 20, 0);
  if (!unit) S.rs[j] = s;
  __syncwarp();
  double a[16];
#pragma unroll
  for (int m = 0; m < 16; m += 2) {
    const double2 v = *reinterpret_cast<const double2*>(S.D + j * P64_DLD + m);
    const double2 sm = *reinterpret_cast<const double2*>(S.rs + m);
    a[m] = unit ? (m == j ? 1.0 : 0.0) : v.x * sm.x * s;
    a[m + 1] = unit ? (m + 1 == j ? 1.0 : 0.0) : v.y * sm.y * s;
  }
  double dg = 1.0;
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    double* rb = S.row + (i & 2) * 16;
    if (!unit) rb[j] = a[i];
    const double p = __shfl_sync(0xffffffffu, a[i], i), q = __shfl_sync(0xffffffffu, a[i], i + 1);
    const double r = __shfl_sync(0xffffffffu, a[i + 1], i + 1);
    const double det = fma(p, r, -q * q);
    const double ip = 1.0 / p, id = 1.0 / det;
    a[i + 1] = fma(-q * ip, a[i], a[i + 1]);
    if (!unit) rb[16 + j] = a[i + 1];
    const double y0 = a[i] * ip, y1 = a[i + 1] * (p * id), second = det * ip;
    ok = ok && p > 0.0 && second > 0.0;
    __syncwarp();
#pragma unroll
    for (int m = i + 2; m < 16; ++m) a[m] = fma(-rb[m], y0, fma(-rb[16 + m], y1, a[m]));
    if (lane == i) dg = p;
    if (lane == i + 1) dg = second;
  }
  if (!ok) return false;
  const double sq = sqrt(dg), back = unit ? s : s_inv;
  if (!unit) S.rs[j] = 1.0 / sq;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const double2 rs = *reinterpret_cast<const double2*>(S.rs + i);
    const double v0 = a[i] * rs.x * back, v1 = a[i + 1] * rs.y * back, d = sq * back;
    if (unit) {
      Wb[i * P64_WLD + j] = (i >= j) ? v0 : 0.0;
      Wb[(i + 1) * P64_WLD + j] = (i + 1 >= j) ? v1 : 0.0;
    } else {
      *reinterpret_cast<double2*>(Rb + j * P64_RLD + i) =
          make_double2(i < j ? v0 : (i == j ? d : 0.0), i + 1 < j ? v1 : (i + 1 == j ? d : 0.0));
    }
  }
  return true;
}

// The steps over the block's kb columns for this warp's column group (0..3: the block's own columns; above: block row;
// group < 0: none) held in acc.  Every thread of the CTA calls it.  Returns false, in every thread, when a pivot fails (S.fail says where).
// On return acc holds the group's rows of R (own columns: rows of the earlier groups; the block itself is in S.R).
__device__ __forceinline__ bool p64_run(P64Smem& S, double (&acc)[8][4], int group, int kb) {
  const int lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
  if (threadIdx.x == 0) S.fail = 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    double* Rb = S.R + 16 * p * P64_RLD + 16 * p;
    if (group == p) {
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          S.D[(g + 8 * (e >> 1)) * P64_DLD + 8 * b + 2 * t + (e & 1)] = acc[2 * p + b][e];
      __syncwarp();
      if (!p64_factor16(S, Rb, S.W[p]) && lane == 0) S.fail = 1 + 16 * p;
    }
    __syncthreads();
    if (S.fail) return false;
    if (group > p) {
      double x[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
      const double* Wg = S.W[p] + g * P64_WLD + 2 * t;
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n) p64_mma_tile(x[n], acc[2 * p + k], 1.0, Wg + 8 * n * P64_WLD + 8 * k);
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n)
          p64_mma_tile(acc[2 * p + n], x[k], -1.0, Rb + (8 * n + g) * P64_RLD + 8 * k + 2 * t);
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n) p64_mma_tile(x[n], acc[2 * p + k], 1.0, Wg + 8 * n * P64_WLD + 8 * k);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[2 * p + n][e] = x[n][e];
      if (group < 4) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            *reinterpret_cast<double2*>(S.R + (16 * group + g + 8 * h) * P64_RLD + 16 * p + 8 * n + 2 * t) =
                make_double2(x[n][2 * h], x[n][2 * h + 1]);
      }
    }
    if (p == 3 || 16 * (p + 1) >= kb) break;  // no columns left: what follows is the padding's identity
    __syncthreads();
    if (group > p) {
#pragma unroll
      for (int r = p + 1; r < 4; ++r) {
        if (group < r) break;  // rows past the group's own diagonal block are not needed
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int k = 0; k < 2; ++k)
            p64_mma_tile(acc[2 * r + n], acc[2 * p + k], -1.0,
                         S.R + (16 * r + 8 * n + g) * P64_RLD + 16 * p + 8 * k + 2 * t);
      }
    }
  }
  return true;
}

// acc <- columns c0 .. c0 + 15 (those below cl exist), rows k0 .. k0 + kb - 1 of the column-major A; zero elsewhere.
// diag >= 0: the group is columns 16 diag.. of the diagonal block: entries below the diagonal read as zero, columns
// and rows at or past kb as the identity.  L2 loads (another CTA of the launch may have written them).
template <bool VEC>
__device__ __forceinline__ void p64_load(double (&acc)[8][4], const double* A, long long lda, int k0, int kb, int c0,
                                         int cl, int diag) {
  const int lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = c0 + g + 8 * h;
    const double* col = A + (long long)c * lda + k0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int i = 8 * b + 2 * t;
      double v0 = 0.0, v1 = 0.0;
      if (c < cl) {
        if (VEC && i + 1 < kb) {
          const double2 v = __ldcg(reinterpret_cast<const double2*>(col + i));
          v0 = v.x;
          v1 = v.y;
        } else {
          if (i < kb) v0 = __ldcg(col + i);
          if (i + 1 < kb) v1 = __ldcg(col + i + 1);
        }
      }
      if (diag >= 0) {
        const int j = 16 * diag + g + 8 * h;
        if (i > j) v0 = 0.0;
        if (i + 1 > j) v1 = 0.0;
        if (j >= kb) {
          if (i == j) v0 = 1.0;
          if (i + 1 == j) v1 = 1.0;
        }
      }
      acc[b][2 * h] = v0;
      acc[b][2 * h + 1] = v1;
    }
  }
}

template <bool VEC>
__device__ __forceinline__ void p64_store(const double (&acc)[8][4], double* A, long long lda, int k0, int kb, int c0,
                                          int cl) {
  const int lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = c0 + g + 8 * h;
    if (c >= cl) continue;
    double* col = A + (long long)c * lda + k0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int i = 8 * b + 2 * t;
      if (VEC && i + 1 < kb) {
        *reinterpret_cast<double2*>(col + i) = make_double2(acc[b][2 * h], acc[b][2 * h + 1]);
      } else {
        if (i < kb) col[i] = acc[b][2 * h];
        if (i + 1 < kb) col[i + 1] = acc[b][2 * h + 1];
      }
    }
  }
}

// The inverses W = R_pp^-T of the block's 16 x 16 diagonal blocks (those that hold one of its kb columns), row major 256
// doubles each, for the triangular solves.
__device__ __forceinline__ void p64_store_inverses(const P64Smem& S, double* W, int kb) {
  for (int e = threadIdx.x; e < (kb + 15) / 16 * 256; e += P64_THREADS)
    W[e] = S.W[e / 256][(e % 256) / 16 * P64_WLD + e % 16];
}

}  // namespace db200
