// coarse.cu -- inverses of small dense SPD matrices (up to 512 rows: 8^3
// aggregates) by Gauss-Jordan elimination with 32 x 32 pivot blocks.
//
// One launch per pivot block K of the sequence: with D the current diagonal
// block, the blocks of the next matrix are
//   KK: D^-1    KJ: D^-1 M_KJ    IK: -M_IK D^-1    IJ: M_IJ - M_IK D^-1 M_KJ,
// all from the previous matrix, so that one launch needs no barrier inside: one
// block per 32 x 32 tile inverts D again for itself (the serial part, which
// every tile would wait for anyway) and multiplies.  The launches go from one
// buffer to the other.
//
// What bounds it: the 32 pivots of D in sequence (a barrier, a shared load, two
// multiply-adds and a reciprocal each); a launch measured 13.4 us at 216 rows (7 of
// them) and 19.4 us at 512 (16).  On the host (Cholesky, triangular inverse, product)
// the same inverse took 1.5 ms and 10 ms and the copies both ways with a
// synchronisation; each solve had to wait for it or use the inverse of the solve
// before.  A coupled step of 24^3 x 6 tetrahedra went from 4.6 to 2.7 ms, one of
// 47^3 x 6 with FP32 elements from 28 to 19 ms.
#include <algorithm>

#include "coarse.h"
#include "internal.h"

namespace ufem {
namespace {

constexpr int kB = kCoarsePanel;
constexpr int kListMax = 32;  // matrices of one launch (kernel arguments)

struct InverseList {
  CoarseInverse e[kListMax];
};

struct Pivot {
  double row[2][kB], next[2];
  __align__(16) double col[2][kB];
};

// Inverts the 32 x 32 SPD block held by the first four warps, warp w its rows
// 8 w .. 8 w + 7 and lane j its column j; false (in every one of their threads) if
// a pivot is not positive and finite.  The pivot's row and column go through
// shared memory (two buffers, so one barrier a pivot); every thread works out the
// next pivot beside them, so that its reciprocal, the longest link of the chain,
// runs while the rest is updated and published.
__device__ __forceinline__ bool invert_block(double (&d)[8], int w, int lane, double first, Pivot& sh) {
  double piv = first;
  bool ok = piv > 0.0 && piv < INFINITY;
  double ip = __drcp_rn(piv);
  for (int g = 0; g < 4; ++g) {
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const int k = 8 * g + kk, b = kk & 1;
      if (w == g) sh.row[b][lane] = d[kk];
      if (w == g + (kk == 7) && lane == k + 1) sh.next[b] = d[(kk + 1) & 7];
      if (lane == k) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) *reinterpret_cast<double2*>(&sh.col[b][8 * w + i]) = make_double2(d[i], d[i + 1]);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const double ipk = ip, m = lane == k ? ipk : sh.row[b][lane] * ipk;
      if (k + 1 < kB) {  // the arithmetic of the entry's owner below
        piv = fma(-sh.col[b][k + 1], sh.row[b][k + 1] * ipk, sh.next[b]);
        ok = ok && piv > 0.0 && piv < INFINITY;
        ip = __drcp_rn(piv);
      }
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const double2 c = *reinterpret_cast<const double2*>(&sh.col[b][8 * w + i]);
        d[i] = w == g && i == kk ? m : fma(-c.x, m, lane == k ? 0.0 : d[i]);
        d[i + 1] = w == g && i + 1 == kk ? m : fma(-c.y, m, lane == k ? 0.0 : d[i + 1]);
      }
    }
  }
  return ok;
}

__global__ void __launch_bounds__(256) coarse_panel_kernel(const __grid_constant__ InverseList list, int p) {
  const CoarseInverse& e = list.e[blockIdx.z];
  const int n = e.n, k0 = p * kB, i0 = int(blockIdx.y) * kB, j0 = int(blockIdx.x) * kB;
  if (k0 >= n || i0 >= n || j0 >= n) return;
  const bool odd = ((n + kB - 1) / kB - p) & 1;
  const double* __restrict__ src = odd ? e.scratch : e.inv;
  double* __restrict__ dst = odd ? e.inv : e.scratch;
  __shared__ double D[kB][kB + 1], C[kB][kB + 1];
  __shared__ __align__(16) double R[kB][kB], W[kB][kB];
  __shared__ Pivot pivot;
  __shared__ int sound;
  const int t = threadIdx.x, r = t >> 3, c4 = (t & 7) * 4;
  const bool inK = i0 == k0, jnK = j0 == k0;
  double own[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    own[j] = !jnK && !inK && i0 + r < n && j0 + c4 + j < n ? src[size_t(i0 + r) * n + j0 + c4 + j] : 0.0;
  if (t < 128) {
    const int wid = t >> 5, lane = t & 31;
    double d[8];
    // past the matrix: the identity, so that the last pivot block is whole
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int gr = k0 + 8 * wid + i, gc = k0 + lane;
      d[i] = gr < n && gc < n ? src[size_t(gr) * n + gc] : (gr == gc ? 1.0 : 0.0);
    }
    const bool good = invert_block(d, wid, lane, src[size_t(k0) * n + k0], pivot);
#pragma unroll
    for (int i = 0; i < 8; ++i) D[8 * wid + i][lane] = d[i];
    if (t == 0) sound = good;
  } else {  // the other four warps bring the panels
    for (int q = t - 128; q < kB * kB; q += 128) {
      const int a = q / kB, b = q % kB;
      C[a][b] = i0 + a < n && k0 + b < n ? src[size_t(i0 + a) * n + k0 + b] : 0.0;
      R[a][b] = !jnK && k0 + a < n && j0 + b < n ? src[size_t(k0 + a) * n + j0 + b] : 0.0;
    }
  }
  __syncthreads();
  const bool ok = sound != 0;
  double w[4] = {D[r][c4], D[r][c4 + 1], D[r][c4 + 2], D[r][c4 + 3]};
  if (!jnK) {  // W = D^-1 M_KJ
    w[0] = w[1] = w[2] = w[3] = 0.0;
#pragma unroll 8
    for (int q = 0; q < kB; ++q) {
      const double a = D[r][q];
      const double2 x = *reinterpret_cast<const double2*>(&R[q][c4]);
      const double2 y = *reinterpret_cast<const double2*>(&R[q][c4 + 2]);
      w[0] = fma(a, x.x, w[0]);
      w[1] = fma(a, x.y, w[1]);
      w[2] = fma(a, y.x, w[2]);
      w[3] = fma(a, y.y, w[3]);
    }
  }
  if (!inK) {
    *reinterpret_cast<double2*>(&W[r][c4]) = make_double2(w[0], w[1]);
    *reinterpret_cast<double2*>(&W[r][c4 + 2]) = make_double2(w[2], w[3]);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = own[j];
#pragma unroll 8
    for (int q = 0; q < kB; ++q) {
      const double a = -C[r][q];
      const double2 x = *reinterpret_cast<const double2*>(&W[q][c4]);
      const double2 y = *reinterpret_cast<const double2*>(&W[q][c4 + 2]);
      w[0] = fma(a, x.x, w[0]);
      w[1] = fma(a, x.y, w[1]);
      w[2] = fma(a, y.x, w[2]);
      w[3] = fma(a, y.y, w[3]);
    }
  }
  // a failed pivot leaves zeros, which fail every later pivot: a zero inverse
  if (i0 + r < n)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j0 + c4 + j < n) dst[size_t(i0 + r) * n + j0 + c4 + j] = ok ? w[j] : 0.0;
}

}  // namespace

int coarse_invert(const CoarseInverse* list, int count, cudaStream_t s) {
  for (int m0 = 0; m0 < count; m0 += kListMax) {
    InverseList l{};
    const int m = std::min(kListMax, count - m0);
    int panels = 0;
    for (int k = 0; k < m; ++k) {
      l.e[k] = list[m0 + k];
      panels = std::max(panels, coarse_panels(l.e[k].n));
    }
    for (int p = 0; p < panels; ++p)
      coarse_panel_kernel<<<dim3(unsigned(panels), unsigned(panels), unsigned(m)), 256, 0, s>>>(l, p);
    UFEM_CUDA_TRY(cudaGetLastError());
  }
  return UFEM_OK;
}

}  // namespace ufem
