// persist.cu -- BiCGStab and CG solves of one system in one launch.
//
// The multi-launch solvers of krylov.cu spend 7 (point Jacobi) to 13 (two-level)
// launches of a few microseconds on an iteration; on systems whose matrix fits
// shared memory or the L2 cache those launches, not the bytes, set the time.
// Here a set of blocks owns the system for the whole solve, each a contiguous
// range of nodes, and meets at barriers: three an iteration for BiCGStab, two
// for CG, each of them also the all-reduce of the dot products (every block folds
// the block partials in block order, so all blocks hold the same scalars).  A
// block copies what its rows touch -- its own nodes and their neighbours -- once a
// product, as the preconditioned combination of two stored vectors,
// ph_j = D^-1 (r_j + beta q_j) with q = p - omega v and sh_j = D^-1 (r_j - alpha v_j),
// which saves the barrier between forming a direction and applying the matrix
// to it; p, s and their preconditioned forms are never stored.  The two-level
// forms add a barrier after the restriction and one after the coarse product
// before each product; the correction enters with that copy.  (In the grid form a
// restriction of the updated residual is summed beside the update, from its
// published terms, and needs no barrier of its own.)
//
// Two forms (persist_plan chooses):
//  - cluster: up to 16 blocks of one thread-block cluster; vectors and matrix live
//    in the cluster's shared memory, the copies go over distributed shared memory
//    and the barriers are the cluster's (0.7-1.0 us with the reduction);
//  - grid: a cooperative launch of one block per SM (2.3 us a barrier with the
//    reduction); the vectors other blocks read live in L2, the rest and as much
//    of the matrix as fits in shared memory.
// Cached values are kept a thread per row, lane-consecutive (no shuffles, no
// bank conflicts).  State that would spill is kept out of registers by 32-bit
// shared-memory offsets: a spilled value costs an L2 round trip after every grid
// barrier, whose acquire invalidates L1.
//
// What bounds it: barriers and the latency of each phase, not bytes.  An
// iteration, launches against this: 64 x 64 x 2 triangles, BiCGStab with point
// Jacobi, 27 -> 9.1 us (cluster of 16); 24^3 x 6 tetrahedra, two-level BiCGStab,
// 46 -> 21 us; 32^3 x 6, two-level CG of the pressure 29 -> 12.8 us, CG of the
// velocity 24 -> 16.3 us (grid).  (With the restriction after the update and its own
// barrier, and the coarse sums' last rows one at a time, the two-level forms took 27
// and 13.5 us.)
//
// A block's rows are a range of node numbers, so a scattered numbering costs: a block
// then touches 7 (triangles) to 14 (tetrahedra) times its own nodes instead of 2 to 5,
// copies as many more a product, and has less room for values.  28^3 x 6 in random
// order: point Jacobi 32.5 us an iteration (natural 23.0; launches 43.5), two-level
// 45.0 (32.5; 67).  From 32^3 x 6 or 260^2 x 2 in random order the lists and vectors
// no longer fit, and the launches take the system (natural order: up to the 96 MB of
// persist_plan, triangles up to 360^2).
//
// All sums run in fixed orders, so a solve is deterministic; FP64 throughout,
// FP32 only in the stored values of the mixed forms.  Grid barriers wait a
// bounded time: one that runs out sets a flag that ends this launch and those
// queued after it, and that the host turns into an error.
#include "persist.h"

#include <algorithm>
#include <vector>

#include "internal.h"
#include "spmv_node.cuh"

namespace ufem {
namespace {

constexpr int kThreads = 512;  // one block an SM: 128 registers a thread
constexpr int kWarps = kThreads / 32;
constexpr int kClusterMax = 16;  // the non-portable cluster size
constexpr unsigned FULL = 0xffffffffu;

extern __shared__ __align__(16) unsigned char g_smem[];

struct Shared {
  double red[3][kWarps];
  double out[3];
  double parts[2][3][kClusterMax];  // cluster form: the blocks' partials, two barriers' worth
  int late;
};

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(int* p) {
  asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this block's shared variable `p` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(const void* p, int rank) {
  uint32_t a = uint32_t(__cvta_generic_to_shared(p)), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(uint32_t addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// Bytes a slice of 32 / neq nodes takes per neighbour: 32 lanes' values (a row's
// neq each) and the nodes' 2-byte neighbour places.
__host__ __device__ constexpr int slice_bytes(int neq, size_t value) {
  return neq * 32 * int(value) + (32 / neq * 2 + 15) / 16 * 16;
}

constexpr int kVecs = 6;  // own vectors of a block
// Aggregates and coarse rows a block takes, and how many rows of an aggregate it
// lists in shared memory.
constexpr int kAggRows = 256;
__host__ __device__ inline int coarse_rows(int nc, int blocks) { return (nc + blocks - 1) / blocks; }

// One block's view of the solve.  Own vectors are indexed by the local row; the
// operand of a product is the block's copy of every node its rows touch (its own
// nodes and their neighbours in other blocks, ascending), filled once a product.
template <int NEQ, typename MT, bool CL>
struct Ctx {
  static constexpr int NB = NEQ * NEQ;
  static constexpr int NPW = 32 / NEQ;                         // nodes of a slice: a lane per row
  static constexpr int kSliceBytes = slice_bytes(NEQ, sizeof(MT));  // ... with the neighbours' places
  static constexpr int kSliceRow = NEQ * 32 * int(sizeof(MT));  // bytes of one neighbour's values in a slice
  const PersistSolve& a;
  Shared& sh;
  int rank, blocks;
  int N, n0, n1;    // the block's nodes
  int U, u0;        // touched nodes, and the place of n0 among them (own nodes are consecutive)
  int nslice;       // slices of NPW nodes whose values are in shared memory (the first of the range)
  int64_t base;     // the range's first block entry
  int epoch = 0;
  int par = 0;      // which of the two global copies of r and q is the current one (grid form)
  int wide;         // entries of one vector's place in shared memory
  // byte places in shared memory (Layout)
  int o_off, o_soff, o_adj, o_touched, o_tagg, o_dinv, o_u, o_vals, o_coarse;

  // Own vectors (local row i): 0 x, 1 r, 2 shadow residual, 3 q, 4 v, 5 t; CG: 3 and
  // 4 the direction's buffers, 5 A p.
  __device__ __forceinline__ double* vec(int k) const { return reinterpret_cast<double*>(g_smem) + k * wide; }
  __device__ __forceinline__ double& x(int i) const { return vec(0)[i]; }
  __device__ __forceinline__ double& r(int i) const { return vec(1)[i]; }
  __device__ __forceinline__ double& rh(int i) const { return vec(2)[i]; }
  __device__ __forceinline__ double& q(int i) const { return vec(3)[i]; }
  __device__ __forceinline__ double& v(int i) const { return vec(4)[i]; }
  __device__ __forceinline__ double& t(int i) const { return vec(5)[i]; }
  // The global copy of vectors 1, 3 and 4 (grid form: what other blocks read).
  __device__ __forceinline__ double* global(int k) const {
    return k == 1 ? (par ? a.r2 : a.r) : k == 3 ? (par ? a.q2 : a.q) : a.v;
  }
  // Stores entry i of vector k where its readers look for it.
  __device__ __forceinline__ void publish(int k, int i, double s) const {
    vec(k)[i] = s;
    if constexpr (!CL) global(k)[n0 * NEQ + i] = s;
  }
  // Coarse vectors (0: c, 1: y1, 2: y2; cluster: this block's copies).
  __device__ __forceinline__ double* coarse_vec(int k) const {
    if constexpr (CL) return vec(kVecs) + k * a.nc;
    else return k == 0 ? a.cvec : a.yvec + (k - 1) * a.nc;
  }
  // The block's copy of y1 or y2, which its entries read (grid form: made by fill; read in
  // L2, every block's gather would meet on the few lines that hold y).
  __device__ __forceinline__ double* near_y(int k) const { return vec(kVecs) + (CL ? k : k - 1) * a.nc; }
  __device__ __forceinline__ const int* off() const { return reinterpret_cast<const int*>(g_smem + o_off); }
  __device__ __forceinline__ const int* soff() const { return reinterpret_cast<const int*>(g_smem + o_soff); }
  __device__ __forceinline__ const uint16_t* adj() const { return reinterpret_cast<const uint16_t*>(g_smem + o_adj); }
  __device__ __forceinline__ const int* touched() const { return reinterpret_cast<const int*>(g_smem + o_touched); }
  // node ids of the touched nodes (cluster: after their addresses)
  __device__ __forceinline__ const int* tnode() const { return touched() + (CL ? U : 0); }
  __device__ __forceinline__ const int16_t* tagg() const { return reinterpret_cast<const int16_t*>(g_smem + o_tagg); }
  __device__ __forceinline__ double* tdinv() const { return reinterpret_cast<double*>(g_smem + o_dinv); }
  __device__ __forceinline__ double dinv(int i) const { return tdinv()[u0 * NEQ + i]; }
  __device__ __forceinline__ double* u() const { return reinterpret_cast<double*>(g_smem + o_u); }
  __device__ __forceinline__ const MT* gvals() const { return static_cast<const MT*>(a.vals) + int64_t(NB) * base; }
  // Coarse rows of this block: I = rank + k * blocks; the rows of aggregate I (the
  // first kAggRows of them) in shared memory.
  __device__ __forceinline__ int* agg_rows_of(int k) const {
    return reinterpret_cast<int*>(g_smem + o_coarse) + k * kAggRows;
  }

  __device__ __forceinline__ int rows() const { return (n1 - n0) * NEQ; }
  // Most neighbours of a node in slice sl.
  __device__ __forceinline__ int swidth(int sl) const { return (soff()[sl + 1] - soff()[sl]) / kSliceBytes; }

  // Barrier and all-reduce of K sums (K = 0: barrier only): every thread brings
  // its share, every thread gets the totals.  `slot`: the partials' place in the
  // grid form (reused at least one barrier apart).  False, in every thread of
  // the block, when a grid barrier ran out.
  template <int K>
  __device__ __forceinline__ bool sum(int slot, double (&w)[K < 1 ? 1 : K]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ++epoch;
    if constexpr (K == 0 && CL) {
      cluster_sync();
      return true;
    }
    if constexpr (K > 0) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const double s = wsum(w[k]);
        if (lane == 0) sh.red[k][warp] = s;
      }
    }
    __syncthreads();
    if constexpr (CL) {
      if (warp == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const double s = wsum(lane < kWarps ? sh.red[k][lane] : 0.0);
          if (lane < blocks) st_cluster(map_rank(&sh.parts[epoch & 1][k][rank], lane), s);
        }
      }
      cluster_sync();
#pragma unroll
      for (int k = 0; k < K; ++k) {  // a fixed tree over the 16 places (unused ones hold zero)
        double s[kClusterMax];
#pragma unroll
        for (int b = 0; b < kClusterMax; ++b) s[b] = sh.parts[epoch & 1][k][b];
#pragma unroll
        for (int o = kClusterMax / 2; o > 0; o >>= 1)
#pragma unroll
          for (int b = 0; b < o; ++b) s[b] += s[b + o];
        w[k] = s[0];
      }
      return true;
    } else {
      if (warp == 0) {
        if constexpr (K > 0) {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const double s = wsum(lane < kWarps ? sh.red[k][lane] : 0.0);
            if (lane == 0) __stcg(a.part + (slot + k) * kPersistMaxBlocks + rank, s);
          }
        }
        if (lane == 0) {
          red_release(a.ictl + kFlagBarrier);
          const int target = epoch * blocks;
          int spins = 0, late = 0;
          while (ld_acquire(a.ictl + kFlagBarrier) < target)
            if (++spins > kPersistPolls) {
              late = 1;
              break;
            }
          sh.late = late;
        }
        __syncwarp();
        if constexpr (K > 0) {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            double s = 0.0;
            for (int b = lane; b < blocks; b += 32) s += __ldcg(a.part + (slot + k) * kPersistMaxBlocks + b);
            s = wsum(s);
            if (lane == 0) sh.out[k] = s;
          }
        }
      }
      __syncthreads();
      if constexpr (K > 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) w[k] = sh.out[k];
      }
      return sh.late == 0;
    }
  }
  __device__ __forceinline__ bool barrier() {
    double none[1];
    return sum<0>(0, none);
  }

  // u = D^-1 (r + k w) on every touched node, w vector kw, plus the coarse
  // correction ky (0: none) on the node's last component.  Four entries a thread
  // in flight: the loads cross the cluster or go to L2.  plain: u = D^-1 r + k w
  // (CG's direction).  28^3 x 6 tetrahedra in random order, two-level BiCGStab: 70.9 us an
  // iteration with y gathered from L2 (67 in 13 launches), 45.3 with the block's copy; in
  // natural order 35.8 -> 32.5.
  __device__ __forceinline__ void fill(int kw, double k, int ky, bool plain = false) const {
    constexpr int Q = 4;
    const uint32_t dw = uint32_t((kw - 1) * wide) * 8u;
    const double* gr = global(1);
    const double* gw = global(kw);
    double* y = ky ? near_y(ky) : nullptr;
    const int* list = touched();
    const double* di = tdinv();
    double* out = u();
    const int n = U * NEQ;
    for (int s0 = 0; s0 < n; s0 += Q * kThreads) {  // the same trips for every thread
      const int i0 = s0 + int(threadIdx.x);
      double g[Q], w[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int i = i0 + q * kThreads;
        if (i < n) {
          const int j = i / NEQ, c = i - j * NEQ;
          if constexpr (CL) {
            const uint32_t addr = uint32_t(list[j]) + 8u * uint32_t(c);
            g[q] = ld_cluster(addr);
            w[q] = ld_cluster(addr + dw);
          } else {
            const int row = list[j] * NEQ + c;
            g[q] = __ldcg(gr + row);
            w[q] = __ldcg(gw + row);
          }
        }
      }
      if constexpr (!CL)
        if (s0 == 0 && y != nullptr) {  // beside the first loads
          for (int J = threadIdx.x; J < a.nc; J += kThreads) y[J] = __ldcg(coarse_vec(ky) + J);
          __syncthreads();
        }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int i = i0 + q * kThreads;
        if (i < n) {
          double z = 0.0;
          if (y != nullptr && (NEQ == 1 || i % NEQ == NEQ - 1)) {
            const int ag = tagg()[i / NEQ];
            if (ag >= 0) z = y[ag];
          }
          out[i] = (plain ? di[i] * g[q] + k * w[q] : di[i] * (g[q] + k * w[q])) + z;
        }
      }
    }
    __syncthreads();
  }
  // u = x on every touched node, x in global memory.
  __device__ __forceinline__ void fill_x() const {
    const int* list = tnode();
    double* out = u();
    for (int i = threadIdx.x; i < U * NEQ; i += kThreads) {
      const int j = i / NEQ;
      out[i] = __ldcg(a.x + list[j] * NEQ + (i - j * NEQ));
    }
    __syncthreads();
  }

  // A u over the block's nodes; epi(local row, sum) runs on one lane per row.
  // Cached slices: a thread per row, its values one after another in shared
  // memory at lane-consecutive places, so nothing is shuffled and no bank
  // conflicts.  The other nodes, from global memory: a warp (NEQ = 4) or 8 lanes
  // per node as in spmv4_walk and spmv_group_walk.
  template <typename E>
  __device__ __forceinline__ void product(E&& epi) const {
    const int nodes = n1 - n0;
    const double* uu = u();
    const int* of = off();
    const uint16_t* ad = adj();
    const MT* gv = gvals();
    const int lane = threadIdx.x & 31, warp = int(threadIdx.x >> 5);
    const int first = min(nodes, nslice * NPW);
    if constexpr (NEQ == 4) {
      using MP = typename Pair<MT>::type;
#pragma unroll 1
      for (int node = first + warp; node < nodes; node += kWarps) {
        const int s0 = of[node], S = of[node + 1] - s0;
        const MP* rp = reinterpret_cast<const MP*>(gv + int64_t(16) * s0);
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
        for (int p = lane; p < 2 * S; p += 32) {
          const double2 xv = *reinterpret_cast<const double2*>(uu + int(ad[s0 + (p >> 1)]) * 4 + (p & 1) * 2);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const MP w = __ldg(rp + (r * 2 * S + p));
            acc[r] = fma(double(w.x), xv.x, acc[r]);
            acc[r] = fma(double(w.y), xv.y, acc[r]);
          }
        }
        const double s = warp_sum4(acc, lane);
        if ((lane & 7) == 0) epi(node * 4 + (lane >> 3), s);
      }
    } else {
      constexpr int kGroups = kThreads / 8;
      const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
      const int wbase = grp & ~3;  // the warp's first group: the same trip count for its 32 lanes
      for (int nb = first; nb + wbase < nodes; nb += kGroups) {
        const int i = nb + grp;
        const bool valid = i < nodes;
        const int s0 = valid ? of[i] : 0, S = valid ? of[i + 1] - s0 : 0;
        double acc[NEQ];
#pragma unroll
        for (int r = 0; r < NEQ; ++r) acc[r] = 0.0;
        const MT* row = gv + NB * s0;
        const int len = NEQ * S;
        for (int s = sub; s < S; s += 8) {
          const double* us = uu + int(ad[s0 + s]) * NEQ;
          MT w[NB];
#pragma unroll
          for (int r = 0; r < NEQ; ++r)
#pragma unroll
            for (int c = 0; c < NEQ; ++c) w[r * NEQ + c] = __ldg(row + r * len + s * NEQ + c);
#pragma unroll
          for (int r = 0; r < NEQ; ++r)
#pragma unroll
            for (int c = 0; c < NEQ; ++c) acc[r] = fma(double(w[r * NEQ + c]), us[c], acc[r]);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < NEQ; ++r) {
          acc[r] += __shfl_xor_sync(FULL, acc[r], 4);
          acc[r] += __shfl_xor_sync(FULL, acc[r], 2);
          acc[r] += __shfl_xor_sync(FULL, acc[r], 1);
        }
        double mine = acc[0];
#pragma unroll
        for (int r = 1; r < NEQ; ++r)
          if (sub == r) mine = acc[r];
        if (valid && sub < NEQ) epi(i * NEQ + sub, mine);
      }
    }
    const int ln = lane / NEQ;  // the lane's node in a slice, its row lane - ln * NEQ
    for (int sl = warp; sl < nslice; sl += kWarps) {
      const int node = sl * NPW + ln;
      if (ln >= NPW || node >= nodes) continue;
      const unsigned char* p = g_smem + o_vals + soff()[sl];
      const int width = swidth(sl);
      const uint16_t* sa = reinterpret_cast<const uint16_t*>(p + size_t(width) * kSliceRow) + ln;
      double acc = 0.0;
      if constexpr (NEQ == 4) {
        using MP = typename Pair<MT>::type;
        const MP* sv = reinterpret_cast<const MP*>(p) + lane;
#pragma unroll 2
        for (int s = 0; s < width; ++s) {
          const double2* us = reinterpret_cast<const double2*>(uu + int(sa[s * NPW]) * 4);
          const double2 x0 = us[0], x1 = us[1];
          const MP w0 = sv[s * 64], w1 = sv[s * 64 + 32];
          acc = fma(double(w0.x), x0.x, acc);
          acc = fma(double(w0.y), x0.y, acc);
          acc = fma(double(w1.x), x1.x, acc);
          acc = fma(double(w1.y), x1.y, acc);
        }
      } else {
        const MT* sv = reinterpret_cast<const MT*>(p) + lane;
#pragma unroll 4
        for (int s = 0; s < width; ++s) {
          const double* us = uu + int(sa[s * NPW]) * NEQ;
#pragma unroll
          for (int c = 0; c < NEQ; ++c) acc = fma(double(sv[(s * NEQ + c) * 32]), us[c], acc);
        }
      }
      epi(sl * NPW * NEQ + lane, acc);
    }
  }

  // Row i of own vector k (cluster: in its owner's shared memory; grid: its
  // global copy gw).
  __device__ __forceinline__ double row_of(int k, const double* gw, int i) const {
    if constexpr (CL) {
      const int node = i / NEQ;
      const int owner = int((uint32_t(node + 1) * uint32_t(blocks) - 1u) / uint32_t(N));
      const int first = int(uint32_t(N) * uint32_t(owner) / uint32_t(blocks));
      return ld_cluster(map_rank(vec(k), owner) + uint32_t(i - first * NEQ) * 8u);
    } else {
      return __ldcg(gw + i);
    }
  }
  // Entry I of a coarse vector, to every block.
  __device__ __forceinline__ void put(double* w, int I, double s) const {
    const int lane = threadIdx.x & 31;
    if constexpr (CL) {
      if (lane < blocks) st_cluster(map_rank(w + I, lane), s);
    } else {
      if (lane == 0) w[I] = s;
    }
  }
  // K coarse vectors (the first of them coarse_vec(0), the others after it: grid form)
  // from the rows of each aggregate, one warp an aggregate, the block's last warps
  // first: at(row, shares) gives a row's shares.  Four rows a lane in flight, the last
  // ones too (a remainder loop would wait for the L2 once a row).
  template <int K, typename F>
  __device__ __forceinline__ void restrict_rows(F&& at) const {
    const int lane = threadIdx.x & 31, warp = int(threadIdx.x >> 5);
    double* cs = coarse_vec(0);
#pragma unroll 1
    for (int k = kWarps - 1 - warp; rank + k * blocks < a.nc; k += kWarps) {
      const int* list = agg_rows_of(k);
      const int p0 = list[0], len = list[1];
      double s[K];
#pragma unroll
      for (int q = 0; q < K; ++q) s[q] = 0.0;
      constexpr int Q = 4;
      const int near = min(len, kAggRows - 2);
#pragma unroll 1
      for (int j0 = lane; j0 < len; j0 += Q * 32) {
        double v[Q][K];
#pragma unroll
        for (int b = 0; b < Q; ++b) {
          const int j = min(j0 + b * 32, len - 1);
          at(j < near ? list[2 + j] : __ldg(a.agg_rows + p0 + j), v[b]);
        }
#pragma unroll
        for (int b = 0; b < Q; ++b)
#pragma unroll
          for (int q = 0; q < K; ++q)
            if (j0 + b * 32 < len) s[q] += v[b][q];
      }
#pragma unroll
      for (int q = 0; q < K; ++q) put(cs + q * a.nc, rank + k * blocks, wsum(s[q]));
    }
  }
  // y = Ac^-1 c (coarse vector ky), c = coarse_vec(0), PAIR: plus k2 times the one
  // after it; one warp a coarse row.  cy: the thread's share of c . y.
  template <bool PAIR>
  __device__ __forceinline__ void coarse_product(int ky, double k2, double* cy) const {
    const double* cs = coarse_vec(0);
    double* y = coarse_vec(ky);
    const int lane = threadIdx.x & 31, warp = int(threadIdx.x >> 5);
    auto entry = [&](int J) {
      double v = CL ? cs[J] : __ldcg(cs + J);
      if constexpr (PAIR) v += k2 * __ldcg(cs + a.nc + J);
      return v;
    };
#pragma unroll 1
    for (int k = warp; rank + k * blocks < a.nc; k += kWarps) {
      const int I = rank + k * blocks;
      const double* inv = a.ainv + int64_t(I) * a.nc;
      double s = 0.0;
      constexpr int Q = 8;  // in flight, the last ones too
#pragma unroll 1
      for (int J0 = lane; J0 < a.nc; J0 += Q * 32) {
        double m[Q], v[Q];
#pragma unroll
        for (int b = 0; b < Q; ++b) {
          const int J = min(J0 + b * 32, a.nc - 1);
          m[b] = __ldg(inv + J);
          v[b] = entry(J);
        }
#pragma unroll
        for (int b = 0; b < Q; ++b)
          if (J0 + b * 32 < a.nc) s += m[b] * v[b];
      }
      s = wsum(s);
      put(y, I, s);
      if (cy != nullptr && lane == 0) *cy += entry(I) * s;
    }
  }
  // y = Ac^-1 R^T value(row), a barrier between the two (the caller's next one
  // covers y).
  template <typename F>
  __device__ __forceinline__ bool correct(int ky, F&& value, double* cy) {
    restrict_rows<1>([&](int i, double (&s)[1]) { s[0] = value(i); });
    if (!barrier()) return false;
    coarse_product<false>(ky, 0.0, cy);
    return true;
  }
};

// Shared memory of a block, in this order: own vectors and coarse vectors (grid form:
// copies of y1 and y2) -- the same places in every block of a cluster -- then row starts, slice
// starts, neighbour places, touched nodes and their aggregates and inverse
// diagonals, the operand, the rows of the block's aggregates, and values in what
// is left.
struct Layout {
  size_t off, soff, adj, touched, tagg, dinv, u, coarse, vals;
};
__host__ __device__ inline size_t align16(size_t b) { return (b + 15) & ~size_t(15); }
__host__ __device__ inline size_t uniform_bytes(int64_t wide, bool cluster, int nc) {
  return align16(size_t(wide) * 8 * kVecs + size_t(nc) * (cluster ? 24 : 16));
}
__host__ __device__ inline Layout layout(size_t uniform, int64_t nodes, int64_t entries, int64_t U, int neq, int nc,
                                         bool cluster, int blocks) {
  Layout l;
  l.off = uniform;
  l.soff = l.off + size_t(nodes + 1) * 4;
  l.adj = align16(l.soff + size_t(nodes * neq / 30 + 3) * 4);
  l.touched = align16(l.adj + size_t(entries) * 2);
  l.tagg = align16(l.touched + size_t(U) * (cluster ? 8 : 4));
  l.dinv = align16(l.tagg + (nc > 0 ? size_t(U) * 2 : 0));
  l.u = align16(l.dinv + size_t(U) * neq * 8);
  l.coarse = align16(l.u + size_t(U) * neq * 8);
  l.vals = align16(l.coarse + size_t(coarse_rows(nc, blocks)) * kAggRows * 4);
  return l;
}
// The set of touched nodes is a bitmap with a running count per word while the
// lists are made, kept in the last bytes of the block's shared memory.
__host__ __device__ inline size_t bitmap_bytes(int64_t N) { return align16(size_t((N + 31) / 32) * 8); }

// Exclusive prefix sum over the block of one value a thread; total in *all.
__device__ __forceinline__ int block_scan(int v, Shared& sh, int* all) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int w = __shfl_up_sync(FULL, s, o);
    if (lane >= o) s += w;
  }
  int* part = reinterpret_cast<int*>(sh.red);
  if (lane == 31) part[warp] = s;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) before += part[w];
    total += part[w];
  }
  __syncthreads();
  *all = total;
  return before + s - v;
}

// The block's range: its vectors, lists and cached values in shared memory.
template <int NEQ, typename MT, bool CL>
__device__ __forceinline__ void setup(Ctx<NEQ, MT, CL>& c, int smem_bytes) {
  unsigned char* smem = g_smem;
  const PersistSolve& a = c.a;
  c.N = int(a.N);
  c.n0 = int(a.N * c.rank / c.blocks);
  c.n1 = int(a.N * (c.rank + 1) / c.blocks);
  c.base = __ldg(a.start + c.n0);
  const int cnt = int(__ldg(a.start + c.n1) - c.base);
  const int nodes = c.n1 - c.n0, nr = nodes * NEQ;
  c.wide = CL ? (c.N + c.blocks - 1) / c.blocks * NEQ : nr;
  const int64_t r0 = int64_t(c.n0) * NEQ;
  // touched nodes: a bitmap, then a running count per word
  const int words = (c.N + 31) / 32;
  uint32_t* bits = reinterpret_cast<uint32_t*>(smem + smem_bytes - bitmap_bytes(c.N));
  int* before = reinterpret_cast<int*>(bits + words);
  for (int k = threadIdx.x; k < words; k += kThreads) bits[k] = 0u;
  __syncthreads();
  for (int k = threadIdx.x; k < cnt; k += kThreads) {
    const int node = __ldg(a.adj + c.base + k);
    atomicOr(bits + (node >> 5), 1u << (node & 31));
  }
  __syncthreads();
  const int per = (words + kThreads - 1) / kThreads;
  const int w0 = min(words, int(threadIdx.x) * per), w1 = min(words, w0 + per);
  int mine = 0;
  for (int w = w0; w < w1; ++w) mine += __popc(bits[w]);
  int at = block_scan(mine, c.sh, &c.U);
  const Layout l = layout(uniform_bytes(c.wide, CL, a.nc), nodes, cnt, c.U, NEQ, a.nc, CL, c.blocks);
  int* touched = reinterpret_cast<int*>(smem + l.touched);
  int16_t* tagg = reinterpret_cast<int16_t*>(smem + l.tagg);
  for (int w = w0; w < w1; ++w) {
    before[w] = at;
    for (uint32_t m = bits[w]; m; m &= m - 1) {
      const int node = w * 32 + __ffs(int(m)) - 1;
      if (node == c.n0) c.sh.late = at;  // (handed to every thread below)
      if constexpr (CL) {
        const int owner = int((uint32_t(node + 1) * uint32_t(c.blocks) - 1u) / uint32_t(c.N));
        const int first = int(uint32_t(c.N) * uint32_t(owner) / uint32_t(c.blocks));
        touched[at] = int(map_rank(c.vec(1), owner) + uint32_t(node - first) * (NEQ * 8u));
        touched[c.U + at] = node;
      } else {
        touched[at] = node;
      }
      if (a.nc > 0) tagg[at] = int16_t(__ldg(a.agg + int64_t(node) * NEQ + NEQ - 1));
      ++at;
    }
  }
  __syncthreads();
  c.u0 = c.sh.late;
  uint16_t* adj = reinterpret_cast<uint16_t*>(smem + l.adj);
  for (int k = threadIdx.x; k < cnt; k += kThreads) {
    const int node = __ldg(a.adj + c.base + k);
    adj[k] = uint16_t(before[node >> 5] + __popc(bits[node >> 5] & ((1u << (node & 31)) - 1u)));
  }
  int* off = reinterpret_cast<int*>(smem + l.off);
  for (int k = threadIdx.x; k <= nodes; k += kThreads) off[k] = int(__ldg(a.start + c.n0 + k) - c.base);
  __syncthreads();  // the bitmap's bytes are free from here
  c.o_off = int(l.off);
  c.o_soff = int(l.soff);
  c.o_adj = int(l.adj);
  c.o_touched = int(l.touched);
  c.o_tagg = int(l.tagg);
  c.o_dinv = int(l.dinv);
  c.o_u = int(l.u);
  c.o_coarse = int(l.coarse);
  c.o_vals = int(l.vals);
  {  // inverse diagonals of the touched rows
    const int* list = c.tnode();
    double* di = c.tdinv();
    for (int i = threadIdx.x; i < c.U * NEQ; i += kThreads) {
      double d = 1.0;
      if (a.jacobi) {
        const int j = i / NEQ;
        d = double(static_cast<const MT*>(a.vals)[__ldg(a.diagpos + int64_t(list[j]) * NEQ + (i - j * NEQ))]);
        d = d != 0.0 ? 1.0 / d : 1.0;
      }
      di[i] = d;
    }
  }
  // values of as many slices as fit
  using X = Ctx<NEQ, MT, CL>;
  int* soff = reinterpret_cast<int*>(smem + l.soff);
  const int ns = (nodes + X::NPW - 1) / X::NPW;
  for (int sl = threadIdx.x; sl < ns; sl += kThreads) {
    int width = 0;
    for (int i = sl * X::NPW; i < min(nodes, (sl + 1) * X::NPW); ++i) width = max(width, off[i + 1] - off[i]);
    soff[sl + 1] = width * X::kSliceBytes;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int room = smem_bytes - int(l.vals);
    int b = 0, k = 0;
    soff[0] = 0;
    for (; k < ns && b + soff[k + 1] <= room; ++k) {
      b += soff[k + 1];
      soff[k + 1] = b;
    }
    c.sh.late = k;
  }
  __syncthreads();
  c.nslice = c.sh.late;
  unsigned char* slices = smem + l.vals;
  const MT* gv = c.gvals();
  const int lane = threadIdx.x & 31, ln = lane / NEQ, lr = lane - ln * NEQ;
  for (int sl = threadIdx.x >> 5; sl < c.nslice; sl += kWarps) {
    const int width = c.swidth(sl), node = sl * X::NPW + ln;
    const bool valid = ln < X::NPW && node < nodes;
    const int s0 = valid ? off[node] : 0, S = valid ? off[node + 1] - s0 : 0;
    const MT* row = gv + int64_t(X::NB) * s0 + lr * NEQ * S;
    MT* sv = reinterpret_cast<MT*>(slices + soff[sl]);
    uint16_t* sa = reinterpret_cast<uint16_t*>(slices + soff[sl] + size_t(width) * X::kSliceRow);
    for (int s = 0; s < width; ++s) {
      // lane-consecutive values: pairs (NEQ = 4) or single values
#pragma unroll
      for (int q = 0; q < NEQ; ++q) {
        const MT w = s < S ? __ldg(row + s * NEQ + q) : MT(0);
        const int at = NEQ == 4 ? ((s * 2 + q / 2) * 32 + lane) * 2 + q % 2 : (s * NEQ + q) * 32 + lane;
        sv[at] = w;
      }
      if (valid && lr == 0) sa[s * X::NPW + ln] = s < S ? adj[s0 + s] : uint16_t(c.u0 + node);
    }
  }
  if constexpr (CL)  // the partials of blocks the cluster does not have
    for (int k = threadIdx.x; k < 2 * 3 * kClusterMax; k += kThreads) (&c.sh.parts[0][0][0])[k] = 0.0;
  for (int i = threadIdx.x; i < nr; i += kThreads) c.x(i) = a.x[r0 + i];
  for (int k = threadIdx.x >> 5; c.rank + k * c.blocks < a.nc; k += kWarps) {
    const int p0 = __ldg(a.agg_ptr + c.rank + k * c.blocks), p1 = __ldg(a.agg_ptr + c.rank + k * c.blocks + 1);
    int* list = c.agg_rows_of(k);  // where its rows start, how many, and the first of them
    if (lane == 0) list[0] = p0;
    if (lane == 0) list[1] = p1 - p0;
    for (int j = lane; j < min(p1 - p0, kAggRows - 2); j += 32) list[2 + j] = __ldg(a.agg_rows + p0 + j);
  }
  __syncthreads();
  if constexpr (CL) cluster_sync();  // every block of the cluster runs and its partials are cleared
}

// Starts a solve: r = b - A x and its norm, ||b||^2 and r . D^-1 r.
template <int NEQ, typename MT, bool CL>
__device__ __forceinline__ bool begin(Ctx<NEQ, MT, CL>& c, double (&rr)[3], bool bicg) {
  const PersistSolve& a = c.a;
  const int r0 = c.n0 * NEQ;
  rr[0] = rr[1] = rr[2] = 0.0;
  c.fill_x();
  c.product([&](int i, double ax) {
    const double bi = a.b[r0 + i];
    const double ri = bi - ax;
    c.publish(1, i, ri);
    c.publish(3, i, 0.0);
    if (bicg) c.rh(i) = ri;
    rr[0] += ri * ri;
    rr[1] += bi * bi;
    rr[2] += ri * (c.dinv(i) * ri);
  });
  return c.template sum<3>(5, rr);  // (the loop's first sum follows at once: other slots)
}

// ||b - A x||^2 of the stored x; every block has passed a barrier since the last
// product, so the operand's place is free.
template <int NEQ, typename MT, bool CL>
__device__ __forceinline__ bool final_residual(Ctx<NEQ, MT, CL>& c, double& out) {
  const PersistSolve& a = c.a;
  const int r0 = c.n0 * NEQ;
  if (!c.barrier()) return false;  // every block's x is stored
  double tr[1] = {0.0};
  c.fill_x();
  c.product([&](int i, double ax) {
    const double ri = a.b[r0 + i] - ax;
    tr[0] += ri * ri;
  });
  const bool ok = c.template sum<1>(5, tr);
  out = tr[0];
  return ok;
}

// ||r|| <= tol ||b|| from the squares (their square roots where those are not
// safely representable).
__device__ __forceinline__ bool within(double rr, double limit) {
  const double l2 = limit * limit;
  return l2 > 1e-280 && l2 < 1e280 ? rr <= l2 : sqrt(rr) <= limit;
}

template <int NEQ, typename MT, bool CL>
__device__ __forceinline__ void bicgstab_body(const PersistSolve& a, Shared& sh, int smem_bytes, int rank, int blocks,
                                              bool first, int iters) {
  if (!first && (a.ictl[0] || a.ictl[kFlagLate])) return;  // every block of the solve reads the same flags
  Ctx<NEQ, MT, CL> c{a, sh, rank, blocks};
  setup(c, smem_bytes);
  const int nr = c.rows(), r0 = c.n0 * NEQ;
  const bool two = a.nc > 0;
  int done = 0, status = 0, count = 0;
  double rho, beta, alpha = 1.0, omega = 1.0, rr, limit;
  bool late = false, fresh = false;
  if (first) {
    double w[3];
    late = !begin(c, w, true);
    rr = rho = w[0];
    const double bnorm = sqrt(w[1]);
    limit = a.tol * bnorm;
    beta = rho;  // rho_old = alpha = omega = 1, and q = 0
    done = (sqrt(rr) <= limit || bnorm == 0.0) ? 1 : 0;
    if (!isfinite(rr)) {
      done = 1;
      status = 3;
    }
    fresh = done != 0;  // x is the initial guess: its true residual is r
    if (bnorm == 0.0)   // a zero right-hand side has the zero solution
      for (int i = threadIdx.x; i < nr; i += kThreads) c.x(i) = 0.0;
    if (rank == 0 && threadIdx.x == 0) {
      a.dctl[kBnorm] = bnorm;
      a.dctl[kBeta] = sqrt(rr);
    }
  } else {
    rho = a.dctl[kRho];
    beta = a.dctl[kHnext];
    limit = a.tol * a.dctl[kBnorm];
    rr = 0.0;
    status = a.ictl[2];
    count = a.ictl[3];
    for (int i = threadIdx.x; i < nr; i += kThreads) {
      c.r(i) = a.r[r0 + i];
      c.rh(i) = a.rh[r0 + i];
      c.q(i) = a.q[r0 + i];
    }
    if (!late) late = !c.barrier();
  }
#pragma unroll 1
  for (int it = 0; it < iters && !done && !late; ++it) {
    if (two) {
      if constexpr (CL) {
        late = !c.correct(1, [&](int i) { return c.row_of(1, a.r, i) + beta * c.row_of(3, a.q, i); }, nullptr);
      } else {
        if (it == 0) {  // later ones: beside the update below
          c.template restrict_rows<2>([&](int i, double (&s)[2]) {
            s[0] = c.row_of(1, a.r, i);
            s[1] = c.row_of(3, a.q, i);
          });
          late = !c.barrier();
        }
        if (!late) c.template coarse_product<true>(1, beta, nullptr);
      }
      if (late || !c.barrier()) {
        late = true;
        break;
      }
    }
    // v = A ph ; rh . v
    double d1[1] = {0.0};
    c.fill(3, beta, two ? 1 : 0);
    c.product([&](int i, double vi) {
      c.publish(4, i, vi);
      d1[0] += c.rh(i) * vi;
    });
    if (!c.template sum<1>(0, d1)) {
      late = true;
      break;
    }
    if (d1[0] == 0.0 || !isfinite(d1[0])) {
      done = 1;
      status = isfinite(d1[0]) ? 2 : 3;
      break;
    }
    const double al = rho / d1[0];
    if (!(fabs(al) < a.alpha_max)) {  // (rh, v) ~ 0: the step would overflow
      done = 1;
      status = 2;
      break;
    }
    alpha = al;
    if (two) {
      const double* gr = c.global(1);
      late = !c.correct(2, [&](int i) { return c.row_of(1, gr, i) - alpha * c.row_of(4, a.v, i); }, nullptr);
      if (late || !c.barrier()) {
        late = true;
        break;
      }
    }
    // t = A sh ; t . s, t . t
    double d2[2] = {0.0, 0.0};
    c.fill(4, -alpha, two ? 2 : 0);
    c.product([&](int i, double ti) {
      c.t(i) = ti;
      if constexpr (!CL)
        if (two) a.t[r0 + i] = ti;
      d2[0] += ti * (c.r(i) - alpha * c.v(i));
      d2[1] += ti * ti;
    });
    if (!c.template sum<2>(1, d2)) {
      late = true;
      break;
    }
    omega = d2[1] != 0.0 ? d2[0] / d2[1] : 0.0;
    if (!isfinite(omega)) {
      done = 1;
      status = 3;
      break;
    }
    // t.s = 0 with t != 0: the next beta would divide by omega (breakdown);
    // x still advances by alpha ph before stopping
    if (omega == 0.0 && d2[1] != 0.0) status = 2;
    // x, r and the next q; r . r and rh . r.  Grid form, two-level: the aggregates'
    // sums of r and q from what was published before the last barrier (so r and q
    // alternate between two copies), which saves a barrier after this update
    double d3[2] = {0.0, 0.0};
    if constexpr (!CL) {
      if (two) {
        const double *gr = c.global(1), *gq = c.global(3);
        c.template restrict_rows<2>([&](int i, double (&s)[2]) {
          const double ri = __ldcg(gr + i), qi = __ldcg(gq + i), vi = __ldcg(a.v + i), ti = __ldcg(a.t + i);
          const double pi = ri + beta * qi, si = ri - alpha * vi;
          s[0] = si - omega * ti;
          s[1] = pi - omega * vi;
        });
      }
      c.par ^= 1;
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < nr; i += kThreads) {
      const double ri = c.r(i), qi = c.q(i), vi = c.v(i), di = c.dinv(i);
      const double pi = ri + beta * qi, si = ri - alpha * vi;
      double phi = di * pi, shi = di * si;
      if (two && (NEQ == 1 || i % NEQ == NEQ - 1)) {
        const int g = c.tagg()[c.u0 + i / NEQ];
        if (g >= 0) {
          phi += c.near_y(1)[g];
          shi += c.near_y(2)[g];
        }
      }
      c.x(i) += alpha * phi + omega * shi;
      const double rn = si - omega * c.t(i);
      c.publish(1, i, rn);
      c.publish(3, i, pi - omega * vi);
      d3[0] += rn * rn;
      d3[1] += c.rh(i) * rn;
    }
    if (!c.template sum<2>(3, d3)) {
      late = true;
      break;
    }
    rr = d3[0];
    beta = (d3[1] / rho) * (alpha / omega);
    rho = d3[1];
    ++count;
    if (status == 2) {
      done = 1;
    } else if (!isfinite(rr) || !isfinite(rho)) {
      done = 1;
      status = 3;
    } else if (within(rr, limit)) {
      done = 1;
    } else if (rho == 0.0) {
      done = 1;
      status = 2;
    } else if (count >= a.maxit) {
      done = 1;
      status = 1;
    }
  }
  for (int i = threadIdx.x; i < nr; i += kThreads) {
    a.x[r0 + i] = c.x(i);
    if (!done) {
      a.rh[r0 + i] = c.rh(i);
      a.r[r0 + i] = c.r(i);
      a.q[r0 + i] = c.q(i);
    }
  }
  double tr = rr;
  if (done && !fresh && !late) late = !final_residual(c, tr);
  if (rank == 0 && threadIdx.x == 0) {
    a.dctl[kEst] = sqrt(rr);
    a.dctl[kRho] = rho;
    a.dctl[kHnext] = beta;
    if (done && !late) a.dctl[kTrue] = sqrt(tr);
    a.ictl[2] = status;
    a.ictl[3] = count;
    a.ictl[0] = done && !late;
  }
  if (late && threadIdx.x == 0) a.ictl[kFlagLate] = 1;
  if constexpr (CL) cluster_sync();  // no block leaves while another may read its shared memory
}

template <int NEQ, typename MT, bool CL>
__device__ __forceinline__ void cg_body(const PersistSolve& a, Shared& sh, int smem_bytes, int rank, int blocks,
                                        bool first, int iters) {
  if (!first && (a.ictl[0] || a.ictl[kFlagLate])) return;
  Ctx<NEQ, MT, CL> c{a, sh, rank, blocks};
  setup(c, smem_bytes);
  const int nr = c.rows(), r0 = c.n0 * NEQ;
  const bool two = a.nc > 0;
  int done = 0, status = 0, count = 0;
  double rho, beta = 0.0, rr, limit;
  bool late = false, fresh = false;
  // y = Ac^-1 R^T r (z = D^-1 r + y[aggregate] is formed where it is read);
  // r . z = r . D^-1 r + c . y
  // (c: the restriction is there already)
  auto coarse = [&](double rz, bool c_ready) {
    double d[1] = {0.0};
    if (!c_ready) late = !c.correct(1, [&](int i) { return c.row_of(1, c.global(1), i); }, d);
    else c.template coarse_product<false>(1, 0.0, d);
    if (late || !c.template sum<1>(6, d)) late = true;
    return rz + d[0];
  };
  if (first) {
    double w[3];
    late = !begin(c, w, false);
    rr = w[0];
    rho = w[2];
    const double bnorm = sqrt(w[1]);
    limit = a.tol * bnorm;
    if (two && !late) rho = coarse(rho, false);
    done = (sqrt(rr) <= limit || bnorm == 0.0) ? 1 : 0;
    if (!isfinite(rr)) {
      done = 1;
      status = 3;
    }
    fresh = done != 0;
    if (bnorm == 0.0)
      for (int i = threadIdx.x; i < nr; i += kThreads) c.x(i) = 0.0;
    if (rank == 0 && threadIdx.x == 0) {
      a.dctl[kBnorm] = bnorm;
      a.dctl[kBeta] = sqrt(rr);
    }
  } else {
    rho = a.dctl[kRho];
    beta = a.dctl[kOmega];
    limit = a.tol * a.dctl[kBnorm];
    rr = 0.0;
    status = a.ictl[2];
    count = a.ictl[3];
    for (int i = threadIdx.x; i < nr; i += kThreads) {
      c.r(i) = a.r[r0 + i];
      c.q(i) = a.q[r0 + i];
      c.v(i) = a.v[r0 + i];
    }
    if (!late) late = !c.barrier();
    if (two && !late) coarse(0.0, false);  // y of the interrupted iteration
  }
#pragma unroll 1
  for (int it = 0; it < iters && !done && !late; ++it) {
    const int kp = (count & 1) ? 4 : 3, kn = (count & 1) ? 3 : 4;  // the direction's old and new place
    // t = A p with p = z + beta p ; p . t
    double d1[1] = {0.0};
    c.fill(kp, beta, two ? 1 : 0, true);
    const double* p = c.u() + c.u0 * NEQ;  // the block's own rows of the operand
    c.product([&](int i, double ti) {
      const double pi = p[i];
      c.publish(kn, i, pi);
      c.t(i) = ti;
      if constexpr (!CL)
        if (two) a.t[r0 + i] = ti;
      d1[0] += pi * ti;
    });
    if (!c.template sum<1>(0, d1)) {
      late = true;
      break;
    }
    if (!isfinite(d1[0]) || !(d1[0] > 0.0)) {  // a non-positive p . A p stops the solve (not SPD)
      done = 1;
      status = isfinite(d1[0]) ? 2 : 3;
      break;
    }
    const double alpha = rho / d1[0];
    double d2[2] = {0.0, 0.0};
    const double* pn = c.vec(kn);
    if constexpr (!CL) {  // the aggregates' sums of the new r, as in BiCGStab
      if (two) {
        const double* gr = c.global(1);
        c.template restrict_rows<1>([&](int i, double (&s)[1]) { s[0] = __ldcg(gr + i) - alpha * __ldcg(a.t + i); });
      }
      c.par ^= 1;
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < nr; i += kThreads) {
      c.x(i) += alpha * pn[i];
      const double ri = c.r(i) - alpha * c.t(i);
      c.publish(1, i, ri);
      d2[0] += ri * ri;
      d2[1] += ri * (c.dinv(i) * ri);
    }
    if (!c.template sum<2>(1, d2)) {
      late = true;
      break;
    }
    rr = d2[0];
    ++count;
    const bool conv = within(rr, limit);
    double rho_new = d2[1];
    if (two && isfinite(rr) && !conv) {
      rho_new = coarse(rho_new, !CL);
      if (late) break;
    }
    beta = rho_new / rho;
    rho = rho_new;
    if (!isfinite(rr) || !isfinite(rho_new)) {
      done = 1;
      status = 3;
    } else if (conv) {
      done = 1;
    } else if (!(rho_new > 0.0)) {  // indefinite preconditioner or exact breakdown
      done = 1;
      status = 2;
    } else if (count >= a.maxit) {
      done = 1;
      status = 1;
    }
  }
  for (int i = threadIdx.x; i < nr; i += kThreads) {
    a.x[r0 + i] = c.x(i);
    if (!done) {
      a.r[r0 + i] = c.r(i);
      if constexpr (CL) {
        a.q[r0 + i] = c.q(i);
        a.v[r0 + i] = c.v(i);
      }
    }
  }
  double tr = rr;
  if (done && !fresh && !late) late = !final_residual(c, tr);
  if (rank == 0 && threadIdx.x == 0) {
    a.dctl[kEst] = sqrt(rr);
    a.dctl[kRho] = rho;
    a.dctl[kOmega] = beta;
    if (done && !late) a.dctl[kTrue] = sqrt(tr);
    a.ictl[2] = status;
    a.ictl[3] = count;
    a.ictl[0] = done && !late;
  }
  if (late && threadIdx.x == 0) a.ictl[kFlagLate] = 1;
  if constexpr (CL) cluster_sync();
}

template <bool CG, int NEQ, typename MT, bool CL>
__global__ void __launch_bounds__(kThreads, 1)
    persist_kernel(const __grid_constant__ PersistSolve a, int smem_bytes, int first, int iters) {
  __shared__ Shared sh;
  if constexpr (CG)
    cg_body<NEQ, MT, CL>(a, sh, smem_bytes, int(blockIdx.x), int(gridDim.x), first != 0, iters);
  else
    bicgstab_body<NEQ, MT, CL>(a, sh, smem_bytes, int(blockIdx.x), int(gridDim.x), first != 0, iters);
}

// One cluster per solve of a list (the members of a batch): cluster k runs solve k,
// with its arguments copied to shared memory (kernel arguments would be indexed by k).
template <int NEQ, typename MT>
__global__ void __launch_bounds__(kThreads, 1)
    persist_members_kernel(const PersistSolve* __restrict__ list, int blocks, int smem_bytes, int iters) {
  __shared__ Shared sh;
  __shared__ PersistSolve a;
  static_assert(sizeof(PersistSolve) % 8 == 0, "copied in 8-byte words");
  const int k = int(blockIdx.x) / blocks;
  for (int q = threadIdx.x; q < int(sizeof(PersistSolve) / 8); q += kThreads)
    reinterpret_cast<unsigned long long*>(&a)[q] = __ldg(reinterpret_cast<const unsigned long long*>(list + k) + q);
  __syncthreads();
  bicgstab_body<NEQ, MT, true>(a, sh, smem_bytes, int(blockIdx.x) - k * blocks, blocks, true, iters);
}

constexpr size_t kSmemMax = 224 * 1024;  // dynamic shared memory of a block (227 KB less the static part)

template <bool CG, int NEQ, typename MT, bool CL>
int launch(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s) {
  auto kernel = persist_kernel<CG, NEQ, MT, CL>;
  UFEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax)));
  if (CL) {
    UFEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  // the barrier counter of every launch; a late barrier stays on record to the solve's end
  if (first) UFEM_CUDA_TRY(cudaMemsetAsync(a.ictl + kFlagLate, 0, 2 * sizeof(int), s));
  if (!CL && (!first || a.stuck))
    UFEM_CUDA_TRY(cudaMemsetAsync(a.ictl + kFlagBarrier, a.stuck ? 0xff : 0, sizeof(int), s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(plan.blocks));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  if (CL) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(plan.blocks);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  UFEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a, int(plan.smem), first ? 1 : 0, iters));
  return UFEM_OK;
}

template <int NEQ, typename MT>
int launch_members(const PersistSolve* list, int count, int blocks, size_t smem, int iters, cudaStream_t s) {
  auto kernel = persist_members_kernel<NEQ, MT>;
  UFEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax)));
  UFEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(count) * unsigned(blocks));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(blocks);
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  UFEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, list, blocks, int(smem), iters));
  return UFEM_OK;
}

template <bool CG, int NEQ>
int launch_n(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s) {
  if (plan.form == kPersistCluster)
    return a.f32 ? launch<CG, NEQ, float, true>(a, plan, first, iters, s)
                 : launch<CG, NEQ, double, true>(a, plan, first, iters, s);
  return a.f32 ? launch<CG, NEQ, float, false>(a, plan, first, iters, s)
               : launch<CG, NEQ, double, false>(a, plan, first, iters, s);
}

template <bool CG>
int launch_any(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s) {
  switch (a.neq) {
    case 1: return launch_n<CG, 1>(a, plan, first, iters, s);
    case 2: return launch_n<CG, 2>(a, plan, first, iters, s);
    case 3: return launch_n<CG, 3>(a, plan, first, iters, s);
    default: return launch_n<CG, 4>(a, plan, first, iters, s);
  }
}

}  // namespace

// Whether the device can run a cluster of C blocks (a part of one may not hold 16 SMs that
// share a cluster); every kernel of the cluster form needs the same of it.
static bool cluster_runs(int C, size_t smem) {
  auto kernel = persist_kernel<false, 4, double, true>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax)) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(C));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(C);
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  return cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
}

// start_h, adj_h: the node graph on the host; nc: aggregates of the coarse space.
static PersistPlan persist_plan(const int64_t* start_h, const int32_t* adj_h, int64_t N, int neq, bool f32, int nc) {
  PersistPlan p;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return p;
  // Above 96 MB of values the matrix no longer stays in L2 beside the rest, and the
  // multi-launch products, with more loads in flight, make up for their launches.
  // Tetrahedra in natural order, point Jacobi, us an iteration (launches / one): 36^3 x 6
  // (89 MB) 60.5 / 43.9, 37^3 (96.3 MB) 61.4 / 54.8, 38^3 (104 MB) 64.3 / 65.1, 40^3
  // (121 MB) 71.8 / 76.4.  Most systems end earlier, where a block's vectors and lists do
  // not fit (needs, below).
  const int64_t vb = int64_t(neq) * neq * (f32 ? 4 : 8);
  const int npw = 32 / neq, sb = slice_bytes(neq, f32 ? 4 : 8);
  const int64_t bytes = start_h[N] * vb;
  if (bytes > int64_t(96) << 20 || N * neq > INT32_MAX / 2) return p;
  std::vector<int32_t> stamp;
  // Shared memory the widest of G blocks needs (cluster: with its values); 0 if that is more than a block has.
  auto needs = [&](int G, bool cluster) -> size_t {
    const int64_t wide = (N + G - 1) / G;
    if (size_t(start_h[N] / G) * 2 + bitmap_bytes(N) > kSmemMax) return 0;
    if (stamp.empty()) stamp.assign(size_t(N), -1);
    std::fill(stamp.begin(), stamp.end(), -1);
    size_t most = 0;
    for (int b = 0; b < G; ++b) {
      const int64_t n0 = N * b / G, n1 = N * (b + 1) / G, e0 = start_h[n0], e1 = start_h[n1];
      int64_t U = 0;
      for (int64_t k = e0; k < e1; ++k)
        if (stamp[size_t(adj_h[k])] != b) {
          stamp[size_t(adj_h[k])] = b;
          ++U;
        }
      if (U > 65535) return 0;
      const Layout l = layout(uniform_bytes((cluster ? wide : n1 - n0) * neq, cluster, nc), n1 - n0, e1 - e0, U,
                              neq, nc, cluster, G);
      size_t values = 0;
      for (int64_t i = n0; cluster && i < n1; i += npw) {
        int64_t width = 0;
        for (int64_t k = i; k < std::min(n1, i + npw); ++k) width = std::max(width, start_h[k + 1] - start_h[k]);
        values += size_t(width) * sb;
      }
      most = std::max({most, align16(l.vals + values), l.u + bitmap_bytes(N)});
      if (most > kSmemMax) return 0;
    }
    return most;
  };
  const int64_t per = neq == 4 ? kWarps : kThreads / 8;  // nodes a block takes at once
  // one cluster: the fewest blocks that hold the system, and not fewer than its
  // nodes can use (two rounds of a block's groups)
  for (int C = 1; C <= kClusterMax; C *= 2) {
    if (C < kClusterMax && N > int64_t(C) * per * 2) continue;
    if (size_t(bytes / C) > kSmemMax) continue;
    if (const size_t s = needs(C, true)) {
      if (!cluster_runs(C, s)) continue;
      p.form = kPersistCluster;
      p.blocks = C;
      p.smem = s;
      return p;
    }
  }
  const int G = int(std::max<int64_t>(1, std::min<int64_t>({(N + per - 1) / per, sms, kPersistMaxBlocks})));
  if (needs(G, false)) {
    p.form = kPersistGrid;
    p.blocks = G;
    p.smem = kSmemMax;  // what the lists and vectors leave holds values
  }
  return p;
}

const PersistPlan& persist_plan_of(ufem_ns_handle* h, bool f32, int nc) {
  PersistPlan& p = h->pplan[f32][nc > 0];
  int& planned = h->pplan_nc[f32][nc > 0];
  if (planned != nc) {
    p = persist_plan(h->start_h.data(), h->adj_h.data(), h->N, h->neq, f32, nc);
    planned = nc;
  }
  return p;
}

int persist_bicgstab_members(const PersistSolve* d_list, int count, int neq, bool f32, int blocks, size_t smem,
                             int iters, cudaStream_t s) {
  if (neq == 3)
    return f32 ? launch_members<3, float>(d_list, count, blocks, smem, iters, s)
               : launch_members<3, double>(d_list, count, blocks, smem, iters, s);
  return f32 ? launch_members<4, float>(d_list, count, blocks, smem, iters, s)
             : launch_members<4, double>(d_list, count, blocks, smem, iters, s);
}

int persist_bicgstab(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s) {
  return launch_any<false>(a, plan, first, iters, s);
}
int persist_cg(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s) {
  return launch_any<true>(a, plan, first, iters, s);
}

}  // namespace ufem
