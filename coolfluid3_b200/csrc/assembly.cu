// assembly.cu -- sm_100a kernels of the UFEM Navier-Stokes step, except the Krylov solve.
//
// Row-owner assembly.  The reference loops over elements and adds each element
// matrix into the FEVbr block rows it touches (Proto/ElementLooper.hpp:173-179,
// TrilinosFEVbrMatrix.cpp:271-357).  Here every CTA owns a contiguous range of
// CSR block rows ("chunk").  Phase 1: one thread per incidence (row node i,
// element e containing i at local position a) gathers the element's nodal data,
// evaluates the element's row block a -- the neq x (n*neq) slice of
// invdt*T + theta*A and the neq entries of -A*x + a -- and stages it in shared
// memory.  Phase 2: one thread per (row, neighbour slot, equation) sums the
// staged contributions of the row's incidences in ascending element order (the
// order in which the reference adds them; the warp kernel's tetrahedra: another
// fixed order of the row's elements) and writes each CSR value exactly
// once, coalesced.  No floating-point atomics, no element matrices in HBM.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "internal.h"
#include "dirichlet.cuh"
#include "element.cuh"

namespace ufem {
namespace {

// ---------------------------------------------------------------------------
// Element row blocks.  For the row node (relabelled to local position 0) the
// neq x (n neq) slice of invdt T + theta A has the same structure in the generic
// (NavierStokesAssembly.hpp:51-67) and the specialised element forms
// (NavierStokesSpecializations.hpp:37-302): with G_b the shape-function gradients,
//   [u_i, u_j b] = tg_i G_jb + delta_ij diag_b     [u_i, p b] = thS G_ib
//   [p,   u_j b] = sWSp G_jb + c_j vem_b            [p,   p b] = dd_b
// so a row block is its head (tg, thS, sWSp, c: 2 D + 2 numbers) and a column of
// D + 3 numbers per node.  The routine hands exactly these to a sink: the warp
// kernel stages them (36 numbers a tetrahedron where the expanded block has 68)
// and multiplies them out while it sums, the chunk kernel expands them, the
// residual kernel applies them to the increment.
//
// The generic form's order-2 Gauss sums (Proto/ElementIntegration.hpp:236-258)
// are taken in closed form: on P1 elements every integrand is a polynomial of
// degree <= 2 in the barycentric coordinates, which that rule integrates exactly:
//   int N_k = m1 = V/n,   int N_k N_l = m2 (1 + d_kl),   m2 = V/(n(n+1)),
// and with alpha_b = ubar . G_b, c_0b = U_0 . G_b, w_b = U_b . G_0, q = sum_k w_k U_k:
//   int N_0 adv_b = m2 (n alpha_b + c_0b)   int adv_0 adv_b = m2 (n^2 alpha_0 alpha_b + q . G_b)
//   int adv_0 N_b = m2 (n alpha_0 + w_b)    int ua_i S_0 = m2 (n ubar_i + U_0i) + tau m2 (n^2 ubar_i alpha_0 + q_i)
// The specialised forms are written with normals n_b = D V G_b; here their terms
// are collected on G_b, including the tetrahedra's use of v where w is meant
// (:224-226, :236-238), and tau comes from the nodal solution with the standard
// constants (a default ComputeTauImpl).
// ---------------------------------------------------------------------------

// Sink of the warp kernel: the record of one incidence in shared memory.
// Tetrahedra: [tg, thS][columns of nodes 1..3: G, diag, p row][diagonal block and
// RHS row]; the column of the row node is multiplied out here, since the diagonal
// block takes it from every incidence, and so is each column's p row (6 loads of 16
// bytes a contributor instead of 7).  Triangles: the expanded row block and the RHS row (an edge has
// two elements at most, so multiplying out while summing would cost more loads than
// it saves).
template <int D, typename T>
struct RecordLayout {
  static constexpr int n = D + 1, neq = D + 1;
  static constexpr int head = D + 1;        // 3D: tg, thS
  static constexpr int col = 2 * D + 2;     // 3D: G, diag, p row
  static constexpr int sums = D == 3 ? head + D * col : n * neq * neq;  // 3D: diagonal block, rhs; 2D: rhs
  // Lane pitch: 16-byte records whose quarter-warp accesses hit distinct banks
  // (3D: 400 B and 208 B, odd multiples of 16), odd for the scalar accesses of 2D.
  static constexpr int pitch = D == 3 ? (sizeof(T) == 8 ? 50 : 52) : 31;
};
template <int D, typename T>
struct RecordSink;
template <typename T>
struct RecordSink<3, T> {
  using L = RecordLayout<3, T>;
  T* __restrict__ rec;
  T tg[3], thS, sWSp, c[3];
  __device__ __forceinline__ void put2(int at, T a, T b) {
    if constexpr (std::is_same<T, float>::value) *reinterpret_cast<float2*>(rec + at) = make_float2(a, b);
    else *reinterpret_cast<double2*>(rec + at) = make_double2(a, b);
  }
  __device__ __forceinline__ void head(const T (&tg_)[3], T thS_, T sWSp_, const T (&c_)[3]) {
    put2(0, tg_[0], tg_[1]);
    put2(2, tg_[2], thS_);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      tg[k] = tg_[k];
      c[k] = c_[k];
    }
    thS = thS_;
    sWSp = sWSp_;
  }
  __device__ __forceinline__ void col(int b, const T (&g)[3], T diag, T vem, T dd) {
    const T p0 = sWSp * g[0] + c[0] * vem, p1 = sWSp * g[1] + c[1] * vem, p2 = sWSp * g[2] + c[2] * vem;
    if (b == 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        put2(L::sums + 4 * i, tg[i] * g[0] + (i == 0 ? diag : T(0)), tg[i] * g[1] + (i == 1 ? diag : T(0)));
        put2(L::sums + 4 * i + 2, tg[i] * g[2] + (i == 2 ? diag : T(0)), thS * g[i]);
      }
      put2(L::sums + 12, p0, p1);
      put2(L::sums + 14, p2, dd);
      return;
    }
    const int at = L::head + (b - 1) * L::col;
    put2(at, g[0], g[1]);
    put2(at + 2, g[2], diag);
    put2(at + 4, p0, p1);
    put2(at + 6, p2, dd);
  }
  __device__ __forceinline__ void rhs(const T (&r)[4]) {
    put2(L::sums + 16, r[0], r[1]);
    put2(L::sums + 18, r[2], r[3]);
  }
};

// Sink of the chunk kernel: the expanded block and the RHS row, value-major with
// pitch CH.
template <int D, typename T>
struct StageSink {
  T* __restrict__ st;
  T* __restrict__ rst;
  int CH;
  T tg[D], thS, sWSp, c[D];
  __device__ __forceinline__ void head(const T (&tg_)[D], T thS_, T sWSp_, const T (&c_)[D]) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      tg[k] = tg_[k];
      c[k] = c_[k];
    }
    thS = thS_;
    sWSp = sWSp_;
  }
  __device__ __forceinline__ void col(int b, const T (&g)[D], T diag, T vem, T dd) {
    constexpr int neq = D + 1;
    T* __restrict__ o = st + b * neq * neq * CH;
#pragma unroll
    for (int i = 0; i < D; ++i) {
#pragma unroll
      for (int j = 0; j < D; ++j) o[(i * neq + j) * CH] = tg[i] * g[j] + (i == j ? diag : T(0));
      o[(i * neq + D) * CH] = g[i] * thS;
    }
#pragma unroll
    for (int j = 0; j < D; ++j) o[(D * neq + j) * CH] = g[j] * sWSp + c[j] * vem;
    o[(D * neq + D) * CH] = dd;
  }
  __device__ __forceinline__ void rhs(const T (&r)[D + 1]) {
#pragma unroll
    for (int k = 0; k <= D; ++k) rst[k * CH] = r[k];
  }
};

template <typename T>
struct RecordSink<2, T> : StageSink<2, T> {
  __device__ __forceinline__ explicit RecordSink(T* rec) {
    this->st = rec;
    this->rst = rec + RecordLayout<2, T>::sums;
    this->CH = 1;
  }
};

template <int D, typename T>
__device__ __forceinline__ void load_state(const NodeData& nd, int node, T (&x)[D + 1]) {
  double s[4];
  ld4(nd.state + 4ll * node, s[0], s[1], s[2], s[3]);
#pragma unroll
  for (int k = 0; k <= D; ++k) x[k] = T(s[k]);
}

// The original local node at relabelled position b (row node a at position 0).
template <int D>
__device__ __forceinline__ int original_node(int b, int a) {
  return D == 3 ? (b ^ a) : (b + a >= 3 ? b + a - 3 : b + a);
}

// Gradients of the relabelled nodes, element volume, and the METRIC tau's sums
// over g = J^-T J^-1 of the element's own frame: sq = sum g_mq^2, itr = 1 / tr g.
template <int D, typename T>
struct ElemGeo {
  T G[D + 1][D];
  T V, sq, itr;
};

// From the coordinates, in relabelled order.
template <int D, typename T>
__device__ __forceinline__ void compute_geometry(const Elem<D, T>& el, int a, ElemGeo<D, T>& g) {
  T J[D][D], Ji[D][D], det;
#pragma unroll
  for (int r = 0; r < D; ++r)
#pragma unroll
    for (int c = 0; c < D; ++c) J[r][c] = el.Xr[r + 1][c];
  inverse_det<T>(J, Ji, det);
  T G[D][D + 1];
#pragma unroll
  for (int r = 0; r < D; ++r) {
    T s = -Ji[r][0];
#pragma unroll
    for (int k = 1; k < D; ++k) s -= Ji[r][k];
    G[r][0] = s;
#pragma unroll
    for (int b = 1; b <= D; ++b) G[r][b] = Ji[r][b - 1];
  }
  T m[D][D];
  metric_tensor<D, T>(G, a, m);
  T sq = 0, tr = 0;
#pragma unroll
  for (int i = 0; i < D; ++i) {
    tr += m[i][i];
#pragma unroll
    for (int j = 0; j < D; ++j) sq += m[i][j] * m[i][j];
  }
#pragma unroll
  for (int b = 0; b <= D; ++b)
#pragma unroll
    for (int k = 0; k < D; ++k) g.G[b][k] = G[k][b];
  g.V = det * T(D == 2 ? 0.5 : 1.0 / 6.0);
  g.sq = sq;
  g.itr = trcp(tr);
}

// tau of METRIC (SUPG.hpp:176-199): adv = | sum_m u_m grad xi_m |^2 with grad xi_m the
// gradient of original node m + 1.
template <int D, typename T>
__device__ __forceinline__ void metric_tau(const KParams<T>& kp, bool standard, const ElemGeo<D, T>& g, int a,
                                           const T (&uc)[D], T nu, T& tsu, T& tbu) {
  T u4[D + 1];
  u4[0] = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) u4[k + 1] = uc[k];
  T co[D + 1];  // u_m at the relabelled position of original node m + 1
  if constexpr (D == 3) {
    const bool x1 = (a & 1) != 0, x2 = (a & 2) != 0;
    const T p0 = x1 ? u4[1] : u4[0], p1 = x1 ? u4[0] : u4[1], p2 = x1 ? u4[3] : u4[2], p3 = x1 ? u4[2] : u4[3];
    co[0] = x2 ? p2 : p0;
    co[1] = x2 ? p3 : p1;
    co[2] = x2 ? p0 : p2;
    co[3] = x2 ? p1 : p3;
  } else {
#pragma unroll
    for (int b = 0; b < 3; ++b) co[b] = sel<3>(u4, original_node<2>(b, a));
  }
  T adv = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    T s = 0;
#pragma unroll
    for (int b = 0; b <= D; ++b) s += co[b] * g.G[b][k];
    adv += s * s;
  }
  const T diff = nu * nu * g.sq;
  const T xs = kp.tau_std + adv + T(16) * diff;
  const T rs = trsqrt(xs);
  tbu = xs * rs * g.itr;  // sqrt(xs) / tr g
  if (standard || (kp.tau_c1 == kp.tau_std && kp.c2 == T(16))) tsu = rs;  // the same argument
  else tsu = trsqrt(kp.tau_c1 + adv + kp.c2 * diff);
}

// The row block of an element (nodes ids, relabelled) for its node at position 0
// (original local node a).  GEN: any tau; otherwise METRIC.  The geometry is formed
// anew for each of the element's rows: reading it from static records (128 B a
// tetrahedron) took as long, since a scattered 128-byte read costs the L1 more
// passes than the coordinates' gather (0.701 against 0.690 ms at 64^3 x 6).
template <int D, typename T, bool SPEC, bool GEN, typename Sink>
__device__ __forceinline__ void element_row(const int (&ids)[4], int a, const NodeData& nd,
                                            const double* __restrict__ force, const KParams<T>& kp, Sink& sk) {
  constexpr int n = D + 1, neq = D + 1;
  const T inv_n = T(1.0 / n), nT = T(n), n2 = T(n * n);
  ElemGeo<D, T> g;
  Elem<D, T> el;
  constexpr bool kEarly = std::is_same<T, float>::value;  // FP32: u_adv and the state share a 32-byte record
  T xe[kEarly ? n : 1][neq];
  if constexpr (kEarly) gather_geometry_node32<D>(ids, nd, el, xe);
  else gather_geometry_uadv<D, T>(ids, nd, el);
  compute_geometry<D, T>(el, a, g);
  auto state = [&](int b, T (&x)[neq]) {
    if constexpr (kEarly) {
#pragma unroll
      for (int k = 0; k < neq; ++k) x[k] = xe[b][k];
    } else {
      load_state<D, T>(nd, ids[b], x);
    }
  };
  T nsum = 0, ub[D];
#pragma unroll
  for (int b = 0; b < n; ++b) nsum += el.NU[b];
  const T nu = tabs(nsum * inv_n);
#pragma unroll
  for (int k = 0; k < D; ++k) {
    T m = 0;
#pragma unroll
    for (int b = 0; b < n; ++b) m += el.U[b][k];
    ub[k] = m * inv_n;
  }
  T tps, tsu, tbu;
  if constexpr (SPEC) {
    T us[D];
#pragma unroll
    for (int k = 0; k < D; ++k) us[k] = 0;
#pragma unroll
    for (int b = 0; b < n; ++b) {
      T x[neq];
      state(b, x);
#pragma unroll
      for (int k = 0; k < D; ++k) us[k] += x[k];
    }
#pragma unroll
    for (int k = 0; k < D; ++k) us[k] *= inv_n;
    metric_tau<D, T>(kp, true, g, a, us, nu, tsu, tbu);
    tps = tsu;
  } else {
    if (!GEN || kp.supg_type == 1) {
      metric_tau<D, T>(kp, false, g, a, ub, nu, tsu, tbu);
      tps = tsu * kp.a_ps;
      tsu *= kp.a_su;
      tbu *= kp.a_bu;
    } else {
      T Gt[D][n], gm[D][D];
#pragma unroll
      for (int k = 0; k < D; ++k) {
#pragma unroll
        for (int b = 0; b < n; ++b) Gt[k][b] = g.G[b][k];
#pragma unroll
        for (int q = 0; q < D; ++q) gm[k][q] = 0;
      }
      compute_tau<D, T>(kp, el, ub, nu, Gt, gm, g.V * T(D == 2 ? 2 : 6), tps, tsu, tbu);
    }
  }
  const T V = g.V, m1 = V * inv_n, m2 = V * T(1.0 / (n * (n + 1)));
  T alpha[n];
#pragma unroll
  for (int b = 0; b < n; ++b) {
    T s = 0;
#pragma unroll
    for (int k = 0; k < D; ++k) s += ub[k] * g.G[b][k];
    alpha[b] = s;
  }
  const T sWS = m1 + tsu * V * alpha[0];
  const T theta = kp.theta, invdt = kp.invdt, inv_rho = kp.inv_rho;
  T gam[D], q[D], w[n], sWSp, ts2 = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) q[k] = 0;
  if constexpr (SPEC) {
    T uw[D], s = 0;
#pragma unroll
    for (int k = 0; k < D; ++k) uw[k] = ub[D == 3 && k == 2 ? 1 : k];
#pragma unroll
    for (int k = 0; k < D; ++k) s += uw[k] * g.G[0][k];
    sWSp = m1 + T(0.5) * tps * V * s;
    const T fu = T(0.5) * sWS, fn = (nu * T(1. / 3.) + tbu) * V;
#pragma unroll
    for (int k = 0; k < D; ++k) gam[k] = fu * uw[k] + fn * g.G[0][k];
  } else {
    ts2 = tsu * m2;
    sWSp = m1 + T(0.5) * tps * V * alpha[0];
#pragma unroll
    for (int b = 0; b < n; ++b) {
      T s = 0;
#pragma unroll
      for (int k = 0; k < D; ++k) s += el.U[b][k] * g.G[0][k];
      w[b] = s;
#pragma unroll
      for (int k = 0; k < D; ++k) q[k] += s * el.U[b][k];
    }
    const T na = n2 * alpha[0];
#pragma unroll
    for (int k = 0; k < D; ++k)
      gam[k] = tbu * V * g.G[0][k] + T(0.5) * (m2 * (nT * ub[k] + el.U[0][k]) + ts2 * (na * ub[k] + q[k]));
  }
  T au[D];
#pragma unroll
  for (int k = 0; k < D; ++k) au[k] = 0;
  if (!SPEC && kp.has_force) {
    T F[n][D];
#pragma unroll
    for (int b = 0; b < n; ++b) {
      double f[4];
      ld4(force + 4ll * ids[b], f[0], f[1], f[2], f[3]);
#pragma unroll
      for (int k = 0; k < D; ++k) F[b][k] = T(f[k]);
    }
#pragma unroll
    for (int i = 0; i < D; ++i) {
      T gs = 0, gw = 0;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        gs += F[k][i];
        gw += w[k] * F[k][i];
      }
      const T gbar = gs * inv_n;
      au[i] = m2 * (nT * gbar + F[0][i]) + ts2 * (n2 * gbar * alpha[0] + gw);
    }
  }
  {
    T tg[D], cj[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      tg[k] = theta * gam[k];
      cj[k] = tps * g.G[0][k];
    }
    sk.head(tg, theta * sWS * inv_rho, sWSp, cj);
  }
  const T tpv = tps * inv_rho * V, em = invdt * m1;
  const T tw = SPEC ? invdt * (m2 + tsu * m1 * alpha[0]) : T(0);  // specialised: T_b of b > 0
  T div = 0, gradp[D], kx[D], ga = 0, pp = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) gradp[k] = kx[k] = 0;
#pragma unroll
  for (int b = 0; b < n; ++b) {
    T x[neq], d0 = 0, gx = 0;  // x: nodal state (u, p)
    state(b, x);
#pragma unroll
    for (int k = 0; k < D; ++k) d0 += g.G[0][k] * g.G[b][k];
    const T vab = V * alpha[b];
    T K, diag;
    if constexpr (SPEC) {
      K = alpha[b] * sWS + nu * V * d0;
      diag = theta * K + tw + (b == 0 ? invdt * m2 : T(0));
    } else {
      T c0 = 0, qg = 0;
#pragma unroll
      for (int k = 0; k < D; ++k) {
        c0 += el.U[0][k] * g.G[b][k];
        qg += q[k] * g.G[b][k];
      }
      K = nu * V * d0 + m2 * (nT * alpha[b] + c0) + ts2 * (n2 * alpha[0] * alpha[b] + qg);
      diag = theta * K + invdt * (m2 * (b == 0 ? T(2) : T(1)) + ts2 * (nT * alpha[0] + w[b]));
    }
    const T dd = d0 * tpv;
    sk.col(b, g.G[b], diag, vab + em, dd);
    // pieces of A x (A before the theta combination)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      div += g.G[b][k] * x[k];
      gx += g.G[0][k] * x[k];
      gradp[k] += g.G[b][k] * x[D];
      kx[k] += K * x[k];
    }
    ga += vab * gx;
    pp += dd * x[D];
  }
  T r[neq];
#pragma unroll
  for (int k = 0; k < D; ++k) r[k] = au[k] - (kx[k] + gam[k] * div + sWS * inv_rho * gradp[k]);
  r[D] = -(sWSp * div + tps * ga + pp);
  sk.rhs(r);
}

// The warp kernel's static lists.  Per incidence: its element and original local
// node (element | a << 30).  Per off-diagonal slot of a row with at most 32
// incidences, in CSR order: one 64-bit word with up to 7 contributors (5 bits: the
// incidence's place in its row, 2 bits: the slot's position in its element), ascending
// element; bits 49-51 their number, 52-57 the slot, 58-62 the row modulo 32.  With
// more contributors bit 63 is set and the low words are a place in `over` (one
// byte a contributor, bits 0-31) and the number (bits 32-39).
template <int D>
__global__ void assembly_items_kernel(int64_t N, const int64_t* __restrict__ start, const int32_t* __restrict__ row_inc,
                                      const int32_t* __restrict__ inc_elem, const uint32_t* __restrict__ inc_info,
                                      uint32_t* __restrict__ inc_ea, unsigned long long* __restrict__ items,
                                      uint8_t* __restrict__ over, unsigned* __restrict__ over_used) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int k0 = row_inc[i], K = row_inc[i + 1] - k0;
  const int64_t s0 = start[i];
  const int S = int(start[i + 1] - s0);
  if (inc_ea)
    for (int k = 0; k < K; ++k) inc_ea[k0 + k] = uint32_t(inc_elem[k0 + k]) | ((inc_info[k0 + k] >> 24) & 3u) << 30;
  if (K < 1 || K > 32) return;
  const uint32_t i0 = inc_info[k0];
  const int self = int((i0 >> (6 * ((i0 >> 24) & 3u))) & 63u);
  for (int s = 0; s < S; ++s) {
    if (s == self) continue;
    unsigned long long word = 0;
    int cnt = 0;
    auto each = [&](auto f) {
      for (int k = 0; k < K; ++k) {
        const uint32_t info = inc_info[k0 + k];
        const int a = int(info >> 24) & 3;
        for (int q = 0; q <= D; ++q)
          if (q != a && int((info >> (6 * q)) & 63u) == s) f(k, D == 3 ? (q ^ a) : (q - a + 3) % 3);
      }
    };
    each([&](int k, int b) {
      if (cnt < 7) word |= (unsigned long long)(k * 4 + b) << (7 * cnt);
      ++cnt;
    });
    if (cnt <= 7) {
      word |= (unsigned long long)cnt << 49;
    } else {
      const unsigned at = atomicAdd(over_used, unsigned(cnt));
      word = (unsigned long long)at | (unsigned long long)cnt << 32 | 1ull << 63;
      if (over) {
        unsigned p = at;
        each([&](int k, int b) { over[p++] = uint8_t(k * 4 + b); });
      }
    }
    word |= (unsigned long long)s << 52 | (unsigned long long)(i & 31) << 58;
    if (items) items[s0 - i + s - (s > self ? 1 : 0)] = word;
  }
}

// Shared memory of one chunk: staged row blocks [value][incidence] (T), staged
// RHS rows, the permuted slot word of every incidence, per-row offsets, and one
// 64-bit contributor mask per (row, neighbour slot).
template <int D, typename T, int CH>
constexpr size_t assembly_smem_bytes() {
  return size_t(P1<D>::nvals + P1<D>::neq) * CH * sizeof(T) +  // st, rst
         size_t(CH) * 8 +                                     // s_mask (sum of row slots <= CH)
         size_t(CH) * 4 +                                     // s_info
         size_t(5 * CH + 3) * 4;                              // s_rowinc, s_pref, s_spref, s_slots, s_self
}

// The row-owner assembly kernel.  One CTA per chunk of whole block rows.
template <int D, typename T, int CH, bool SPEC, bool GEN>
__global__ void __launch_bounds__(CH) ns_assembly_kernel(
    const int2* __restrict__ chunk_rows, const int32_t* __restrict__ row_inc,
    const int32_t* __restrict__ inc_elem, const uint32_t* __restrict__ inc_info, const int4* __restrict__ conn,
    const double* __restrict__ coords, const double* __restrict__ uadv, const double* __restrict__ state,
    const float* __restrict__ node32, const double* __restrict__ force, const int64_t* __restrict__ start,
    NSParams p, double* __restrict__ vals,
    float* __restrict__ vals32, double* __restrict__ rhs) {
  constexpr int n = P1<D>::n, neq = P1<D>::neq, nvals = P1<D>::nvals;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* st = reinterpret_cast<T*>(smem_raw);
  T* rst = st + nvals * CH;
  unsigned long long* s_mask = reinterpret_cast<unsigned long long*>(rst + neq * CH);  // CH
  uint32_t* s_info = reinterpret_cast<uint32_t*>(s_mask + CH);                         // CH
  int* s_rowinc = reinterpret_cast<int*>(s_info + CH);                                 // CH + 1
  int* s_pref = s_rowinc + CH + 1;                                                     // CH + 1
  int* s_spref = s_pref + CH + 1;                                                      // CH + 1
  int* s_slots = s_spref + CH + 1;                                                     // CH
  int* s_self = s_slots + CH;                                                          // CH: slot of the row node

  const int2 cr = chunk_rows[blockIdx.x];
  const int row0 = cr.x, row1 = cr.y;
  const int R = row1 - row0;  // 1 <= R <= K <= CH (every node has an incidence)
  const int inc0 = row_inc[row0];
  const int K = row_inc[row1] - inc0;
  const int t = threadIdx.x;

  // Row metadata and zeroed contributor masks
  for (int rl = t; rl <= R; rl += CH) s_rowinc[rl] = row_inc[row0 + rl] - inc0;
  for (int rl = t; rl < R; rl += CH) s_slots[rl] = int(start[row0 + rl + 1] - start[row0 + rl]);
  for (int k = t; k < CH; k += CH) s_mask[k] = 0ull;
  __syncthreads();
  if (t == 0) {
    int items = 0, slots = 0;
    s_pref[0] = 0;
    s_spref[0] = 0;
    for (int rl = 0; rl < R; ++rl) {
      items += (s_slots[rl] - 1) * neq;  // off-diagonal blocks
      slots += s_slots[rl];
      s_pref[rl + 1] = items;
      s_spref[rl + 1] = slots;
    }
  }
  __syncthreads();

  // Phase 1: element row blocks, one thread per incidence.  The element's
  // nodes are relabelled by the even permutation k -> k ^ a (tetrahedra) or the
  // rotation k -> (k + a) mod 3 (triangles), which brings the row node to local
  // position 0 and leaves det J, the orientation and the symmetric order-2 Gauss
  // rules unchanged; the element routines then see a compile-time row index.
  if (t < K) {
    const int k = inc0 + t;
    const int e = __ldg(inc_elem + k);
    const uint32_t info = __ldg(inc_info + k);
    const int a = int(info >> 24) & 3;
    const int4 cn = __ldg(conn + e);
    const int ids0[4] = {cn.x, cn.y, cn.z, cn.w};
    int ids[4];
    uint32_t pslots = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int src = (D == 3) ? (q ^ a) : (q < 3 ? (q + a) % 3 : 3);
      ids[q] = ids0[src];
      const uint32_t sl = (q < n) ? ((info >> (6 * src)) & 63u) : 0xFFu;
      pslots |= sl << (8 * q);
    }
    s_info[t] = pslots;
    const KParams<T> kp = make_kparams<T>(p);
    const NodeData nd{coords, uadv, state, node32};
    StageSink<D, T> sk{st + t, rst + t, CH};
    element_row<D, T, SPEC, GEN>(ids, a, nd, force, kp, sk);
    // contributor masks: bit = position of this incidence within its row
    int lo = 0, hi = R - 1;
    while (lo < hi) {  // last rl with s_rowinc[rl] <= t
      const int mid = (lo + hi + 1) >> 1;
      if (s_rowinc[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const int bit = t - s_rowinc[lo];
    if (bit == 0) s_self[lo] = int(pslots & 0xFFu);  // relabelled node 0 is the row node
    if (bit < 64) {
      const int sb = s_spref[lo];
#pragma unroll
      for (int q = 1; q < n; ++q) {  // off-diagonal slots; the diagonal block takes every incidence
        unsigned* word = reinterpret_cast<unsigned*>(s_mask + sb + int((pslots >> (8 * q)) & 0xFFu)) + (bit >> 5);
        atomicOr(word, 1u << (bit & 31));
      }
    }
  }
  __syncthreads();

  // Phase 2a: off-diagonal CSR blocks, one thread per (row, equation,
  // neighbour slot != self); the slot's contributors are visited in ascending
  // element order.  Off-diagonal slots have a few contributors each, so the
  // warps stay converged; the diagonal blocks (every incidence of the row)
  // follow in phase 2b.
  const int nitems = s_pref[R];
  for (int it = t; it < nitems; it += CH) {
    int lo = 0, hi = R - 1;
    while (lo < hi) {  // last rl with s_pref[rl] <= it
      const int mid = (lo + hi + 1) >> 1;
      if (s_pref[mid] <= it) lo = mid; else hi = mid - 1;
    }
    const int rl = lo;
    const int S = s_slots[rl];
    const int local = it - s_pref[rl];
    const int r = local / (S - 1);
    const int s1 = local - r * (S - 1);
    const int s = s1 + (s1 >= s_self[rl] ? 1 : 0);
    const int kb = s_rowinc[rl], ke = s_rowinc[rl + 1];
    const uint32_t key = uint32_t(s) * 0x01010101u;
    double acc[neq];
#pragma unroll
    for (int c = 0; c < neq; ++c) acc[c] = 0.0;
    if (ke - kb <= 64) {
      unsigned long long m = s_mask[s_spref[rl] + s];
      while (m) {
        const int kk = kb + __ffsll(static_cast<long long>(m)) - 1;
        m &= m - 1;
        const int b = (__ffs(__vcmpeq4(s_info[kk], key)) - 1) >> 3;
        const T* src = st + ((b * neq + r) * neq) * CH + kk;
#pragma unroll
        for (int c = 0; c < neq; ++c) acc[c] += double(src[c * CH]);
      }
    } else {  // rows with more than 64 incident elements: scan
      for (int kk = kb; kk < ke; ++kk) {
        const uint32_t eq = __vcmpeq4(s_info[kk], key);
        if (eq) {
          const int b = (__ffs(eq) - 1) >> 3;
          const T* src = st + ((b * neq + r) * neq) * CH + kk;
#pragma unroll
          for (int c = 0; c < neq; ++c) acc[c] += double(src[c * CH]);
        }
      }
    }
    const int64_t base = int64_t(neq) * neq * start[row0 + rl] + int64_t(r * S + s) * neq;
#pragma unroll
    for (int c = 0; c < neq; ++c) vals[base + c] = acc[c];
    if (vals32 != nullptr) {
#pragma unroll
      for (int c = 0; c < neq; ++c) vals32[base + c] = float(acc[c]);
    }
  }
  // Phase 2b: diagonal blocks and RHS, one thread per (row, equation): every
  // incidence of the row contributes, with the row node at local position 0.
  for (int it = t; it < R * neq; it += CH) {
    const int rl = it / neq, r = it - rl * neq;
    const int kb = s_rowinc[rl], ke = s_rowinc[rl + 1];
    double acc[neq];
#pragma unroll
    for (int c = 0; c < neq; ++c) acc[c] = 0.0;
    double racc = 0.0;
    const T* src = st + (r * neq) * CH;  // b = 0
    for (int kk = kb; kk < ke; ++kk) {
#pragma unroll
      for (int c = 0; c < neq; ++c) acc[c] += double(src[c * CH + kk]);
      racc += double(rst[r * CH + kk]);
    }
    const int S = s_slots[rl];
    const int64_t base = int64_t(neq) * neq * start[row0 + rl] + int64_t(r * S + s_self[rl]) * neq;
#pragma unroll
    for (int c = 0; c < neq; ++c) vals[base + c] = acc[c];
    if (vals32 != nullptr) {
#pragma unroll
      for (int c = 0; c < neq; ++c) vals32[base + c] = float(acc[c]);
    }
    rhs[int64_t(row0 + rl) * neq + r] = racc;
  }
}

// ---------------------------------------------------------------------------
// Warp-per-row-group assembly.  A warp owns a range of consecutive block rows
// with at most 32 incidences in total; lane l evaluates incidence l of the range
// (incidences are sorted by row, then element id) and stages its row block's head,
// columns and RHS row (RecordLayout).  The lanes then own CSR items: products and
// plain sums over the row's lanes that make up the diagonal block and the RHS, and
// the off-diagonal (row, slot) blocks, whose contributors the static item words
// list in ascending element order -- one lane a block in 2D, two in 3D, each
// taking every other contributor of the whole block (16 sums in registers; the
// halves are added at the end).  Every sum runs in a fixed order that depends on
// the row alone, and each value is written once.
//
// What bounds it: passes through the L1 / shared-memory pipe (84% busy at 16 warps
// an SM), then issue (45%) and FP64 (28%), not bytes (DRAM 16% of the measured copy
// rate).  So the records hold what the blocks are made of (3D: 50 numbers an
// incidence with the row node's column multiplied out, against 68 of the whole
// block), a node's 32 bytes are gathered by one load, the contributor lists are
// static words instead of masks built by shared-memory atomics, and the smaller
// staging leaves room for 16 warps (128 registers) where 12 fitted.  64^3 x 6 on a
// B200, before -> after: FP64 generic 0.737 -> 0.591 ms, specialised 0.843 -> 0.530,
// FP32 generic 0.545 -> 0.457; 301^2 x 2 triangles in random order, FP64 generic 45.6
// -> 42.2 us, specialised 50.1 -> 41.7; FP32 elements with the conditions 61.2 -> 51.5 and
// 60.8 -> 49.3.
// ---------------------------------------------------------------------------
constexpr size_t kDescSlot = (sizeof(AsmDesc) + 15) / 16 * 16;

// KC: lanes that evaluate incidences (group capacity); the staging holds KC lanes.
template <int D, typename T, int KC = 32, bool BATCH = false>
constexpr size_t warp_stage_bytes() {
  return (size_t(KC) * RecordLayout<D, T>::pitch * sizeof(T) + 15) / 16 * 16 +  // one record per lane
         size_t(36 + 36) * 4 +                  // lane offset and CSR block offset of each row
         (BATCH ? 2 * kDescSlot : 0);           // batch: descriptors of the current and next mesh
}

// Resident-CTA hints (register budgets): warps an SM.  64^3 x 6, generic, 4-warp
// CTAs: FP64 0.595 ms at 16 warps, 0.737 at 12 and 0.771 at 20 (spills); FP32 0.480 at
// 16, 0.457 at 20.  The batched 3D FP64 kernel spills at 16 (its descriptors are in
// shared memory), so it keeps 12.  Triangles, FP64: 16 (20 and 24 spill and take a fifth to
// a half longer); FP32: 24 (fewer took longer: 455 us at 20 and 497 at 16 where 24 took
// 442), batched 20 (at 24 the generic form spills: 8 meshes of 300^2 in random order 371
// us, 326 at 20).
template <int D, typename T, bool BATCH, int WPB>
constexpr int warp_min_blocks() {
  const int warps = D == 3 ? (sizeof(T) == 4 ? 20 : (BATCH ? 12 : 16)) : (sizeof(T) == 4 ? (BATCH ? 20 : 24) : 16);
  return warps / WPB > 0 ? warps / WPB : 1;
}

// Reduction of a group's rows from its staged records, tetrahedra.  Row by row, 16
// off-diagonal blocks at a time: two lanes a block, each summing every other
// contributor's whole block (16 sums in registers), then rows 0-1 of the block end
// up in the even lane and rows 2-3 in the odd one and are written.  Every order
// depends on the row's elements alone (not on its place in the group nor on the
// order of its neighbours).
// `next` runs once, with the loads it starts hidden behind the second half.
template <typename T, int KC, typename F>
__device__ __forceinline__ void reduce_rows_3d(const T* stage, const int* s_off, const int* s_start, int R, int row0,
                                               int64_t gstart, const unsigned long long* __restrict__ words,
                                               unsigned long long word, const AsmDesc& d, F&& next) {
  using L = RecordLayout<3, T>;
  constexpr int LS = L::pitch;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool odd = (lane & 1) != 0;
  double* __restrict__ vals = d.vals;
  float* __restrict__ vals32 = d.vals32;
  for (int rl = 0; rl < R; ++rl) {
    const int kb = s_off[rl], ke = s_off[rl + 1];
    const int w0 = s_start[rl] - rl;                     // the row's first item word
    const int S = s_start[rl + 1] - s_start[rl];
    const int64_t base0 = 16 * (gstart + s_start[rl]);   // the row's first CSR value
    const int64_t row = row0 + rl;
    int self = 0;
    for (int p0 = 0; p0 < S - 1; p0 += 16) {
      const int it = p0 + (lane >> 1);
      const bool on = it < S - 1;
      if (rl + p0 > 0) word = on ? __ldg(words + w0 + it) : 0ull;
      const bool over = (word >> 63) != 0;
      const int slot = int(word >> 52) & 63;
      const int cnt = over ? int(word >> 32) & 0xff : int(word >> 49) & 7;
      const uint8_t* more = d.over + uint32_t(word);
      const T* base = stage + kb * LS;
      double acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
      unsigned long long list = word >> (odd ? 7 : 0);
#pragma unroll 1
      for (int c = odd ? 1 : 0; c < cnt; c += 2, list >>= 14) {
        const int id = over ? int(__ldg(more + c)) : int(list & 127u);
        const T* rec = base + (id >> 2) * LS;
        const T* col = rec + (L::head - L::col) + (id & 3) * L::col;
        double h[4], q[8];  // tg (3), thS; G (3), diag, p row (4)
        if constexpr (std::is_same<T, double>::value) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const double2 x = reinterpret_cast<const double2*>(rec)[k];
            h[2 * k] = x.x;
            h[2 * k + 1] = x.y;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double2 x = reinterpret_cast<const double2*>(col)[k];
            q[2 * k] = x.x;
            q[2 * k + 1] = x.y;
          }
        } else {
          const float4 x = *reinterpret_cast<const float4*>(rec);
          h[0] = double(x.x); h[1] = double(x.y); h[2] = double(x.z); h[3] = double(x.w);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float4 y = reinterpret_cast<const float4*>(col)[k];
            q[4 * k] = double(y.x); q[4 * k + 1] = double(y.y); q[4 * k + 2] = double(y.z); q[4 * k + 3] = double(y.w);
          }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int j = 0; j < 3; ++j) acc[i][j] = fma(h[i], q[j], acc[i][j]);
          acc[i][i] += q[3];
          acc[i][3] = fma(h[3], q[i], acc[i][3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[3][j] += q[4 + j];
      }
      // slot of the row node: the slots are ascending, so it is where they skip one
      self += __popc(__ballot_sync(FULL, on && !odd && slot == it));
      double out[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double give = odd ? acc[i][j] : acc[i + 2][j];
          const double keep = odd ? acc[i + 2][j] : acc[i][j];
          const double got = __shfl_xor_sync(FULL, give, 1);
          out[i][j] = odd ? got + keep : keep + got;  // even contributors first
        }
      if (on) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int64_t pos = base0 + int64_t(((odd ? 2 : 0) + i) * S + slot) * 4;
          st4_cs(vals + pos, out[i][0], out[i][1], out[i][2], out[i][3]);  // streamed: L2 keeps the node data
          if (vals32 != nullptr)
            __stcs(reinterpret_cast<float4*>(vals32 + pos),
                   make_float4(float(out[i][0]), float(out[i][1]), float(out[i][2]), float(out[i][3])));
        }
      }
    }
    if (rl == R - 1) next();
    // diagonal block and RHS row: lane e of ten sums a pair of entries over every
    // third incidence, three sets of ten lanes, then the sets in order
    {
      const int part = lane / 10, e = lane - part * 10;
      double a0 = 0.0, a1 = 0.0;
      if (part < 3) {
        const T* q = stage + L::sums + 2 * e;
#pragma unroll 4
        for (int k = kb + part; k < ke; k += 3) {
          if constexpr (std::is_same<T, double>::value) {
            const double2 x = *reinterpret_cast<const double2*>(q + k * LS);
            a0 += x.x;
            a1 += x.y;
          } else {
            const float2 x = *reinterpret_cast<const float2*>(q + k * LS);
            a0 += double(x.x);
            a1 += double(x.y);
          }
        }
      }
      const double b0 = __shfl_down_sync(FULL, a0, 10), b1 = __shfl_down_sync(FULL, a1, 10);
      const double c0 = __shfl_down_sync(FULL, a0, 20), c1 = __shfl_down_sync(FULL, a1, 20);
      a0 = (a0 + b0) + c0;
      a1 = (a1 + b1) + c1;
      if (lane < 8) {
        const int64_t pos = base0 + int64_t((lane >> 1) * S + self) * 4 + (lane & 1) * 2;
        __stcs(reinterpret_cast<double2*>(vals + pos), make_double2(a0, a1));
        if (vals32 != nullptr) __stcs(reinterpret_cast<float2*>(vals32 + pos), make_float2(float(a0), float(a1)));
      } else if (lane < 10) {
        __stcs(reinterpret_cast<double2*>(d.rhs + row * 4 + (lane - 8) * 2), make_double2(a0, a1));
      }
    }
  }
}

// ... triangles: a lane an entry of the diagonal blocks and the RHS rows (summed
// over the row's lanes), then a lane an off-diagonal block.
template <typename T, typename F>
__device__ __forceinline__ void reduce_rows_2d(const T* stage, const int* s_off, const int* s_start, int R, int row0,
                                               int64_t gstart, const unsigned long long* __restrict__ words,
                                               unsigned long long word, const AsmDesc& d, F&& next) {
  using L = RecordLayout<2, T>;
  constexpr int LS = L::pitch;
  const int lane = threadIdx.x & 31;
  double* __restrict__ vals = d.vals;
  float* __restrict__ vals32 = d.vals32;
  for (int it = lane; it < R * 12; it += 32) {
    const int rl = it / 12, dl = it - rl * 12;
    const int64_t row = row0 + rl;
    const int er = dl / 3, ec = dl - er * 3;
    int64_t pos = 0;
    if (dl < 9) pos = __ldg(d.diagpos + row * 3 + er) - er + ec;
    const T* q = stage + (dl < 9 ? dl : L::sums + dl - 9);
    double acc = 0.0;
    const int ke = s_off[rl + 1];
#pragma unroll 4
    for (int k = s_off[rl]; k < ke; ++k) acc += double(q[k * LS]);
    if (dl < 9) {
      __stcs(vals + pos, acc);
      if (vals32 != nullptr) __stcs(vals32 + pos, float(acc));
    } else {
      __stcs(d.rhs + row * 3 + (dl - 9), acc);
    }
  }
  next();
  const int nslot = s_start[R] - R;
  for (int it = lane; it < nslot; it += 32) {
    if (it >= 32) word = __ldg(words + it);
    const bool over = (word >> 63) != 0;
    const int rl = (int(word >> 58) - row0) & 31;
    const int slot = int(word >> 52) & 63;
    const int cnt = over ? int(word >> 32) & 0xff : int(word >> 49) & 7;
    const uint8_t* more = d.over + uint32_t(word);
    const T* base = stage + s_off[rl] * LS;
    double acc[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) acc[e] = 0.0;
    unsigned long long list = word;
#pragma unroll 1
    for (int c = 0; c < cnt; ++c, list >>= 7) {
      const int id = over ? int(__ldg(more + c)) : int(list & 127u);
      const T* q = base + (id >> 2) * LS + (id & 3) * 9;
#pragma unroll
      for (int e = 0; e < 9; ++e) acc[e] += double(q[e]);
    }
    const int S = s_start[rl + 1] - s_start[rl];
    const int64_t base0 = 9 * (gstart + s_start[rl]) + slot * 3;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t pos = base0 + int64_t(r) * S * 3 + c;
        __stcs(vals + pos, acc[r * 3 + c]);
        if (vals32 != nullptr) __stcs(vals32 + pos, float(acc[r * 3 + c]));
      }
  }
}

// Triangles with FP32 elements.  The values of a group are one run of the CSR: a group of
// usual size (five rows of six elements, at most 32 off-diagonal blocks) puts them
// together over its records and writes the run, FP64 and FP32 copy, lane by lane.
// Written where they are summed, 24 and 12 bytes a lane and row, every sector goes to L2
// in three parts.  1000^2 in natural order, with the conditions: generic 448 -> 402 us,
// specialised 437 -> 395, random order 512 -> 474.  FP64 elements, with one copy and fewer
// warps to hide the second pass over shared memory behind, lose by it (471 -> 537) and
// write directly.
template <typename F>
__device__ __forceinline__ void reduce_run_2d(float* stage, const int* s_off, const int* s_start, int R, int row0,
                                              int64_t gstart, const unsigned long long* __restrict__ words,
                                              unsigned long long word, const AsmDesc& d, F&& next) {
  using L = RecordLayout<2, float>;
  constexpr int LS = L::pitch;
  constexpr int kRows = 5, kBlocks = 32;
  static_assert((kRows + kBlocks) * 9 * sizeof(double) <= size_t(32) * LS * sizeof(float), "the run fits the records' place");
  const int lane = threadIdx.x & 31;
  const int nslot = s_start[R] - R;
  if (R > kRows || nslot > kBlocks) {  // the whole warp
    reduce_rows_2d<float>(stage, s_off, s_start, R, row0, gstart, words, word, d, next);
    return;
  }
  double dv[2] = {0.0, 0.0}, acc[9];
  int at[3] = {-1, -1, 0}, step = 0;  // places in the run
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int it = lane + 32 * h;
    if (it >= R * 12) continue;
    const int rl = it / 12, dl = it - rl * 12;
    const int64_t row = row0 + rl;
    const int er = dl / 3, ec = dl - er * 3;
    if (dl < 9) at[h] = int(__ldg(d.diagpos + row * 3 + er) - er + ec - 9 * gstart);
    const float* q = stage + (dl < 9 ? dl : L::sums + dl - 9);
    const int ke = s_off[rl + 1];
#pragma unroll 4
    for (int k = s_off[rl]; k < ke; ++k) dv[h] += double(q[k * LS]);
    if (dl >= 9) __stcs(d.rhs + row * 3 + (dl - 9), dv[h]);
  }
  next();
  if (lane < nslot) {
    const bool over = (word >> 63) != 0;
    const int rl = (int(word >> 58) - row0) & 31;
    const int cnt = over ? int(word >> 32) & 0xff : int(word >> 49) & 7;
    const uint8_t* more = d.over + uint32_t(word);
    const float* base = stage + s_off[rl] * LS;
#pragma unroll
    for (int e = 0; e < 9; ++e) acc[e] = 0.0;
    unsigned long long list = word;
#pragma unroll 1
    for (int c = 0; c < cnt; ++c, list >>= 7) {
      const int id = over ? int(__ldg(more + c)) : int(list & 127u);
      const float* q = base + (id >> 2) * LS + (id & 3) * 9;
#pragma unroll
      for (int e = 0; e < 9; ++e) acc[e] += double(q[e]);
    }
    at[2] = 9 * s_start[rl] + (int(word >> 52) & 63) * 3;
    step = (s_start[rl + 1] - s_start[rl]) * 3;
  }
  __syncwarp();  // the records are summed
  double* out = reinterpret_cast<double*>(stage);
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (at[h] >= 0) out[at[h]] = dv[h];
  if (lane < nslot)
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) out[at[2] + r * step + c] = acc[r * 3 + c];
  __syncwarp();
  const int n = 9 * s_start[R];
  for (int i = lane; i < n; i += 32) {
    const double v = out[i];
    __stcs(d.vals + 9 * gstart + i, v);
    if (d.vals32 != nullptr) __stcs(d.vals32 + 9 * gstart + i, float(v));
  }
}

template <int D, typename T, bool SPEC, bool GEN, int WPB, bool BATCH, int KC>
__global__ void __launch_bounds__(32 * WPB, warp_min_blocks<D, T, BATCH, WPB>()) ns_assembly_warp_kernel(
    int ngroups, int nmesh, const AsmDesc* __restrict__ descs, const int* __restrict__ gprefix,
    const __grid_constant__ AsmDesc one) {
  constexpr int LS = RecordLayout<D, T>::pitch;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* slice = smem_raw + size_t(warp) * warp_stage_bytes<D, T, KC, BATCH>();
  T* stage = reinterpret_cast<T*>(slice);
  int* s_off = reinterpret_cast<int*>(slice + (size_t(KC) * LS * sizeof(T) + 15) / 16 * 16);  // 33 (+3 pad)
  int* s_start = s_off + 36;                                                                  // 33 (+3 pad)
  // Mesh descriptors: a one-mesh launch reads its descriptor from the kernel
  // parameters; a batch keeps the descriptors of the current and the next
  // group's mesh in the warp's slice (copied when the mesh changes).
  AsmDesc* s_desc = reinterpret_cast<AsmDesc*>(reinterpret_cast<unsigned char*>(s_start + 36));
  int mesh0 = -1, mesh1 = -1;  // mesh held by descriptor slot 0 / 1
  auto load_desc = [&](int m, int slot) {
    if constexpr (BATCH) {
      const int held = slot ? mesh1 : mesh0;
      if (held != m) {  // warp-uniform
        constexpr int W = int(sizeof(AsmDesc) / 8);
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(descs + m);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(s_desc + slot);
        for (int q = lane; q < W; q += 32) dst[q] = __ldg(src + q);
        if (slot) mesh1 = m; else mesh0 = m;
        __syncwarp();
      }
    }
  };
  // The descriptor of the mesh in slot `slot`: a batch's shared copy, or the
  // launch's parameter.
#define UFEM_DESC(slot) (BATCH ? s_desc[(slot)] : one)
  // Persistent warps: a warp walks the global groups g, g + stride, ... of all
  // meshes of the launch (mesh m owns groups [gprefix[m], gprefix[m + 1])).
  // While it reduces one group it already loads the incidence records, the
  // connectivity and the item words of the next.
  int g = blockIdx.x * WPB + warp;
  if (g >= ngroups) return;  // whole warp; no CTA-wide barrier below
  const int gstride = gridDim.x * WPB;
  auto mesh_of = [&](int q) {  // last m with gprefix[m] <= q
    int lo = 0, hi = nmesh - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(gprefix + mid) <= q) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  int cm = BATCH ? mesh_of(g) : 0;
  int cs = 0;  // descriptor slot of the current mesh
  load_desc(cm, cs);
  // first row, end row, first incidence, incidences
  int4 G = BATCH ? __ldg(UFEM_DESC(cs).groups + (g - __ldg(gprefix + cm))) : __ldg(one.groups + g);
  uint32_t pea = 0;                 // the lane's incidence
  int poff = 0, pstart = 0;         // the lane's row: lane offset, CSR block offset from the group's first
  int pend = 0;                     // CSR blocks of the group
  int64_t gs = 0;                   // CSR block offset of the group's first row
  int4 pcn = make_int4(0, 0, 0, 0);
  auto fetch_records = [&](const int4& q, const AsmDesc& d) {
    if (lane < q.w) pea = __ldg(d.inc_ea + q.z + lane);
    gs = __ldg(d.start + q.x);
    if (lane < q.y - q.x) poff = __ldg(d.row_inc + q.x + lane) - q.z;
    if (lane < q.y - q.x) pstart = int(__ldg(d.start + q.x + lane) - gs);
    pend = int(__ldg(d.start + q.y) - gs);
  };
  fetch_records(G, UFEM_DESC(cs));
  if (lane < G.w) pcn = __ldg(UFEM_DESC(cs).conn + (pea & 0x3fffffffu));
  for (;;) {
    const int row0 = G.x, R = G.y - G.x, K = G.w;  // 1 <= R <= K <= KC
    const int gn = g + gstride;
    const int mn = (BATCH && gn < ngroups) ? mesh_of(gn) : cm;
    const int ns = (mn == cm) ? cs : 1 - cs;  // descriptor slot of the next group's mesh
    int4 Gn = make_int4(0, 0, 0, 0);
    if constexpr (!BATCH) {
      if (gn < ngroups) Gn = __ldg(one.groups + gn);
    }
    __syncwarp();  // the previous group's reads of the shared slice are complete
    if constexpr (BATCH) {
      load_desc(mn, ns);
      if (gn < ngroups) Gn = __ldg(s_desc[ns].groups + (gn - __ldg(gprefix + mn)));
    }
    if (lane < R) {
      s_off[lane] = poff;
      s_start[lane] = pstart;
    }
    if (lane == 0) {
      s_off[R] = K;
      s_start[R] = pend;
    }
    const int64_t gstart = gs;
    const unsigned long long* __restrict__ words = UFEM_DESC(cs).items + (gstart - row0);

    // Phase 1: one lane per incidence, the element's nodes relabelled so that the
    // row node is local node 0.
    // A batch's launch leaves the meshes of the other kind (GEN) to their own.
    const bool skip = BATCH && (UFEM_DESC(cs).gen != 0) != GEN;  // warp-uniform
    if (lane < K && !skip) {
      const int a = int(pea >> 30);
      const int ids0[4] = {pcn.x, pcn.y, pcn.z, pcn.w};
      int ids[4] = {0, 0, 0, 0};
      if constexpr (D == 3) {
        const bool x1 = (a & 1) != 0, x2 = (a & 2) != 0;
        const int p0 = x1 ? ids0[1] : ids0[0], p1 = x1 ? ids0[0] : ids0[1], p2 = x1 ? ids0[3] : ids0[2],
                  p3 = x1 ? ids0[2] : ids0[3];
        ids[0] = x2 ? p2 : p0;
        ids[1] = x2 ? p3 : p1;
        ids[2] = x2 ? p0 : p2;
        ids[3] = x2 ? p1 : p3;
      } else {
        ids[0] = a == 0 ? ids0[0] : (a == 1 ? ids0[1] : ids0[2]);
        ids[1] = a == 0 ? ids0[1] : (a == 1 ? ids0[2] : ids0[0]);
        ids[2] = a == 0 ? ids0[2] : (a == 1 ? ids0[0] : ids0[1]);
      }
      const AsmDesc& d = UFEM_DESC(cs);
      const KParams<T> kp = make_kparams<T>(d.p);
      const NodeData nd{d.coords, d.uadv, d.state, d.node32};
      RecordSink<D, T> sk{stage + lane * LS};
      element_row<D, T, SPEC, GEN>(ids, a, nd, d.force, kp, sk);
    }
    __syncwarp();
    constexpr int PAR = D == 3 ? 2 : 1;  // lanes per off-diagonal block
    // item words of the group's first pass (3D: the first row's, 2D: the group's)
    const int nfirst = D == 3 ? s_start[1] - 1 : s_start[R] - R;
    unsigned long long word = lane < nfirst * PAR ? __ldg(words + lane / PAR) : 0ull;
    fetch_records(Gn, UFEM_DESC(ns));  // next group's records load while this group is reduced
    if (skip) {
      if (lane < Gn.w) pcn = __ldg(UFEM_DESC(ns).conn + (pea & 0x3fffffffu));
    } else if constexpr (D == 3) {
      reduce_rows_3d<T, KC>(stage, s_off, s_start, R, row0, gstart, words, word, UFEM_DESC(cs),
                            [&] { if (lane < Gn.w) pcn = __ldg(UFEM_DESC(ns).conn + (pea & 0x3fffffffu)); });
    } else {
      auto next = [&] { if (lane < Gn.w) pcn = __ldg(UFEM_DESC(ns).conn + (pea & 0x3fffffffu)); };
      if constexpr (std::is_same<T, float>::value)
        reduce_run_2d(stage, s_off, s_start, R, row0, gstart, words, word, UFEM_DESC(cs), next);
      else
        reduce_rows_2d<T>(stage, s_off, s_start, R, row0, gstart, words, word, UFEM_DESC(cs), next);
    }
    if (gn >= ngroups) break;
    g = gn;
    G = Gn;
    cm = mn;
    cs = ns;
  }
#undef UFEM_DESC
}

// LinearizeU (NavierStokes.cpp:105), evaluated left to right without FMA
// contraction: u_adv = ((2.1875u - 2.1875u1) + 1.3125u2) - 0.3125u3.  Also
// copies nu_eff into the node record read by the assembly.
__global__ void linearize_kernel(int64_t N, int dim, const double* __restrict__ state,
                                 const double* __restrict__ u1, const double* __restrict__ u2,
                                 const double* __restrict__ u3, const double* __restrict__ nu,
                                 double* __restrict__ uadv, float* __restrict__ node32) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double out[4] = {0, 0, 0, 0};
  for (int k = 0; k < dim; ++k) {
    const int64_t o = 4 * i + k;
    double v = __dsub_rn(__dmul_rn(2.1875, state[o]), __dmul_rn(2.1875, u1[o]));
    v = __dadd_rn(v, __dmul_rn(1.3125, u2[o]));
    v = __dsub_rn(v, __dmul_rn(0.3125, u3[o]));
    out[k] = v;
  }
  out[3] = nu[i];
  reinterpret_cast<double2*>(uadv + 4 * i)[0] = make_double2(out[0], out[1]);
  reinterpret_cast<double2*>(uadv + 4 * i)[1] = make_double2(out[2], out[3]);
  if (node32 != nullptr) {  // FP32 copy for the FP32 element path: (u_adv, nu), (u, p)
    float4* q = reinterpret_cast<float4*>(node32) + 2 * i;
    q[0] = make_float4(float(out[0]), float(out[1]), float(out[2]), float(out[3]));
    const double* x = state + 4 * i;
    q[1] = make_float4(float(x[0]), float(x[1]), dim == 3 ? float(x[2]) : 0.0f, float(x[dim]));
  }
}

// UpdateActions (NavierStokes.cpp:172-179): u3=u2, u2=u1, u1=u, u+=du, p+=dp.
__global__ void update_kernel(int64_t N, int dim, double* __restrict__ state, double* __restrict__ u1,
                              double* __restrict__ u2, double* __restrict__ u3, const double* __restrict__ sol) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int neq = dim + 1;
  for (int k = 0; k < dim; ++k) {
    const int64_t o = 4 * i + k;
    u3[o] = u2[o];
    u2[o] = u1[o];
    const double u = state[o];
    u1[o] = u;
    state[o] = __dadd_rn(u, sol[i * neq + k]);
  }
  state[4 * i + dim] = __dadd_rn(state[4 * i + dim], sol[i * neq + dim]);
}

// Point CSR from the node graph: row node*neq + r, columns adj*neq + c.
__global__ void build_csr_kernel(int64_t N, int neq, const int64_t* __restrict__ start,
                                 const int32_t* __restrict__ adj, int64_t* __restrict__ rowptr,
                                 int32_t* __restrict__ colidx, int64_t* __restrict__ diagpos) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int64_t s0 = start[i];
  const int S = int(start[i + 1] - s0);
  const int64_t base = int64_t(neq) * neq * s0;
  int self = 0;
  for (int s = 0; s < S; ++s)
    if (adj[s0 + s] == i) self = s;
  for (int r = 0; r < neq; ++r) {
    const int64_t rb = base + int64_t(r) * S * neq;
    rowptr[i * neq + r] = rb;
    diagpos[i * neq + r] = rb + int64_t(self) * neq + r;
    for (int s = 0; s < S; ++s) {
      const int32_t cn = adj[s0 + s] * neq;
      for (int c = 0; c < neq; ++c) colidx[rb + int64_t(s) * neq + c] = cn + c;
    }
  }
  if (i == N - 1) rowptr[N * neq] = int64_t(neq) * neq * start[N];
}

// Symmetric Dirichlet: the first column_blocks blocks move the constrained columns
// of the other rows to the RHS, the rest write the constrained rows, eight lanes
// per row.  In one launch: on small meshes the pass is bound by launches.  Three
// launches (values, columns, rows) took 1.7, 2.9 and 2.6 us with the gaps between
// them; assembly and conditions of 64 x 64 x 2 triangles 24.5 -> 16.3 us, of
// 17^3 x 6 tetrahedra 36.9 -> 30.4 us.
__global__ void __launch_bounds__(256) dirichlet_kernel(int column_blocks, DirichletPlan bp,
                                                        const int64_t* __restrict__ rowptr,
                                                        const double* __restrict__ state, double* __restrict__ vals,
                                                        float* __restrict__ vals32, double* __restrict__ rhs,
                                                        double* __restrict__ sol) {
  if (int(blockIdx.x) < column_blocks) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if ((t >> 5) * 4 >= bp.nfix_rows) return;  // whole warp
    const int64_t q = t >> 3;
    const bool valid = q < bp.nfix_rows;
    const int64_t k0 = valid ? bp.fix_ptr[q] : 0;
    dirichlet_columns(valid, valid ? bp.fix_row[q] : 0, k0, valid ? int(bp.fix_ptr[q + 1] - k0) : 0, bp.fix_pos,
                      bp.fix_bc, bp.bc_at, bp.bc_first, state, vals, vals32, rhs);
  } else {
    const int64_t u = (int64_t(blockIdx.x - column_blocks) * blockDim.x + threadIdx.x) >> 3;
    if (u < bp.nbc)
      dirichlet_row(u, bp.bc_dof, bp.bc_at, bp.bc_first, bp.bc_last, bp.bc_diag, rowptr, state, vals, vals32, rhs, sol,
                    bp.vfirst);
  }
}

}  // namespace

void fill_params(const ufem_ns_handle* h, NSParams& p) {
  const double dt = h->opt.dt, c1 = h->opt.c1;
  p.theta = h->opt.theta; p.inv_theta = 1.0 / h->opt.theta; p.dt = dt; p.invdt = 1.0 / dt;
  p.rho = h->opt.rho; p.inv_rho = 1.0 / h->opt.rho;
  p.tau_c1 = 4. * c1 * c1 / (dt * dt);  // SUPG.hpp:184
  p.tau_std = 4. / (dt * dt);           // SUPG.hpp:188
  p.two_dt = 2. / dt;                   // SUPG.hpp:169
  p.c2 = h->opt.c2; p.a_ps = h->opt.alpha_ps; p.a_su = h->opt.alpha_su;
  p.a_bu = h->opt.alpha_bu; p.u_ref = h->opt.u_ref; p.supg_type = h->opt.supg_type;
  p.has_force = h->d_force != nullptr;
}

// Without rows of more than 24 incidences the 24-lane plan serves the "warp" variant of
// tetrahedra too: less staging a warp leaves the L1 more of the SM's array (the rows'
// values are the same bits under both plans).
bool warp_takes_24(const ufem_ns_handle* h) {
  return h->dim == 3 && h->wplan24.big64.nchunks == 0 && h->wplan24.ngroups > 0;
}

// Whether the handle's element routine is the general one (another tau than METRIC).
bool assembly_general(const ufem_ns_handle* h) { return h->opt.use_specializations == 0 && h->opt.supg_type != 1; }

void fill_desc(const ufem_ns_handle* h, bool write32, AsmDesc& d, const WarpPlan* plan) {
  d.coords = h->d_coords;
  d.uadv = h->d_uadv;
  d.state = h->d_state;
  d.node32 = h->d_node32;
  d.force = h->d_force;
  d.start = h->d_start;
  d.row_inc = h->d_row_inc;
  d.inc_ea = h->d_inc_ea;
  d.items = h->d_items;
  d.over = h->d_over;
  d.diagpos = h->d_diagpos;
  d.gen = assembly_general(h) ? 1 : 0;
  d.conn = reinterpret_cast<const int4*>(h->d_conn);
  d.groups = (plan ? plan : &h->wplan)->groups;
  d.vals = h->d_vals;
  d.vals32 = write32 ? h->d_vals32 : nullptr;
  d.rhs = h->d_rhs;
  fill_params(h, d.p);
}

namespace {

template <int D, typename T, int CH, bool SPEC, bool GEN>
int launch_chunk_g(const ufem_ns_handle* h, const AssemblyPlan& plan, const NSParams& p, cudaStream_t s,
                   bool write32) {
  constexpr size_t smem = assembly_smem_bytes<D, T, CH>();
  ns_assembly_kernel<D, T, CH, SPEC, GEN><<<plan.nchunks, CH, smem, s>>>(
      plan.chunks, h->d_row_inc, h->d_inc_elem, h->d_inc_info, reinterpret_cast<const int4*>(h->d_conn),
      h->d_coords, h->d_uadv, h->d_state, h->d_node32, h->d_force, h->d_start, p, h->d_vals,
      write32 ? h->d_vals32 : nullptr, h->d_rhs);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

// f with the element routine of the handle as a type; the specialised form has one only.
template <bool SPEC, typename F>
int with_gen(const ufem_ns_handle* h, F&& f) {
  if constexpr (!SPEC)
    if (assembly_general(h)) return f(std::true_type{});
  return f(std::false_type{});
}

template <int D, typename T, int CH, bool SPEC>
int launch_chunk_t(const ufem_ns_handle* h, const AssemblyPlan& plan, const NSParams& p, cudaStream_t s,
                   bool write32) {
  if (plan.nchunks == 0) return UFEM_OK;
  if (plan.cap != CH) return set_error(UFEM_ERR_STATE, "assembly plan does not match the kernel width");
  return with_gen<SPEC>(h, [&](auto gen) {
    return launch_chunk_g<D, T, CH, SPEC, decltype(gen)::value>(h, plan, p, s, write32);
  });
}

// Resident CTAs of a kernel on the current device (persistent-warp grids).
template <typename K>
int resident_ctas(K kernel, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
    return 0;
  return sms * per_sm;
}

template <int D, typename T, bool SPEC, bool GEN, int WPB, bool BATCH, int KC>
int launch_warp_t(int ngroups, int nmesh, const AsmDesc* descs, const int* gprefix, const AsmDesc& one,
                  cudaStream_t s) {
  if (ngroups == 0) return UFEM_OK;
  constexpr size_t smem = warp_stage_bytes<D, T, KC, BATCH>() * WPB;
  static const int resident =
      resident_ctas(ns_assembly_warp_kernel<D, T, SPEC, GEN, WPB, BATCH, KC>, 32 * WPB, smem);
  if (resident <= 0) return set_error(UFEM_ERR_CUDA, "occupancy query of the warp assembly kernel failed");
  const unsigned grid = unsigned(std::min<int64_t>((ngroups + WPB - 1) / WPB, resident));
  ns_assembly_warp_kernel<D, T, SPEC, GEN, WPB, BATCH, KC><<<grid, 32 * WPB, smem, s>>>(ngroups, nmesh, descs, gprefix,
                                                                                        one);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

template <int D, typename T, bool SPEC, bool GEN, bool BATCH, int KC = 32>
int launch_warp_w(int warps, int ngroups, int nmesh, const AsmDesc* descs, const int* gprefix, const AsmDesc& one,
                  cudaStream_t s) {
  switch (warps) {
    case 2: return launch_warp_t<D, T, SPEC, GEN, 2, BATCH, KC>(ngroups, nmesh, descs, gprefix, one, s);
    case 8: return launch_warp_t<D, T, SPEC, GEN, 8, BATCH, KC>(ngroups, nmesh, descs, gprefix, one, s);
    default: return launch_warp_t<D, T, SPEC, GEN, 4, BATCH, KC>(ngroups, nmesh, descs, gprefix, one, s);
  }
}

template <int D, typename T, int CH, bool SPEC>
int launch_assembly_t(ufem_ns_handle* h, cudaStream_t s, bool write32) {
  NSParams p;
  fill_params(h, p);
  constexpr bool f32 = std::is_same<T, float>::value;
  if (h->asm_variant == kAsmChunk) return launch_chunk_t<D, T, CH, SPEC>(h, f32 ? h->plan32 : h->plan64, p, s, write32);
  int rc;
  const bool w24 = D == 3 && (h->asm_variant == kAsmWarp24 || warp_takes_24(h));
  const WarpPlan& wp = w24 ? h->wplan24 : h->wplan;
  AsmDesc one;  // this handle's descriptor, passed as a kernel parameter
  fill_desc(h, write32, one, &wp);
  rc = with_gen<SPEC>(h, [&](auto gen) {
    constexpr bool G = decltype(gen)::value;
    if constexpr (D == 3) {
      if (w24) return launch_warp_w<D, T, SPEC, G, false, 24>(h->asm_warps, wp.ngroups, 1, nullptr, nullptr, one, s);
    }
    return launch_warp_w<D, T, SPEC, G, false, 32>(h->asm_warps, wp.ngroups, 1, nullptr, nullptr, one, s);
  });
  if (rc) return rc;
  return launch_chunk_t<D, T, CH, SPEC>(h, f32 ? wp.big32 : wp.big64, p, s, write32);
}

template <int D, typename T, bool SPEC, bool GEN, bool BATCH, int KC>
int set_warp_smem_attr() {
  UFEM_CUDA_TRY(cudaFuncSetAttribute(ns_assembly_warp_kernel<D, T, SPEC, GEN, 2, BATCH, KC>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(2 * warp_stage_bytes<D, T, KC, BATCH>())));
  UFEM_CUDA_TRY(cudaFuncSetAttribute(ns_assembly_warp_kernel<D, T, SPEC, GEN, 4, BATCH, KC>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(4 * warp_stage_bytes<D, T, KC, BATCH>())));
  UFEM_CUDA_TRY(cudaFuncSetAttribute(ns_assembly_warp_kernel<D, T, SPEC, GEN, 8, BATCH, KC>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(8 * warp_stage_bytes<D, T, KC, BATCH>())));
  return UFEM_OK;
}

template <int D, typename T, int CH, bool SPEC, bool GEN>
int set_smem_attr_g() {
  constexpr size_t smem = assembly_smem_bytes<D, T, CH>();
  UFEM_CUDA_TRY(cudaFuncSetAttribute(ns_assembly_kernel<D, T, CH, SPEC, GEN>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  int rc;
  if ((rc = set_warp_smem_attr<D, T, SPEC, GEN, false, 32>()) || (rc = set_warp_smem_attr<D, T, SPEC, GEN, true, 32>()))
    return rc;
  if constexpr (D == 3) {
    if ((rc = set_warp_smem_attr<D, T, SPEC, GEN, false, 24>())) return rc;
  }
  return UFEM_OK;
}

template <int D, typename T, int CH, bool SPEC>
int set_smem_attr() {
  const int rc = set_smem_attr_g<D, T, CH, SPEC, false>();
  if constexpr (SPEC) return rc;
  else return rc ? rc : set_smem_attr_g<D, T, CH, SPEC, true>();
}

// ---------------------------------------------------------------------------
// Matrix-free FP64 residual.  The refinement residual of the mixed-precision
// solve when the element matrices are assembled in FP32: for the current
// increment dx, r = b - M dx of the FP64 system that the FP64 assembly and the
// symmetric Dirichlet conditions would have built, evaluated element by element
// without forming M.  Per incidence (row node, element) the FP64 element
// routine runs with a sink that applies the row block of M = invdt T + theta A
// (NavierStokesAssembly.hpp:69-71) to the element's increment instead of staging
// it, and keeps the RHS row a - A x (the reference's system_rhs += -_A _x + _a,
// :69); the rows' contributions are then summed in element order.
// Constrained columns take the value of their dof's first application (what the
// symmetric Dirichlet pass moves to the RHS), constrained rows get r = 0 (their
// increment already holds the row value, which the inner corrections keep).
// ---------------------------------------------------------------------------
template <int D>
struct ResidSink {
  double dl[D + 1][D + 1];  // increment of the relabelled element nodes (u, v, [w], p)
  double acc[D + 1];        // (M dx) of the row
  double rr[D + 1];         // a - A x of the row
  double tg[D], thS, sWSp, c[D];
  __device__ __forceinline__ void head(const double (&tg_)[D], double thS_, double sWSp_, const double (&c_)[D]) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      tg[k] = tg_[k];
      c[k] = c_[k];
    }
    thS = thS_;
    sWSp = sWSp_;
  }
  __device__ __forceinline__ void col(int b, const double (&g)[D], double diag, double vem, double dd) {
    double div = 0.0, cd = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      div += g[k] * dl[b][k];
      cd += c[k] * dl[b][k];
    }
#pragma unroll
    for (int i = 0; i < D; ++i) acc[i] += tg[i] * div + (diag * dl[b][i] + thS * (g[i] * dl[b][D]));
    acc[D] += sWSp * div + (vem * cd + dd * dl[b][D]);
  }
  __device__ __forceinline__ void rhs(const double (&v)[D + 1]) {
#pragma unroll
    for (int r = 0; r <= D; ++r) rr[r] = v[r];
  }
};

// One CTA per chunk of whole rows (the chunk plan), one thread per incidence.
// 128 registers a thread (16 warps an SM): the gathers' latency is what it waits for.
template <int D, int CH, bool SPEC, bool GEN>
__global__ void __launch_bounds__(CH, 512 / CH) ns_residual_kernel(
    const int2* __restrict__ chunk_rows, const int32_t* __restrict__ row_inc, const int32_t* __restrict__ inc_elem,
    const uint32_t* __restrict__ inc_info, const int4* __restrict__ conn, const double* __restrict__ coords,
    const double* __restrict__ uadv, const double* __restrict__ state, const double* __restrict__ force, NSParams p,
    const double* __restrict__ dx, double* __restrict__ res) {
  constexpr int n = D + 1, neq = D + 1;
  __shared__ double s_res[neq * CH];
  __shared__ int s_rowinc[CH + 1];
  const int2 cr = chunk_rows[blockIdx.x];
  const int row0 = cr.x, R = cr.y - cr.x;  // 1 <= R <= K <= CH
  const int inc0 = row_inc[row0];
  const int K = row_inc[cr.y] - inc0;
  const int t = threadIdx.x;
  for (int rl = t; rl <= R; rl += CH) s_rowinc[rl] = row_inc[row0 + rl] - inc0;
  if (t < K) {
    const int k = inc0 + t;
    const int e = __ldg(inc_elem + k);
    const int a = int(__ldg(inc_info + k) >> 24) & 3;
    const int4 cn = __ldg(conn + e);
    const int ids0[4] = {cn.x, cn.y, cn.z, cn.w};
    int ids[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) ids[q] = ids0[(D == 3) ? (q ^ a) : (q < 3 ? (q + a) % 3 : 3)];
    ResidSink<D> sk;
#pragma unroll
    for (int q = 0; q < n; ++q)
#pragma unroll
      for (int c = 0; c < neq; ++c) sk.dl[q][c] = __ldg(dx + int64_t(ids[q]) * neq + c);
#pragma unroll
    for (int r = 0; r < neq; ++r) sk.acc[r] = 0.0;
    const KParams<double> kp = make_kparams<double>(p);
    const NodeData nd{coords, uadv, state, nullptr};
    element_row<D, double, SPEC, GEN>(ids, a, nd, force, kp, sk);
#pragma unroll
    for (int r = 0; r < neq; ++r) s_res[r * CH + t] = sk.rr[r] - sk.acc[r];
  }
  __syncthreads();
  for (int it = t; it < R * neq; it += CH) {  // sums over the row's incidences in element order
    const int rl = it / neq, r = it - rl * neq;
    double acc = 0.0;
    for (int kk = s_rowinc[rl]; kk < s_rowinc[rl + 1]; ++kk) acc += s_res[r * CH + kk];
    res[int64_t(row0 + rl) * neq + r] = acc;
  }
}

// dx' = dx with each constrained dof replaced by its first application's value
// (value - old), the column value the symmetric Dirichlet pass moves to the RHS.
__global__ void mf_columns_kernel(int64_t nbc, const int64_t* __restrict__ bc_dof, const double* __restrict__ vfirst,
                                  double* __restrict__ dxp) {
  const int64_t u = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (u < nbc) dxp[bc_dof[u]] = vfirst[u];
}

__global__ void mf_rows_kernel(int64_t nbc, const int64_t* __restrict__ bc_dof, double* __restrict__ res) {
  const int64_t u = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (u < nbc) res[bc_dof[u]] = 0.0;
}

template <int D, int CH, bool SPEC>
int launch_residual_t(ufem_ns_handle* h, const double* dxp, double* res, cudaStream_t s) {
  NSParams p;
  fill_params(h, p);
  if (h->plan64.cap != CH) return set_error(UFEM_ERR_STATE, "chunk plan does not match the residual kernel width");
  return with_gen<SPEC>(h, [&](auto gen) {
    ns_residual_kernel<D, CH, SPEC, decltype(gen)::value><<<h->plan64.nchunks, CH, 0, s>>>(
        h->plan64.chunks, h->d_row_inc, h->d_inc_elem, h->d_inc_info, reinterpret_cast<const int4*>(h->d_conn),
        h->d_coords, h->d_uadv, h->d_state, h->d_force, p, dxp, res);
    UFEM_CUDA_TRY(cudaGetLastError());
    return int(UFEM_OK);
  });
}

constexpr int kChunk2D = 256;
constexpr int kChunk3D64 = 128;
constexpr int kChunk3D32 = 256;

}  // namespace

int assembly_chunk_capacity(int dim, int precision) {
  if (dim == 2) return kChunk2D;
  return precision == 1 ? kChunk3D32 : kChunk3D64;
}

int configure_kernels() {
  static bool done = false;
  if (done) return UFEM_OK;
  int rc;
  if ((rc = set_smem_attr<2, double, kChunk2D, false>())) return rc;
  if ((rc = set_smem_attr<2, double, kChunk2D, true>())) return rc;
  if ((rc = set_smem_attr<2, float, kChunk2D, false>())) return rc;
  if ((rc = set_smem_attr<2, float, kChunk2D, true>())) return rc;
  if ((rc = set_smem_attr<3, double, kChunk3D64, false>())) return rc;
  if ((rc = set_smem_attr<3, double, kChunk3D64, true>())) return rc;
  if ((rc = set_smem_attr<3, float, kChunk3D32, false>())) return rc;
  if ((rc = set_smem_attr<3, float, kChunk3D32, true>())) return rc;
  done = true;
  return UFEM_OK;
}

int launch_assembly(ufem_ns_handle* h, cudaStream_t s, bool write32) {
  const bool spec = h->opt.use_specializations != 0;
  const bool f32 = h->opt.precision == 1;
  if (h->dim == 2) {
    if (f32) return spec ? launch_assembly_t<2, float, kChunk2D, true>(h, s, write32)
                         : launch_assembly_t<2, float, kChunk2D, false>(h, s, write32);
    return spec ? launch_assembly_t<2, double, kChunk2D, true>(h, s, write32)
                : launch_assembly_t<2, double, kChunk2D, false>(h, s, write32);
  }
  if (f32) return spec ? launch_assembly_t<3, float, kChunk3D32, true>(h, s, write32)
                       : launch_assembly_t<3, float, kChunk3D32, false>(h, s, write32);
  return spec ? launch_assembly_t<3, double, kChunk3D64, true>(h, s, write32)
              : launch_assembly_t<3, double, kChunk3D64, false>(h, s, write32);
}

namespace {
template <int D, typename T, bool SPEC>
int launch_batch_t(int warps, int kinds, int ngroups, int nmesh, const AsmDesc* d_descs, const int* d_gprefix,
                   cudaStream_t s) {
  int rc;
  if ((kinds & 1) && (rc = launch_warp_w<D, T, SPEC, false, true>(warps, ngroups, nmesh, d_descs, d_gprefix, AsmDesc{}, s)))
    return rc;
  if constexpr (!SPEC)
    if ((kinds & 2) && (rc = launch_warp_w<D, T, SPEC, true, true>(warps, ngroups, nmesh, d_descs, d_gprefix, AsmDesc{}, s)))
      return rc;
  return UFEM_OK;
}
}  // namespace

int launch_assembly_batch(int dim, int precision, bool spec, int warps, int kinds, int ngroups, int nmesh,
                          const AsmDesc* d_descs, const int* d_gprefix, cudaStream_t s) {
  const bool f32 = precision == 1;
  if (dim == 2) {
    if (f32) return spec ? launch_batch_t<2, float, true>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s)
                         : launch_batch_t<2, float, false>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s);
    return spec ? launch_batch_t<2, double, true>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s)
                : launch_batch_t<2, double, false>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s);
  }
  if (f32) return spec ? launch_batch_t<3, float, true>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s)
                       : launch_batch_t<3, float, false>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s);
  return spec ? launch_batch_t<3, double, true>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s)
              : launch_batch_t<3, double, false>(warps, kinds, ngroups, nmesh, d_descs, d_gprefix, s);
}

int launch_assembly_big_rows(ufem_ns_handle* h, cudaStream_t s, bool write32) {
  NSParams p;
  fill_params(h, p);
  const bool spec = h->opt.use_specializations != 0;
  const bool f32 = h->opt.precision == 1;
  const WarpPlan& w = h->wplan;
  if (h->dim == 2) {
    if (f32) return spec ? launch_chunk_t<2, float, kChunk2D, true>(h, w.big32, p, s, write32)
                         : launch_chunk_t<2, float, kChunk2D, false>(h, w.big32, p, s, write32);
    return spec ? launch_chunk_t<2, double, kChunk2D, true>(h, w.big64, p, s, write32)
                : launch_chunk_t<2, double, kChunk2D, false>(h, w.big64, p, s, write32);
  }
  if (f32) return spec ? launch_chunk_t<3, float, kChunk3D32, true>(h, w.big32, p, s, write32)
                       : launch_chunk_t<3, float, kChunk3D32, false>(h, w.big32, p, s, write32);
  return spec ? launch_chunk_t<3, double, kChunk3D64, true>(h, w.big64, p, s, write32)
              : launch_chunk_t<3, double, kChunk3D64, false>(h, w.big64, p, s, write32);
}

int launch_assembly_items(ufem_ns_handle* h, unsigned* over_used, cudaStream_t s) {
  const unsigned blocks = unsigned((h->N + 127) / 128);
  unsigned long long* items = h->d_items;
  auto kernel = h->dim == 2 ? assembly_items_kernel<2> : assembly_items_kernel<3>;
  kernel<<<blocks, 128, 0, s>>>(h->N, h->d_start, h->d_row_inc, h->d_inc_elem, h->d_inc_info, h->d_inc_ea, items,
                                h->d_over, over_used);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

int launch_linearize(ufem_ns_handle* h, cudaStream_t s) {
  const int64_t N = h->N;
  const double* u1 = h->d_hist;
  const double* u2 = h->d_hist + 4 * N;
  const double* u3 = h->d_hist + 8 * N;
  linearize_kernel<<<unsigned((N + 255) / 256), 256, 0, s>>>(N, h->dim, h->d_state, u1, u2, u3, h->d_nu, h->d_uadv,
                                                            h->opt.precision == 1 ? h->d_node32 : nullptr);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

int launch_update(ufem_ns_handle* h, cudaStream_t s) {
  const int64_t N = h->N;
  update_kernel<<<unsigned((N + 255) / 256), 256, 0, s>>>(N, h->dim, h->d_state, h->d_hist, h->d_hist + 4 * N,
                                                        h->d_hist + 8 * N, h->d_sol);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

int launch_build_csr(ufem_ns_handle* h, cudaStream_t s) {
  const int64_t N = h->N;
  build_csr_kernel<<<unsigned((N + 127) / 128), 128, 0, s>>>(N, h->neq, h->d_start, h->d_adj, h->d_rowptr,
                                                           h->d_colidx, h->d_diagpos);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

// Tie rows of linked (periodic) nodes, after the assembly: the element
// contributions at a slave node were assembled into its master's rows and
// columns; the slave's own rows become x_slave - x_master = 0 (identity block
// at the slave, minus identity at the master, rhs 0), so the solution and the
// update give the slave its master's values.
__global__ void tie_rows_kernel(int64_t ntie, int neq, const int32_t* __restrict__ tie,
                                const int64_t* __restrict__ start, const int32_t* __restrict__ adj,
                                double* __restrict__ vals, float* __restrict__ vals32, double* __restrict__ rhs) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= ntie) return;
  const int sl = tie[2 * t], ms = tie[2 * t + 1];
  const int64_t s0 = start[sl];
  const int S = int(start[sl + 1] - s0);
  for (int r = 0; r < neq; ++r) {
    const int64_t rs = int64_t(neq) * neq * s0 + int64_t(r) * S * neq;
    for (int k = 0; k < S; ++k) {
      const int col = adj[s0 + k];
      for (int c = 0; c < neq; ++c) {
        const double v = (c != r) ? 0.0 : (col == sl ? 1.0 : (col == ms ? -1.0 : 0.0));
        vals[rs + k * neq + c] = v;
        if (vals32 != nullptr) vals32[rs + k * neq + c] = float(v);
      }
    }
    rhs[int64_t(sl) * neq + r] = 0.0;
  }
}

int launch_tie_rows(ufem_ns_handle* h, cudaStream_t s, bool write32) {
  if (h->ntie == 0) return UFEM_OK;
  tie_rows_kernel<<<unsigned((h->ntie + 127) / 128), 128, 0, s>>>(h->ntie, h->neq, h->d_tie, h->d_start, h->d_adj,
                                                                  h->d_vals, write32 ? h->d_vals32 : nullptr,
                                                                  h->d_rhs);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

// rhs[dof] += contributions of the constant Neumann faces, in face order.
__global__ void neumann_kernel(int64_t n, const int64_t* __restrict__ dof, const int64_t* __restrict__ ptr,
                               const double* __restrict__ val, double* __restrict__ rhs) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double r = rhs[dof[i]];
  for (int64_t k = ptr[i]; k < ptr[i + 1]; ++k) r = __dadd_rn(r, val[k]);
  rhs[dof[i]] = r;
}

int launch_neumann(ufem_ns_handle* h, cudaStream_t s) {
  const DirichletPlan& bp = h->bcp;
  if (bp.nneu == 0) return UFEM_OK;
  neumann_kernel<<<unsigned((bp.nneu + 255) / 256), 256, 0, s>>>(bp.nneu, bp.neu_dof, bp.neu_ptr, bp.neu_val,
                                                                  h->d_rhs);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

int launch_dirichlet(ufem_ns_handle* h, cudaStream_t s) {
  const DirichletPlan& bp = h->bcp;
  if (bp.nbc == 0) return UFEM_OK;
  const int64_t cb = (bp.nfix_rows * 8 + 255) / 256, rb = (bp.nbc * 8 + 255) / 256;
  dirichlet_kernel<<<unsigned(cb + rb), 256, 0, s>>>(int(cb), bp, h->d_rowptr, h->d_state, h->d_vals, h->d_vals32,
                                                     h->d_rhs, h->d_sol);
  UFEM_CUDA_TRY(cudaGetLastError());
  return UFEM_OK;
}

}  // namespace ufem

namespace ufem {

int launch_mf_residual(ufem_ns_handle* h, double* dx_work, double* res, cudaStream_t s) {
  if (h->ntie > 0)
    return set_error(UFEM_ERR_ARG, "the matrix-free FP64 residual does not support periodic node links");
  const DirichletPlan& bp = h->bcp;
  UFEM_CUDA_TRY(cudaMemcpyAsync(dx_work, h->d_sol, size_t(h->nrows) * 8, cudaMemcpyDeviceToDevice, s));
  if (bp.nbc > 0) {
    mf_columns_kernel<<<unsigned((bp.nbc + 255) / 256), 256, 0, s>>>(bp.nbc, bp.bc_dof, bp.vfirst, dx_work);
    UFEM_CUDA_TRY(cudaGetLastError());
  }
  const bool spec = h->opt.use_specializations != 0;
  int rc;
  if (h->dim == 2)
    rc = spec ? launch_residual_t<2, kChunk2D, true>(h, dx_work, res, s) : launch_residual_t<2, kChunk2D, false>(h, dx_work, res, s);
  else
    rc = spec ? launch_residual_t<3, kChunk3D64, true>(h, dx_work, res, s)
              : launch_residual_t<3, kChunk3D64, false>(h, dx_work, res, s);
  if (rc) return rc;
  if (bp.nneu > 0) {
    neumann_kernel<<<unsigned((bp.nneu + 255) / 256), 256, 0, s>>>(bp.nneu, bp.neu_dof, bp.neu_ptr, bp.neu_val, res);
    UFEM_CUDA_TRY(cudaGetLastError());
  }
  if (bp.nbc > 0) {
    mf_rows_kernel<<<unsigned((bp.nbc + 255) / 256), 256, 0, s>>>(bp.nbc, bp.bc_dof, res);
    UFEM_CUDA_TRY(cudaGetLastError());
  }
  return UFEM_OK;
}

}  // namespace ufem
