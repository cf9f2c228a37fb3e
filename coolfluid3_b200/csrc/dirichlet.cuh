// dirichlet.cuh -- the two parts of the symmetric Dirichlet pass, on disjoint rows,
// so one launch runs both (one mesh: assembly.cu, batches: batch.cu).  The columns'
// values, value - old, are formed where they are used.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ufem {

// A row that is not constrained moves its constrained columns to the RHS in
// first-application order (the order of the sequential reference).  Eight lanes
// per row, four rows per warp: the lanes load eight of the row's constrained
// entries at a time, the terms are added to the RHS one by one in
// first-application order (the rounding of the sequential form: no FMA, no
// reassociation), then the lanes zero the entries.  A whole warp calls it.
__device__ __forceinline__ void dirichlet_columns(bool valid, int64_t row, int64_t k0, int len,
                                                  const int64_t* __restrict__ fix_pos,
                                                  const int32_t* __restrict__ fix_bc, const int32_t* __restrict__ bc_at,
                                                  const double* __restrict__ first, const double* __restrict__ state,
                                                  double* __restrict__ vals, float* __restrict__ vals32,
                                                  double* __restrict__ rhs) {
  constexpr unsigned FULL = 0xffffffffu;
  const int sub = int(threadIdx.x & 7), gbase = int(threadIdx.x & 31) & ~7;
  double r = valid ? rhs[row] : 0.0;
  int maxlen = len;  // the warp's longest row: every lane runs the same shuffles
  maxlen = max(maxlen, __shfl_xor_sync(FULL, maxlen, 8));
  maxlen = max(maxlen, __shfl_xor_sync(FULL, maxlen, 16));
  for (int kb = 0; kb < maxlen; kb += 8) {
    const int n = len - kb;  // this row's terms left
    double term = 0.0;
    int64_t pos = -1;
    if (sub < n) {
      pos = fix_pos[k0 + kb + sub];
      const int32_t u = fix_bc[k0 + kb + sub];
      term = __dmul_rn(-vals[pos], __dsub_rn(first[u], state[bc_at[u]]));
    }
    for (int j = 0; j < 8; ++j) {  // added one by one, in first-application order
      const double tj = __shfl_sync(FULL, term, gbase + j);
      if (j < n) r = __dadd_rn(r, tj);
    }
    if (sub < n) {
      vals[pos] = 0.0;
      if (vals32) vals32[pos] = 0.0f;
    }
  }
  if (valid && sub == 0) rhs[row] = r;
}

// Constrained dof u: its row becomes an identity row, rhs = sol = last value - old,
// and vfirst = first value - old (for the matrix-free residual).  Eight lanes: they
// zero the row (the diagonal entry is written 1 in the same pass, so no ordering
// between lanes is needed).
__device__ __forceinline__ void dirichlet_row(int64_t u, const int64_t* __restrict__ bc_dof,
                                              const int32_t* __restrict__ bc_at, const double* __restrict__ first,
                                              const double* __restrict__ last, const int64_t* __restrict__ bc_diag,
                                              const int64_t* __restrict__ rowptr, const double* __restrict__ state,
                                              double* __restrict__ vals, float* __restrict__ vals32,
                                              double* __restrict__ rhs, double* __restrict__ sol,
                                              double* __restrict__ vfirst) {
  const int sub = int(threadIdx.x & 7);
  const int64_t dof = bc_dof[u];
  const int64_t diag = bc_diag[u];
  for (int64_t p = rowptr[dof] + sub; p < rowptr[dof + 1]; p += 8) {
    const double v = (p == diag) ? 1.0 : 0.0;
    vals[p] = v;
    if (vals32) vals32[p] = float(v);
  }
  if (sub == 0) {
    const double old = state[bc_at[u]];
    const double v = __dsub_rn(last[u], old);
    rhs[dof] = v;
    sol[dof] = v;
    vfirst[u] = __dsub_rn(first[u], old);
  }
}

}  // namespace ufem
