// persist.h -- whole Krylov solves in one launch (persist.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

struct ufem_ns_handle;

namespace ufem {

// Scalar slots of a solve's dctl array, shared with the multi-launch solvers.
constexpr int kBnorm = 0, kBeta = 1, kEst = 2, kHnext = 3, kTrue = 4;
constexpr int kRho = 5, kRhoOld = 6, kAlpha = 7, kOmega = 8, kRhV = 9, kTS = 10, kTT = 11, kR2 = 12, kScale = 13;

// Flag slots of ictl used by the persistent solvers beside [0] done, [2] status
// and [3] iterations: whether a barrier wait ran out, and the barrier counter of
// a launch.
constexpr int kFlagLate = 4, kFlagBarrier = 5;

constexpr int kPersistMaxBlocks = 148;
constexpr int kPersistSlots = 8;
constexpr int kPersistPartials = kPersistSlots * kPersistMaxBlocks;
// Polls of a grid barrier (about three seconds) before it gives up.  A constant: read from the
// arguments, the limit cost 4 us an iteration (160 x 160 cells, point Jacobi: 15.1 -> 19.2).
constexpr int kPersistPolls = 1 << 23;
// One solve of A x = b on a node graph (the point-CSR values of the assembled
// system); every vector has N * neq entries.
struct PersistSolve {
  int64_t N = 0;
  int neq = 0;
  const int64_t* start = nullptr;
  const int32_t* adj = nullptr;
  const void* vals = nullptr;  // FP64 or FP32 operator
  bool f32 = false;
  const int64_t* diagpos = nullptr;
  const double* b = nullptr;
  double* x = nullptr;
  // State between launches; r, q and v are also what other blocks gather in the
  // grid form.  BiCGStab: residual, shadow residual, q = p - omega v, v; CG:
  // residual, -, the direction's two buffers.
  double *r = nullptr, *rh = nullptr, *q = nullptr, *v = nullptr;
  // Grid form, two-level: second copies of r and (BiCGStab) q, and A p or A sh, which
  // the restrictions read; point Jacobi: r, q and null.
  double *r2 = nullptr, *q2 = nullptr, *t = nullptr;
  // coarse space of the two-level preconditioners (nc = 0: point Jacobi, or
  // nothing where jacobi is false)
  bool jacobi = true;
  int nc = 0;
  const int32_t* agg = nullptr;
  const int32_t* agg_ptr = nullptr;
  const int32_t* agg_rows = nullptr;
  const double* ainv = nullptr;
  double* cvec = nullptr;  // 2 * nc
  double* yvec = nullptr;  // 2 * nc: the corrections of the two products of an iteration
  double* part = nullptr;  // kPersistPartials block partials (grid form)
  double* dctl = nullptr;
  int* ictl = nullptr;
  double tol = 0.0, alpha_max = 0.0;
  int maxit = 0;
  bool stuck = false;  // the grid barriers' counter starts below 0, so that they run out of time (tests)
};

// Launch plan of a system: the form, its blocks and their shared memory.
enum PersistForm {
  kPersistNone = 0,  // the multi-launch solvers take it
  kPersistCluster,   // one cluster, everything in shared memory
  kPersistGrid,      // a block per SM: values in shared memory as far as they fit
};
struct PersistPlan {
  int form = kPersistNone;
  int blocks = 0;
  size_t smem = 0;
};

// The handle's plan for its FP64 or FP32 operator and nc aggregates of a coarse space,
// made where it is first asked for (a walk over the graph on the host) and kept.
const PersistPlan& persist_plan_of(ufem_ns_handle* h, bool f32, int nc);
// Up to `iters` iterations (first: from the initial residual of x; otherwise
// continuing the stored state).  When the solve ends in this launch, the true
// residual norm is left in dctl[kTrue].
int persist_bicgstab(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s);
int persist_cg(const PersistSolve& a, const PersistPlan& plan, bool first, int iters, cudaStream_t s);

// BiCGStab of `count` systems of the cluster form (device list; the same `blocks` for
// all), one cluster each, from their initial residuals to their end or `iters`
// iterations.  The arithmetic of a solve is persist_bicgstab's.
int persist_bicgstab_members(const PersistSolve* d_list, int count, int neq, bool f32, int blocks, size_t smem,
                             int iters, cudaStream_t s);

}  // namespace ufem
