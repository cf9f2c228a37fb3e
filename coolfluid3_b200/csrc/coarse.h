// coarse.h -- inverses of small dense SPD matrices on the device (the coarse
// matrices of the two-level preconditioners).
#ifndef UFEM_B200_COARSE_H
#define UFEM_B200_COARSE_H

#include <cuda_runtime.h>

namespace ufem {

constexpr int kCoarsePanel = 32;  // rows and columns of a pivot block and of an output tile
inline int coarse_panels(int n) { return (n + kCoarsePanel - 1) / kCoarsePanel; }

// An n x n row-major matrix and its inverse: the panels write the two buffers
// in turn and the last one writes `inv`, so the matrix is put into coarse_source().
struct CoarseInverse {
  double* scratch;  // n * n
  double* inv;      // n * n
  int n;
};
inline double* coarse_source(const CoarseInverse& e) { return coarse_panels(e.n) & 1 ? e.scratch : e.inv; }

// Inverts every matrix of the list on `s` (no synchronisation).  An inverse is
// all zero if a pivot of its matrix is not positive and finite.  Each inverse
// depends on its own matrix alone, bitwise.
int coarse_invert(const CoarseInverse* list, int count, cudaStream_t s);

}  // namespace ufem

#endif
