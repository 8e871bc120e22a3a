// Shared by the adjoint's translation units.
#pragma once
#include "engine_internal.h"

namespace gbs {

constexpr int kMaxCoefGrad = 32;    // coefficient gradients for stencils of at most this many terms
constexpr int kAdjPartRows = 1024;  // CTAs of a kernel that sums products (one partial row each)
constexpr int kAdjMaxB = 4;         // most adjoint steps per launch

struct AdjGeom {
  long long pitch, plane;  // elements
  int d0, d1, d2, dim, shift, rad;
  int rows, last;          // rows per plane (d0 or d0*d1), cells per row
  long long cells;         // d0*d1*d2
};

// One launch of b steps of the 2-D linear adjoint (adjoint2d.cu).
struct AdjStep2D {
  const AdjGeom *g;
  const void *lam;       // lam_{t+1}
  const void *u;         // u_t; u_{t-l} lies l planes before it (coefficient gradients only)
  void *lam_out, *hg;    // lam_{t+1-b}; the halo's gradient, accumulated
  double *part;          // kAdjPartRows x terms, accumulated (coefficient gradients only)
  const double *coef;    // as the source writes them
  double div;            // the divisor, 1 where there is none
};
using AdjStep2DFn = cudaError_t (*)(const AdjStep2D &, cudaStream_t);
// launchers of one stencil: [coefficient gradients][degree], null where none is built
struct AdjPicks2D {
  AdjStep2DFn step[2][kAdjMaxB + 1];
};
// The stencils whose adjoint step is built: one per set of offsets (j2d5pt is
// star2d1r's, j2d9pt star2d2r's, j2d9pt-gol box2d1r's).
#define GBS_FOR_EACH_ADJ2D(X) X(0) X(1) X(2) X(3) X(4) X(5)
#define GBS_ADJ2D_DECL(id) AdjPicks2D adj2d_picks_##id##_f(); AdjPicks2D adj2d_picks_##id##_d();
GBS_FOR_EACH_ADJ2D(GBS_ADJ2D_DECL)
#undef GBS_ADJ2D_DECL

// dynamic shared memory above which the adjoint's kernels are opted in (48 KB
// is the default, with a kernel's static part)
constexpr size_t kOptInSmem = 40 * 1024;

// CTAs of `kernel` that the current device holds at once (smem: dynamic)
int adj_wave(const void *kernel, int threads, size_t smem);

}  // namespace gbs
