// Engine internals shared by the host-side translation units.
#pragma once
#include <cstdarg>
#include <cstddef>
#include <vector>

#include "../../include/gbstencil.h"
#include "gbs_launch.h"
#include "stencil_defs.h"
#include "stencil_table.cuh"

namespace gbs {

// Device layout of a two-plane grid (see gbs_layout in gbstencil.h).
struct Layout {
  int dim, rad, V;
  size_t esize;
  int dims[3];          // dimsize per axis
  long long shift;      // element offset of column 0
  long long pitch;      // elements per padded innermost row
  long long rows;       // rows per plane
  long long plane;      // elements per plane
  size_t bytes;         // both planes
};

struct Geometry2D {
  int b, wout, nstrips, nblocks, sl;
};

struct Geometry3D {
  int b, tj, jout, wk, ntk, ntj, nblocks, sl;
  int tile;  // the tensor-map tile kernel (its copies are bounds-checked by the hardware)
};
// Tile shape of the 3-D launcher of degree b: computed rows, valid rows and
// valid columns per tile, and whether it is the tensor-map tile kernel.
struct Tile3DShape {
  int tj, jout, wk, tile;
};
Tile3DShape tile_shape_3d(int sid, int dtype, int fma, int b, int variant);
// block-shape variant of the 3-D launcher of degree b for d: the one whose
// tile rows equal d->bs1, else the tuning table's, else variant 0; -1 (and
// an error recorded) when d->bs1 names no built shape
int variant_3d(const gbs_desc *d, int b);
Geometry3D geometry3d(const Layout &L, int b, const Tile3DShape &ts, int sl_req, long long resident_ctas);
gbs_status validate3d(const Layout &L, const Geometry3D &g);
long long resident_ctas_3d(int sid, int dtype, int fma, int b, int variant);

gbs_status fail(gbs_status st, const char *fmt, ...);
gbs_status cuda_fail(cudaError_t e, const char *what);
const gbs_stencil_def_t *stencil_def(int sid);
gbs_status check_desc(const gbs_desc *d);
Layout make_layout(const gbs_desc *d);
std::vector<int> split_steps(int T, int bt);
// The launches of d's time loop at degree bt: split_steps, but for odd T the
// last launch takes the steps that the degree of tuned_last would give it.
std::vector<int> loop_steps(const gbs_desc *d, int bt);
int sm_count();
// rows per stream block of a 2-D launch of nstrips strips over ni rows whose
// blocks overlap by br rows at each end; resident_warps: warps the GPU holds at
// once for this kernel (0 = unknown)
int stream_rows_2d(int nstrips, int ni, int br, bool f64, long long resident_warps);
Geometry2D geometry2d(const Layout &L, int b, int sl_req, long long resident_warps);
long long resident_warps_2d(int sid, int dtype, int fma, int b);
// rows per stream block of a 2-D grid's launches of degree b where many grids'
// launches share the GPU
int shared_rows_2d(const gbs_desc *d, const Layout &L, int b);
// output columns per strip of the 2-D kernels (Pipe2D::WOUT): the window loses
// b*r columns on the right and b*r rounded up to whole lanes on the left
inline int wout2d(int rad, int b, int V) {
  const int left = (b * rad + V - 1) / V * V;
  return (32 * V - left - b * rad) / V * V;
}
gbs_status validate2d(const Layout &L, const Geometry2D &g);
gbs_status error_word(int **out);
gbs_status run_loop(const gbs_desc *d, const Layout &L, void *dev_A, cudaStream_t stream, int *err);
// One kernel launch of b fused steps, planned: everything but its planes.
struct BlockPlan {
  int dim;
  Launch2D a2;
  Launch2DFn f2;
  Launch3D a3;
  Launch3DFn f3;
};
// `coef` must outlive the plan. stash: the launch also stores the states after
// 1 .. b-1 steps (interior cells) to the planes stash, stash + plane, ... (2-D
// grids)
gbs_status plan_block(const gbs_desc *d, const Layout &L, const double *coef, double div, double eps, int sl, int b,
                      bool stash, int *err, BlockPlan *out);
gbs_status launch_plan(BlockPlan &plan, const void *src, void *dst, void *stash, cudaStream_t stream);
gbs_status launch_block(const gbs_desc *d, const Layout &L, const double *coef, double div, double eps, int sl,
                        int b, const void *src, void *dst, cudaStream_t stream, int *err);
// the layered batched launchers of a stencil (Picks::lb) and their row costs
const Picks &batch_picks(int sid, int fma);
int max_bt(int sid, int dtype, int fma);
// the tuning table's (bt, sl) for d's stencil, dtype, mode and size class
bool tuned_lookup(const gbs_desc *d, int *bt, int *sl, int *bs1 = nullptr);
// the degree that fixes the last launch's steps of a loop of odd T for d's
// stencil, dtype, mode and size class (0: no entry); see loop_steps
int tuned_last(const gbs_desc *d);
bool div_proven_exact(double d);

}  // namespace gbs
