// Adjoint (reverse-mode gradient) of the stencil time loop.
//
// No counterpart in the artifact: it differentiates the time loop that
// kernel_stencil runs. For u_{t+1} = F(u_t) on the interior (halo fixed)
// and a loss L(u_T) whose gradient lam_T = dL/du_T the caller supplies, it
// returns dL/du_0 (interior and halo) and, on request, dL/dc_k for the
// coefficients as the source writes them (before any divisor).
//
// Linear stencils, u_{t+1}(x) = sum_k c_k u_t(x + o_k) / d:
//  * lam_t(y) = sum_k c_k/d lam_{t+1}(y - o_k) on the interior, zero on the
//    halo. Every offset set in the catalogue is symmetric (o in the set iff
//    -o is), so this is the forward stencil with each coefficient moved to
//    the mirrored offset: the engine's own kernels run it (FMA mode), one
//    launch per step from one lam plane to the other.
//  * a halo cell h feeds every step: dL/du_0(h) = sum_t sum_k c_k/d
//    lam_{t+1}(h - o_k), accumulated by a kernel over the halo cells only.
//  * dL/dc_k = sum_t sum_x lam_{t+1}(x) u_t(x + o_k) / d needs the forward
//    states: only then are they recomputed (below), and a streaming kernel
//    accumulates the products per thread and reduces them per CTA into a
//    partial buffer (no atomics; summed in double at the end).
// gradient2d, u_{t+1} = u + c q, q = (eps + s)^{-1/2}, s = sum_n (u - u_{x+n})^2:
//    the linearised update, dF(x)/du(x) = 1 - c q^3 sum_n d_n(x),
//    dF(x)/du(x+n) = c q^3 d_n(x), dF(x)/dc = q(x), evaluated on u_t, whose
//    transpose one streaming pass applies.
//
// Checkpointing: gbs_adjoint_forward advances the grid and saves u_t every
// C steps into the caller's workspace. When the states are needed,
// gbs_adjoint_backward walks the chunks backwards and recomputes a chunk's C
// states from its checkpoint with the forward engine (one launch per step,
// each into its own stash slot), then runs the chunk's adjoint steps. With
// fewer than 2C stash slots (a smaller memory budget) each chunk is
// reversed by the binomial (revolve) schedule instead: a recursion that
// advances from the newest stored state into a free slot, reverses the
// right part with one slot fewer and then the left part, which is the
// fewest forward steps any schedule with that many slots can take (Griewank
// and Walther, ACM TOMS 26(1), 2000, Algorithm 799).
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <map>
#include <mutex>
#include <cstring>
#include <vector>

#include "adjoint_internal.h"
#include "gbs_device.cuh"

namespace gbs {
namespace {

constexpr int kAdjThreads = 256;
__device__ __forceinline__ long long cell_off(const AdjGeom &g, int i, int j, int k) {
  return g.dim == 2 ? (long long)i * g.pitch + g.shift + j
                    : ((long long)i * g.d1 + j) * g.pitch + g.shift + k;
}

// (i, j) of row r; for 2-D rows j = 0 and the column is the second index
__device__ __forceinline__ void row_ij(const AdjGeom &g, int r, int &i, int &j) {
  if (g.dim == 2) {
    i = r;
    j = 0;
  } else {
    i = r / g.d1;
    j = r - i * g.d1;
  }
}

__device__ __forceinline__ bool row_interior(const AdjGeom &g, int i, int j) {
  const int R = g.rad;
  return i >= R && i < g.d0 - R && (g.dim == 2 || (j >= R && j < g.d1 - R));
}

template <typename T, int NT> struct LinCoef {
  T c[NT];  // c_k / d
};

// Halo cells, enumerated without touching the interior:
//  A: the 2R edge columns of every interior row, one thread per cell;
//  B: every cell of the all-halo rows, one warp per 32-column segment.
// All-halo rows: 2-D rows i < R or i >= d0 - R; 3-D the planes i < R or
// i >= d0 - R (every row j), then the rows j < R or j >= d1 - R of each
// interior plane.
struct HaloPlan {
  long long na;      // A cells, rounded up to whole warps
  long long rows_b;  // all-halo rows
  int nseg;          // 32-column segments per row
};

__host__ __device__ inline HaloPlan halo_plan(const AdjGeom &g) {
  HaloPlan h{};
  const int R = g.rad;
  const long long inner_rows = g.dim == 2 ? (long long)(g.d0 - 2 * R) : (long long)(g.d0 - 2 * R) * (g.d1 - 2 * R);
  h.na = (inner_rows * 2 * R + 31) / 32 * 32;
  h.rows_b = (long long)g.rows - inner_rows;
  h.nseg = (g.last + 31) / 32;
  return h;
}

// halo cell number tid of the enumeration above: (i, j, c); false past the end
__device__ __forceinline__ bool halo_cell(const AdjGeom &g, const HaloPlan &hp, long long tid, int &i, int &j,
                                          int &c) {
  const int R = g.rad;
  j = 0;
  if (tid < hp.na) {
    const long long row = tid / (2 * R);
    const int e = (int)(tid - row * 2 * R);
    if (g.dim == 2) {
      if (row >= g.d0 - 2 * R) return false;
      i = R + (int)row;
    } else {
      const int w1 = g.d1 - 2 * R;
      if (row >= (long long)(g.d0 - 2 * R) * w1) return false;
      i = R + (int)(row / w1);
      j = R + (int)(row - (long long)(i - R) * w1);
    }
    c = e < R ? e : g.last - 2 * R + e;
    return true;
  }
  const long long b = tid - hp.na;
  const long long wrow = (b >> 5) / hp.nseg;
  const int seg = (int)((b >> 5) - wrow * hp.nseg);
  if (wrow >= hp.rows_b) return false;
  c = seg * 32 + (int)(b & 31);
  if (c >= g.last) return false;
  if (g.dim == 2) {
    i = wrow < R ? (int)wrow : g.d0 - 2 * R + (int)wrow;
  } else {
    const long long full = 2LL * R * g.d1;  // rows of the all-halo planes
    if (wrow < full) {
      const int p = (int)(wrow / g.d1);
      i = p < R ? p : g.d0 - 2 * R + p;
      j = (int)(wrow - (long long)p * g.d1);
    } else {
      const long long q = wrow - full;
      i = R + (int)(q / (2 * R));
      const int jj = (int)(q - (long long)(i - R) * 2 * R);
      j = jj < R ? jj : g.d1 - 2 * R + jj;
    }
  }
  return true;
}

// hg(h) += sum_k c_k/d lam(h - o_k) for every halo cell h of a 3-D grid (2-D
// stencils of many terms too). lam is zero off the interior, so only the
// offsets that lead there are read: which planes, rows and columns around the
// cell are interior is found once, not per term. A face cell of a radius-1 box
// reads 9 of its 27 neighbours; with every term bounds-checked and read, the
// pass took longer than the step itself (j3d27pt f32, four instances of
// 96..192 cells a side at once: 22 us a pass, 9.8 now).
template <class ST, typename T>
__global__ void __launch_bounds__(kAdjThreads) halo_kernel(const __grid_constant__ AdjGeom g, const T *lam, T *hg,
                                                           const __grid_constant__ LinCoef<T, ST::kTerms> cf) {
  constexpr int R = ST::kRad, W = 2 * R + 1;
  const HaloPlan hp = halo_plan(g);
  int i, j, c;
  if (!halo_cell(g, hp, (long long)blockIdx.x * kAdjThreads + threadIdx.x, i, j, c)) return;
  // 2-D offsets are (row, column); 3-D (plane, row, column)
  bool pi[W], pj[W], pc[W];
  static_for<W>([&](auto XI) GBS_INL {
    constexpr int x = decltype(XI)::value - R;
    pi[x + R] = i + x >= R && i + x < g.d0 - R;
    pj[x + R] = ST::kDim == 2 || (j + x >= R && j + x < g.d1 - R);
    pc[x + R] = c + x >= R && c + x < g.last - R;
  });
  const long long line = ST::kDim == 2 ? g.pitch : (long long)g.d1 * g.pitch;  // elements per step of i
  const long long o = (ST::kDim == 2 ? (long long)i * g.pitch : ((long long)i * g.d1 + j) * g.pitch) + g.shift + c;
  T acc = T(0);
  static_for<ST::kTerms>([&](auto TI) GBS_INL {
    constexpr int t = decltype(TI)::value;
    constexpr int di = ST::kOff[t][0], dj = ST::kDim == 2 ? 0 : ST::kOff[t][1];
    constexpr int dk = ST::kDim == 2 ? ST::kOff[t][1] : ST::kOff[t][2];
    const bool in = pi[R - di] && pj[R - dj] && pc[R - dk];
    const T l = in ? lam[o - di * line - dj * g.pitch - dk] : T(0);
    acc = fma(cf.c[t], l, acc);
  });
  hg[o] += acc;
}

// part[blockIdx.x][k] += sum over interior x of lam(x) u(x + o_k) / d.
// Work units of one warp: (interior row, 128-column segment), four
// independent columns per lane in flight; products summed per thread in T,
// reduced per CTA in double.
template <class ST, typename T>
__global__ void __launch_bounds__(kAdjThreads) coef_kernel(const __grid_constant__ AdjGeom g, const T *lam, const T *u,
                                                           double *part, T inv_div) {
  constexpr int NT = ST::kTerms;
  constexpr int SEG = 128;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int R = g.rad;
  const int width = g.last - 2 * R;
  const long long nseg = (width + SEG - 1) / SEG;
  const long long units = (long long)g.rows * nseg;
  const long long nwarps = ((long long)gridDim.x * kAdjThreads) >> 5;
  T acc[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t] = T(0);
  for (long long un = ((long long)blockIdx.x * kAdjThreads + threadIdx.x) >> 5; un < units; un += nwarps) {
    const int r = (int)(un / nseg), seg = (int)(un - (long long)r * nseg);
    int i, j;
    row_ij(g, r, i, j);
    if (!row_interior(g, i, j)) continue;
    const long long row = (ST::kDim == 2 ? (long long)i * g.pitch : ((long long)i * g.d1 + j) * g.pitch) + g.shift;
    const int c0 = R + seg * SEG + lane;
    T l[SEG / 32];
    bool in[SEG / 32];
#pragma unroll
    for (int q = 0; q < SEG / 32; ++q) {
      const int c = c0 + 32 * q;
      in[q] = c < g.last - R;
      l[q] = in[q] ? lam[row + c] : T(0);
    }
    static_for<NT>([&](auto TI) {
      constexpr int t = decltype(TI)::value;
      constexpr int di = ST::kOff[t][0], dj = ST::kOff[t][1], dk = ST::kOff[t][2];
      const long long o = ST::kDim == 2 ? (long long)di * g.pitch + dj : ((long long)di * g.d1 + dj) * g.pitch + dk;
#pragma unroll
      for (int q = 0; q < SEG / 32; ++q)
        if (in[q]) acc[t] = fma(l[q], u[row + c0 + 32 * q + o], acc[t]);
    });
  }
  __shared__ double red[kAdjThreads / 32][NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    T v = acc[t];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
    if (lane == 0) red[w][t] = (double)v;
  }
  __syncthreads();
  if (threadIdx.x < NT) {
    double s = 0.0;
#pragma unroll
    for (int ww = 0; ww < kAdjThreads / 32; ++ww) s += red[ww][threadIdx.x];
    part[(size_t)blockIdx.x * NT + threadIdx.x] += s * (double)inv_div;
  }
}

// gradient2d adjoint step, one pass over u_t and lam_{t+1}:
//   lam_t(y) = lam(y) + sum_x (w(x) + w(y)) (u(x) - u(y)),  w = num q^3 lam,
// over y's four neighbours x, w = 0 on the halo (the transposed linearised
// Jacobian: -w(y) sum_n d_n(y) and the neighbours' c q^3 d_n share their
// differences). A term belongs to the edge between two cells and enters both
// with opposite sign, so each edge's difference, square and flux is formed
// once. At a halo cell the same sum is the increment of its gradient. An edge
// without an interior end has no term: its difference is set to 0 before it
// meets w + w = 0, for its states may be infinite or NaN.
//
// A warp owns a strip of output columns and a block of output rows and
// streams the rows of u and lam like the 2-D stencil kernels: every lane
// copies its own 16 bytes of each row into a ring in shared memory (cp.async)
// groups ahead of use. At step p, row p-1 gets its q and w, row p-2 its
// result; row p's differences with row p-1 stay in registers. In-row
// neighbours come by shuffles.
//
// Bound for double: the FP64 pipe, 25 operations a cell. The two passes this
// replaced (q and sum of differences to memory, then a gather) took about 60.
// With the forward step's shared squares: forward and gradient of f64
// 1024x1100, T=64, 18.7 -> 11.2 ms (GB300).
template <class ST, typename T> struct GradPipe {
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int COLS = 32 * V;
  static constexpr int ML = (2 + V - 1) / V * V;             // window columns left of the outputs
  static constexpr int WOUT = (COLS - ML - 2) / V * V;       // output columns per strip
  static constexpr int NPH = 3, PG = 2;                      // rows per group, groups in flight
  static constexpr unsigned ROWB = 1024;                     // ring row: u, then lam
  static constexpr unsigned GROUP = NPH * ROWB, RING = (PG + 1) * GROUP;
};
constexpr int kGradWarps = 4;

template <class ST, typename T>
__global__ void __launch_bounds__(kGradWarps * 32)
    grad2d_kernel(const __grid_constant__ AdjGeom g, const T *u, const T *lam, T *lam_out, T *hg, double *part, T num,
                  T eps, int want_coef, int nstrips, int nblocks, int sl, long long item0) {
  using GP = GradPipe<ST, T>;
  using A = Arith<T>;
  constexpr int V = GP::V, R = 1, NPH = GP::NPH, PG = GP::PG;
  static_assert(ST::kKind != KIND_GRADIENT || ST::kRad == 1, "radius 1");
  __shared__ __align__(128) unsigned char smem[kGradWarps * GP::RING];
  __shared__ double red[kGradWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long gw = item0 + (long long)blockIdx.x * kGradWarps + wid;
  double pnum = 0.0;
  if (gw < (long long)nstrips * nblocks) {
    const int strip = (int)(gw % nstrips), blk = (int)(gw / nstrips);
    const int cs = R + strip * GP::WOUT, ce = min(cs + GP::WOUT, g.d1 - R);
    const int own_lo = strip == 0 ? 0 : cs, own_hi = strip == nstrips - 1 ? g.d1 : ce;
    const int el = cs + g.shift - GP::ML + lane * V;
    const int col0 = el - g.shift;
    const bool in_row = el >= 0 && el + V <= g.pitch;
    const bool edge = cs - GP::ML < R || cs - GP::ML + GP::COLS > g.d1 - R;
    bool inner[V], hedge[V], sum_col[V];  // hedge: an end of the edge to column e + 1 is an interior column
    bool whole = true;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int c = col0 + e;
      inner[e] = c >= R && c < g.d1 - R;
      hedge[e] = c >= R - 1 && c < g.d1 - R;
      sum_col[e] = c >= cs && c < ce;
      whole = whole && sum_col[e];
    }
    const int i0 = R + blk * sl, i1 = min(i0 + sl, g.d0 - R);
    const int o0 = blk == 0 ? 0 : i0, o1 = blk == nblocks - 1 ? g.d0 : i1;  // result rows
    const int pstart = max(0, o0 - 2), pend = min(g.d0, o1 + 2);
    const int ng = (o1 + 2 - pstart + NPH - 1) / NPH;

    unsigned char *my = smem + (size_t)wid * GP::RING + lane * 16;
    const uint32_t my_s = smem_u32(my);
    long long ld = (long long)pstart * g.pitch + el;
    int ld_left = pend - pstart;
    unsigned wr = 0, rd = 0;
    auto request_group = [&]() GBS_INL {
#pragma unroll
      for (int ph = 0; ph < NPH; ++ph) {
        if (in_row && ph < ld_left) {
          cp_async16(my_s + wr + ph * GP::ROWB, u + ld);
          cp_async16(my_s + wr + ph * GP::ROWB + 512, lam + ld);
        }
        ld += g.pitch;
      }
      cp_async_commit();
      ld_left -= NPH;
      wr = wr + GP::GROUP == GP::RING ? 0u : wr + GP::GROUP;
    };
#pragma unroll 1
    for (int k = 0; k < PG; ++k) request_group();

    // rows p-1 (u1, l1), its differences with row p-2 (dv, their squares sv),
    // row p-2's w and its result but for the edge to row p-1
    T u1[V], l1[V], dv[V], sv[V], w2[V], acc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) u1[e] = l1[e] = dv[e] = sv[e] = w2[e] = acc[e] = T(0);
    int p = pstart;
#pragma unroll 1
    for (int k = 0; k < ng; ++k) {
      request_group();
      cp_async_wait<PG>();
      static_for<NPH>([&](auto PHI) GBS_INL {
        constexpr int ph = decltype(PHI)::value;
        const int pp = p + ph;
        T x[V], lx[V];
        ld_vec<T, V>(x, reinterpret_cast<const T *>(my + rd + ph * GP::ROWB));
        ld_vec<T, V>(lx, reinterpret_cast<const T *>(my + rd + ph * GP::ROWB + 512));
        const bool row_in = pp - 1 >= R && pp - 1 < g.d0 - R;  // row p-1 is interior
        const bool vedge = pp >= R && pp - 1 < g.d0 - R;       // row p-1 or row p is
        const bool rim = edge || !row_in;
        // horizontal edges of row p-1 (e: between columns e and e+1)
        T dh[V], sh[V];
        const T after = row_elem<V, V>(u1);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          dh[e] = A::sub(e + 1 < V ? u1[e + 1 < V ? e + 1 : e] : after, u1[e]);
          if (rim) dh[e] = row_in && hedge[e] ? dh[e] : T(0);
          sh[e] = A::mul(dh[e], dh[e]);
        }
        const T sleft = shfl_up(sh[V - 1], 1);
        T dn[V], sn[V], w1[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          dn[e] = A::sub(x[e], u1[e]);
          if (rim) dn[e] = vedge && inner[e] ? dn[e] : T(0);
          sn[e] = A::mul(dn[e], dn[e]);
          const T s = A::add(A::add(A::add(A::add(eps, sv[e]), sn[e]), sh[e]), e > 0 ? sh[e > 0 ? e - 1 : 0] : sleft);
          const bool in = row_in && inner[e];
          const T lv = in ? l1[e] : T(0);
          T y, res;
          rsqrt_split(s, y, res);
          const T w = rsqrt_cube(A::mul(num, lv), y, res);
          w1[e] = in ? w : T(0);
          l1[e] = lv;
          if (want_coef && in && sum_col[e] && pp - 1 >= i0 && pp - 1 < i1)
            pnum += (double)A::mul(lv, rsqrt_of(y, res));
        }
        // fluxes: horizontal edges of row p-1, vertical edges between rows p-2 and p-1
        const T wafter = row_elem<V, V>(w1);
        T fh[V], out[V];
#pragma unroll
        for (int e = 0; e < V; ++e) fh[e] = A::mul(A::add(w1[e], e + 1 < V ? w1[e + 1 < V ? e + 1 : e] : wafter), dh[e]);
        const T fleft = shfl_up(fh[V - 1], 1);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const T fv = A::mul(A::add(w2[e], w1[e]), dv[e]);
          out[e] = A::add(acc[e], fv);
          acc[e] = A::add(l1[e], A::sub(A::sub(fh[e], e > 0 ? fh[e > 0 ? e - 1 : 0] : fleft), fv));
          w2[e] = w1[e];
          dv[e] = dn[e];
          sv[e] = sn[e];
          u1[e] = x[e];
          l1[e] = lx[e];
        }
        const int q = pp - 2;  // the row whose result is complete
        if (q >= o0 && q < o1) {
          const long long o = (long long)q * g.pitch + el;
          const bool in_rows = q >= R && q < g.d0 - R;
          if (whole && in_rows) {
            st_vec_global<T, V>(lam_out + o, out);
          } else {
#pragma unroll
            for (int e = 0; e < V; ++e) {
              const int c = col0 + e;
              if (c < own_lo || c >= own_hi) continue;
              if (in_rows && inner[e]) lam_out[o + e] = out[e];
              else hg[o + e] += out[e];
            }
          }
        }
      });
      p += NPH;
      rd = rd + GP::GROUP == GP::RING ? 0u : rd + GP::GROUP;
    }
    cp_async_wait<0>();
  }
  if (want_coef) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pnum += __shfl_down_sync(0xffffffffu, pnum, o);
    if (lane == 0) red[wid] = pnum;
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < kGradWarps; ++k) sum += red[k];
      part[blockIdx.x] += sum;
    }
  }
}

// The halo cells of `planes` planes, `stride` elements apart, from src (the
// fixed boundary of recomputed states: launches never write it).
template <typename T>
__global__ void __launch_bounds__(kAdjThreads) copy_halo_kernel(const __grid_constant__ AdjGeom g, const T *src, T *dst,
                                                                long long stride) {
  const HaloPlan hp = halo_plan(g);
  int i, j, c;
  if (!halo_cell(g, hp, (long long)blockIdx.x * kAdjThreads + threadIdx.x, i, j, c)) return;
  const long long o = g.dim == 2 ? cell_off(g, i, c, 0) : cell_off(g, i, j, c);
  dst[(long long)blockIdx.y * stride + o] = src[o];
}

// zero the halo of a plane (lam_T's halo carries no gradient)
template <typename T>
__global__ void zero_halo_kernel(T *x, AdjGeom g) {
  const long long c = (long long)blockIdx.x * kAdjThreads + threadIdx.x;
  if (c >= g.cells) return;
  int i, j, k = 0;
  if (g.dim == 2) {
    i = (int)(c / g.d1);
    j = (int)(c % g.d1);
  } else {
    i = (int)(c / ((long long)g.d1 * g.d2));
    const long long r = c % ((long long)g.d1 * g.d2);
    j = (int)(r / g.d2);
    k = (int)(r % g.d2);
  }
  const int R = g.rad;
  const bool interior = i >= R && i < g.d0 - R && j >= R && j < g.d1 - R && (g.dim == 2 || (k >= R && k < g.d2 - R));
  if (!interior) x[cell_off(g, i, j, k)] = T(0);
}

// grad_u0 = lam_0 on the interior, the accumulated halo gradient on the halo
template <typename T>
__global__ void combine_kernel(const T *lam0, const T *hg, T *out, AdjGeom g) {
  const long long c = (long long)blockIdx.x * kAdjThreads + threadIdx.x;
  if (c >= g.cells) return;
  int i, j, k = 0;
  if (g.dim == 2) {
    i = (int)(c / g.d1);
    j = (int)(c % g.d1);
  } else {
    i = (int)(c / ((long long)g.d1 * g.d2));
    const long long r = c % ((long long)g.d1 * g.d2);
    j = (int)(r / g.d2);
    k = (int)(r % g.d2);
  }
  const int R = g.rad;
  const bool interior = i >= R && i < g.d0 - R && j >= R && j < g.d1 - R && (g.dim == 2 || (k >= R && k < g.d2 - R));
  const long long o = cell_off(g, i, j, k);
  out[o] = interior ? lam0[o] : hg[o];
}

__global__ void sum_parts_kernel(const double *part, int nblocks, int nt, double *out) {
  const int t = blockIdx.x;
  double s = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += part[(size_t)b * nt + t];
  __shared__ double red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[t] = red[0];
}

// ---------------------------------------------------------------------------
// workspace
// ---------------------------------------------------------------------------
struct Workspace {
  int ncp, C, nblocks, nt;
  int slots;            // stash planes: 2C (two chunk buffers) or fewer (revolve)
  bool revolve;         // chunks reversed by the binomial schedule
  size_t plane_bytes;
  size_t off_cp, off_stash, off_lam, off_hg, off_part, total;
};

// The stash holds two chunk buffers of C planes when slots >= 2C; with fewer
// slots it holds `slots` snapshot planes plus two work planes of the
// binomial schedule.
Workspace workspace_of(const gbs_desc *d, const Layout &L, int C, int slots) {
  Workspace w{};
  const gbs_stencil_def_t *s = stencil_def(d->stencil);
  w.C = C;
  w.ncp = (d->timestep + C - 1) / C;
  if (w.ncp < 1) w.ncp = 1;
  w.revolve = slots < 2 * C;
  w.slots = w.revolve ? slots : 2 * C;
  w.plane_bytes = (size_t)L.plane * L.esize;
  w.nblocks = kAdjPartRows;
  w.nt = s->kind == 1 ? 1 : std::min(s->nterms, kMaxCoefGrad);
  w.off_cp = 0;
  w.off_stash = w.off_cp + (size_t)w.ncp * w.plane_bytes;
  w.off_lam = w.off_stash + (size_t)(w.revolve ? w.slots + 2 : 2 * C) * w.plane_bytes;
  w.off_hg = w.off_lam + 2 * w.plane_bytes;
  // gradient2d: two planes more than its step needs, so that a workspace or a
  // budget holds as many checkpoints and slots as it did when that step kept
  // per-cell values between two passes
  w.off_part = w.off_hg + (s->kind == 1 ? 3 : 1) * w.plane_bytes;
  w.total = w.off_part + (size_t)w.nblocks * w.nt * sizeof(double) + 256;
  return w;
}

AdjGeom geom_of(const Layout &L) {
  AdjGeom g{};
  g.pitch = L.pitch;
  g.plane = L.plane;
  g.d0 = L.dims[0];
  g.d1 = L.dims[1];
  g.d2 = L.dims[2];
  g.dim = L.dim;
  g.shift = (int)L.shift;
  g.rad = L.rad;
  g.rows = (int)L.rows;
  g.last = L.dims[L.dim - 1];
  g.cells = (long long)L.dims[0] * L.dims[1] * L.dims[2];
  return g;
}

// coefficients of the forward update as the source writes them, divisor and eps
void forward_coefficients(const gbs_desc *d, std::vector<double> &coef, double &div, double &eps) {
  const gbs_stencil_def_t *s = stencil_def(d->stencil);
  const int nt = s->kind == 1 ? 1 : s->nterms;
  coef.assign(nt, 0.0);
  for (int t = 0; t < nt; ++t) {
    double c;
    if (d->coef) c = d->dtype == GBS_F64 ? ((const double *)d->coef)[t] : ((const float *)d->coef)[t];
    else c = s->kind == 1 ? (double)s->numerator : (double)s->terms[t].coef;
    coef[t] = c;
  }
  div = d->divisor != 0.0 ? d->divisor : (double)s->divisor;
  eps = d->eps != 0.0 ? d->eps : (double)s->eps;
}

// the forward coefficient of the mirrored offset, per term (linear stencils)
bool transposed_coefficients(const gbs_stencil_def_t *s, const std::vector<double> &coef, std::vector<double> &out) {
  out.assign(s->nterms, 0.0);
  for (int t = 0; t < s->nterms; ++t) {
    int m = -1;
    for (int u = 0; u < s->nterms; ++u)
      if (s->terms[u].di == -s->terms[t].di && s->terms[u].dj == -s->terms[t].dj &&
          s->terms[u].dk == -s->terms[t].dk)
        m = u;
    if (m < 0) return false;
    out[t] = coef[m];
  }
  return true;
}

// kernels of one stencil and dtype
struct AdjKernels {
  cudaError_t (*halo)(const AdjGeom &, const void *, void *, const std::vector<double> &, double, cudaStream_t);
  cudaError_t (*coef)(const AdjGeom &, const void *, const void *, double *, double, cudaStream_t);
  cudaError_t (*grad)(const AdjGeom &, const void *, const void *, void *, void *, double *, double, double, bool,
                      cudaStream_t);
};

// one thread per halo cell of the interior rows, one warp per segment of an all-halo row
unsigned halo_grid(const AdjGeom &g) {
  const HaloPlan h = halo_plan(g);
  const long long threads = h.na + h.rows_b * h.nseg * 32;
  return (unsigned)std::max<long long>(1, (threads + kAdjThreads - 1) / kAdjThreads);
}

// the halo of `planes` consecutive planes at dst from the plane src
cudaError_t copy_halo(int dtype, const AdjGeom &g, const void *src, void *dst, int planes, cudaStream_t s) {
  for (int k = 0; k < planes; k += 32768) {  // grid.y is at most 65535
    const dim3 grid(halo_grid(g), (unsigned)std::min(planes - k, 32768));
    if (dtype == GBS_F64)
      copy_halo_kernel<double><<<grid, kAdjThreads, 0, s>>>(g, (const double *)src, (double *)dst + (size_t)k * g.plane,
                                                            g.plane);
    else
      copy_halo_kernel<float><<<grid, kAdjThreads, 0, s>>>(g, (const float *)src, (float *)dst + (size_t)k * g.plane,
                                                           g.plane);
  }
  return cudaGetLastError();
}

template <class ST, typename T>
cudaError_t run_halo(const AdjGeom &g, const void *lam, void *hg, const std::vector<double> &coef, double div,
                     cudaStream_t s) {
  if constexpr (ST::kKind == KIND_GRADIENT) {
    return cudaErrorInvalidValue;
  } else {
    LinCoef<T, ST::kTerms> cf;
    const double dv = ST::kHasDiv ? div : 1.0;
    for (int t = 0; t < ST::kTerms; ++t) cf.c[t] = (T)(coef[t] / dv);
    return launch_kernel(halo_kernel<ST, T>, halo_grid(g), kAdjThreads, 0, s, g, static_cast<const T *>(lam),
                         static_cast<T *>(hg), cf);
  }
}

template <class ST, typename T>
cudaError_t run_coef(const AdjGeom &g, const void *lam, const void *u, double *part, double div, cudaStream_t s) {
  if constexpr (ST::kKind == KIND_GRADIENT || ST::kTerms > kMaxCoefGrad) {
    return cudaErrorInvalidValue;
  } else {
    const double dv = ST::kHasDiv ? div : 1.0;
    const int wave = std::min(kAdjPartRows, adj_wave(reinterpret_cast<const void *>(coef_kernel<ST, T>), kAdjThreads, 0));
    return launch_kernel(coef_kernel<ST, T>, (unsigned)wave, kAdjThreads, 0, s, g, static_cast<const T *>(lam),
                         static_cast<const T *>(u), part, (T)(1.0 / dv));
  }
}

template <class ST, typename T>
cudaError_t run_grad(const AdjGeom &g, const void *u, const void *lam, void *lam_out, void *hg, double *part,
                     double num, double eps, bool want_coef, cudaStream_t s) {
  if constexpr (ST::kKind != KIND_GRADIENT) {
    return cudaErrorInvalidValue;
  } else {
    using GP = GradPipe<ST, T>;
    const int ni = g.d0 - 2, nstrips = (g.d1 - 2 + GP::WOUT - 1) / GP::WOUT;
    const int wave = adj_wave(reinterpret_cast<const void *>(grad2d_kernel<ST, T>), kGradWarps * 32, 0);
    int sl = stream_rows_2d(nstrips, ni, 2, sizeof(T) == 8, (long long)wave * kGradWarps);
    // with the sum for num every CTA has its own row of the partial-sum table:
    // blocks as long as that takes, and where one block per strip is still too
    // many (more than 4096 strips), several launches over the items
    constexpr long long kMost = (long long)kAdjPartRows * kGradWarps;
    while (sl < ni && (long long)nstrips * ((ni + sl - 1) / sl) > kMost) ++sl;
    const int nblocks = (ni + sl - 1) / sl;
    const long long items = (long long)nstrips * nblocks, most = want_coef ? kMost : items;
    for (long long item0 = 0; item0 < items; item0 += most) {
      const unsigned grid = (unsigned)((std::min(most, items - item0) + kGradWarps - 1) / kGradWarps);
      const cudaError_t e =
          launch_kernel(grad2d_kernel<ST, T>, grid, kGradWarps * 32, 0, s, g,
                        static_cast<const T *>(u), static_cast<const T *>(lam), static_cast<T *>(lam_out),
                        static_cast<T *>(hg), part, (T)num, (T)eps, want_coef ? 1 : 0, nstrips, nblocks, sl, item0);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
}

AdjKernels adj_kernels(int sid, int dtype) {
  switch (sid) {
#define GBS_ADJ(id, S)                                                               \
  case id:                                                                            \
    return dtype == GBS_F64                                                          \
               ? AdjKernels{&run_halo<S, double>, &run_coef<S, double>, &run_grad<S, double>} \
               : AdjKernels{&run_halo<S, float>, &run_coef<S, float>, &run_grad<S, float>};
    GBS_FOR_EACH_STENCIL(GBS_ADJ)
#undef GBS_ADJ
    default:
      return AdjKernels{nullptr, nullptr, nullptr};
  }
}

// launchers of the built stencil with sd's offsets, term by term
AdjPicks2D adj2d_picks(const gbs_stencil_def_t *sd, int dtype) {
#define GBS_ADJ2D(id)                                                                        \
  {                                                                                          \
    const gbs_stencil_def_t *o = stencil_def(id);                                            \
    bool same = o->dim == sd->dim && o->kind == sd->kind && o->nterms == sd->nterms;         \
    for (int t = 0; same && t < o->nterms; ++t)                                              \
      same = o->terms[t].di == sd->terms[t].di && o->terms[t].dj == sd->terms[t].dj;         \
    if (same) return dtype == GBS_F64 ? adj2d_picks_##id##_d() : adj2d_picks_##id##_f();     \
  }
  GBS_FOR_EACH_ADJ2D(GBS_ADJ2D)
#undef GBS_ADJ2D
  return AdjPicks2D{};
}

// ---------------------------------------------------------------------------
// binomial (revolve) schedule
// ---------------------------------------------------------------------------
// beta(s, r) = (s + r)! / (s! r!): the most steps s snapshots reverse with
// every step advanced at most r times (saturating)
long long revolve_beta(int s, int r) {
  long long v = 1;
  for (int i = 1; i <= s; ++i) {
    v = v * (r + i) / i;
    if (v > (1LL << 40)) return 1LL << 40;
  }
  return v;
}

// Where to place the next snapshot when reversing l >= 2 steps from a stored
// state with k >= 1 free snapshot slots (k + 1 stored states in all): r is
// the least number of advances per step with beta(k+1, r) >= l. The split
// m = l - beta(k, r-1), kept within [1, min(l-1, beta(k+1, r-1))], leaves
// the right part (l - m steps, from the new snapshot, k - 1 slots left) as
// long as r - 1 advances per step allow and the left part (m steps, k
// slots) no longer than r - 1 advances allow; the total is then
// r*l - beta(k+2, r-1) forward steps, the minimum (checked against an
// exhaustive search over every split by the tests).
int revolve_split(int l, int k) {
  int r = 1;
  while (revolve_beta(k + 1, r) < l) ++r;
  long long m = l - revolve_beta(k, r - 1);
  if (m < 1) m = 1;
  const long long hi = std::min<long long>(l - 1, revolve_beta(k + 1, r - 1));
  return (int)std::max(1LL, std::min(m, hi));
}

// forward steps the schedule takes to reverse l steps with s free slots, and
// the most slots it holds at once
void revolve_count(int l, int s, long long *steps, int *peak, int depth = 0) {
  if (depth > *peak) *peak = depth;
  if (l <= 1) return;
  if (s == 0) {
    *steps += (long long)l * (l - 1) / 2;
    return;
  }
  const int m = revolve_split(l, s);
  *steps += m;
  revolve_count(l - m, s - 1, steps, peak, depth + 1);
  revolve_count(m, s, steps, peak, depth);
}

gbs_status check_adjoint_args(const gbs_desc *d, int C, const void *ws) {
  gbs_status st = check_desc(d);
  if (st != GBS_OK) return st;
  if (C < 1) return fail(GBS_ERR_INVALID, "checkpoint interval must be >= 1");
  if (!ws) return fail(GBS_ERR_INVALID, "workspace is NULL");
  if (reinterpret_cast<uintptr_t>(ws) % 256 != 0) return fail(GBS_ERR_INVALID, "workspace must be 256-byte aligned");
  return GBS_OK;
}

#define CK(call, what)                                   \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return cuda_fail(e_, what);   \
  } while (0)

// Branch streams of the batched entry points, per device: work forked from
// the caller's stream (an event), spread over the branches, joined back.
constexpr int kBranches = 16;
struct Branches {
  cudaStream_t s[kBranches] = {};
  cudaEvent_t fork = nullptr, join[kBranches] = {};
};
std::mutex g_branch_mu;  // held while a batched call enqueues (one set of events per device)
Branches g_branches[64];

gbs_status device_branches(Branches **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) return fail(GBS_ERR_NODEVICE, "device ordinal %d unsupported", dev);
  Branches &b = g_branches[dev];
  if (!b.fork) {
    for (int k = 0; k < kBranches && e == cudaSuccess; ++k) {
      e = cudaStreamCreateWithFlags(&b.s[k], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.join[k], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_fail(e, "adjoint batch: branch streams");
  }
  *out = &b;
  return GBS_OK;
}

// Runs run(i, branch_stream) for i < n on the branches (instance i on branch
// i % kBranches), ordered after the work already on `stream`, and makes
// `stream` wait for all of it.
template <class F>
gbs_status on_branches(int n, cudaStream_t stream, F run) {
  std::lock_guard<std::mutex> lk(g_branch_mu);
  Branches *b = nullptr;
  gbs_status st = device_branches(&b);
  if (st != GBS_OK) return st;
  const int used = std::min(n, kBranches);
  CK(cudaEventRecord(b->fork, stream), "adjoint batch: fork");
  for (int k = 0; k < used; ++k) CK(cudaStreamWaitEvent(b->s[k], b->fork, 0), "adjoint batch: fork");
  for (int i = 0; i < n && st == GBS_OK; ++i) st = run(i, b->s[i % kBranches]);
  // join even after a failure, so that `stream` never runs ahead of work already enqueued
  for (int k = 0; k < used; ++k) {
    cudaEventRecord(b->join[k], b->s[k]);
    cudaStreamWaitEvent(stream, b->join[k], 0);
  }
  return st;
}

}  // namespace

// computed once per (device ordinal, kernel): a process may drive GPUs with
// different SM counts. The kernel is opted in to its shared memory first: the
// query holds no CTA of one that is not (above 48 KB), and the answer, which
// decides the blocks of a step and with them the order of its sums, must not
// depend on whether the kernel has been launched before.
int adj_wave(const void *kernel, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    dev = 0;
  }
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find({dev, kernel});
  if (it != cache.end()) return it->second;
  int nb = 0, sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      (smem > kOptInSmem &&
       cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem) != cudaSuccess || nb <= 0) {
    (void)cudaGetLastError();
    return kAdjPartRows;
  }
  return cache.emplace(std::make_pair(dev, kernel), nb * sms).first->second;
}
}  // namespace gbs

using namespace gbs;

namespace gbs {
namespace {
gbs_status adjoint_forward(const gbs_desc *d, void *dev_A, int checkpoint_every, void *workspace, void *stream,
                           bool shared);
// rows per stream block of the forward launches of one of many instances: at
// least 4 b r (see shared_rows_2d; a whole wave of blocks measured slower here)
int instance_rows(const gbs_desc *d, const Layout &L, int b) {
  const int fma = d->fp_mode == GBS_FP_FMA ? 1 : 0;
  const int own = geometry2d(L, b, 0, resident_warps_2d(d->stencil, d->dtype, fma, b)).sl;
  return std::min(d->n[0], std::max({own, 8, 4 * b * L.rad}));
}
}  // namespace
}  // namespace gbs

extern "C" {

gbs_status gbs_adjoint_workspace(const gbs_desc *d, int checkpoint_every, size_t *bytes) {
  return gbs_adjoint_workspace_slots(d, checkpoint_every, 2 * std::max(1, checkpoint_every), bytes);
}

gbs_status gbs_adjoint_workspace_slots(const gbs_desc *d, int checkpoint_every, int slots, size_t *bytes) {
  gbs_status st = check_desc(d);
  if (st != GBS_OK) return st;
  if (checkpoint_every < 1 || !bytes) return fail(GBS_ERR_INVALID, "bad checkpoint interval or NULL bytes");
  if (slots < 0) return fail(GBS_ERR_INVALID, "slots must be >= 0");
  const Layout L = make_layout(d);
  *bytes = workspace_of(d, L, checkpoint_every, slots).total;
  return GBS_OK;
}

gbs_status gbs_revolve_cost(int steps, int slots, long long *forward_steps, int *peak_slots) {
  if (steps < 0 || slots < 0 || !forward_steps) return fail(GBS_ERR_INVALID, "bad revolve arguments");
  long long n = 0;
  int peak = 0;
  revolve_count(steps, slots, &n, &peak);
  *forward_steps = n;
  if (peak_slots) *peak_slots = peak;
  return GBS_OK;
}

gbs_status gbs_adjoint_plan_budget(const gbs_desc *d, size_t budget_bytes, int *checkpoint_every, int *slots,
                                   size_t *bytes) {
  gbs_status st = check_desc(d);
  if (st != GBS_OK) return st;
  if (!checkpoint_every || !slots) return fail(GBS_ERR_INVALID, "NULL output");
  const Layout L = make_layout(d);
  const int T = std::max(1, d->timestep);
  // every checkpoint interval C, every slot count: the fewest recomputed
  // forward steps whose workspace fits (ties: the smaller workspace)
  long long best_cost = -1;
  size_t best_bytes = 0;
  int best_c = 0, best_s = 0;
  for (int C = 1; C <= T; ++C) {
    const int ncp = (T + C - 1) / C;
    const Workspace w0 = workspace_of(d, L, C, 0);
    if (w0.total > budget_bytes) continue;
    // slots that still fit: revolve below 2C, the double stash at 2C
    const long long room = (long long)((budget_bytes - w0.total) / w0.plane_bytes);
    int s = (int)std::min<long long>(room, 2LL * C);
    long long cost;
    if (s >= 2 * C) {
      cost = (long long)T - ncp;  // each chunk recomputed once (its states after the checkpoint)
    } else {
      cost = 0;
      for (int j = 0; j < ncp; ++j) {
        long long n = 0;
        int peak = 0;
        revolve_count(std::min(C, T - j * C), s, &n, &peak);
        cost += n;
      }
    }
    const size_t b = workspace_of(d, L, C, s).total;
    if (b > budget_bytes) continue;
    if (best_cost < 0 || cost < best_cost || (cost == best_cost && b < best_bytes)) {
      best_cost = cost;
      best_bytes = b;
      best_c = C;
      best_s = s;
    }
  }
  if (best_cost < 0) return fail(GBS_ERR_NOMEM, "no checkpoint schedule fits %zu bytes", budget_bytes);
  *checkpoint_every = best_c;
  *slots = best_s;
  if (bytes) *bytes = best_bytes;
  return GBS_OK;
}

gbs_status gbs_adjoint_forward(const gbs_desc *d, void *dev_A, int checkpoint_every, void *workspace,
                               void *stream) {
  return adjoint_forward(d, dev_A, checkpoint_every, workspace, stream, false);
}
}  // extern "C"

namespace gbs {
namespace {
// shared: one of many instances side by side
gbs_status adjoint_forward(const gbs_desc *d, void *dev_A, int checkpoint_every, void *workspace, void *stream,
                           bool shared) {
  gbs_status st = check_adjoint_args(d, checkpoint_every, workspace);
  if (st != GBS_OK) return st;
  if (!dev_A) return fail(GBS_ERR_INVALID, "dev_A is NULL");
  int *err = nullptr;
  if ((st = error_word(&err)) != GBS_OK) return st;
  const Layout L = make_layout(d);
  const Workspace w = workspace_of(d, L, checkpoint_every, 2 * checkpoint_every);
  char *ws = static_cast<char *>(workspace);
  char *A = static_cast<char *>(dev_A);
  cudaStream_t s = (cudaStream_t)stream;
  for (int j = 0; j < w.ncp; ++j) {
    const int t0 = j * w.C;
    const int c = std::min(w.C, d->timestep - t0);
    CK(cudaMemcpyAsync(ws + w.off_cp + (size_t)j * w.plane_bytes, A, w.plane_bytes, cudaMemcpyDeviceToDevice, s),
       "adjoint: checkpoint");
    if (c <= 0) break;
    gbs_desc dc = *d;
    dc.timestep = c;
    if (shared && L.dim == 2) {
      gbs_plan_info pi{};
      if ((st = gbs_plan(&dc, &pi)) != GBS_OK) return st;
      dc.sl = instance_rows(&dc, L, pi.bt);
    }
    if ((st = run_loop(&dc, L, dev_A, s, err)) != GBS_OK) return st;
    if (c % 2) CK(cudaMemcpyAsync(A, A + w.plane_bytes, w.plane_bytes, cudaMemcpyDeviceToDevice, s), "adjoint: plane");
  }
  // u_T in both planes
  CK(cudaMemcpyAsync(A + w.plane_bytes, A, w.plane_bytes, cudaMemcpyDeviceToDevice, s), "adjoint: plane");
  return GBS_OK;
}

gbs_status adjoint_backward(const gbs_desc *d, const void *dev_lamT, void *dev_grad_u0, double *dev_coef_grad,
                            int checkpoint_every, int slots, void *workspace, void *stream, bool shared) {
  gbs_status st = check_adjoint_args(d, checkpoint_every, workspace);
  if (st != GBS_OK) return st;
  if (slots < 0) return fail(GBS_ERR_INVALID, "slots must be >= 0");
  if (!dev_lamT || !dev_grad_u0) return fail(GBS_ERR_INVALID, "NULL lam_T or grad_u0");
  const gbs_stencil_def_t *sd = stencil_def(d->stencil);
  const bool gradient = sd->kind == 1;
  if (dev_coef_grad && !gradient && sd->nterms > kMaxCoefGrad)
    return fail(GBS_ERR_UNSUPPORTED, "coefficient gradients need at most %d terms", kMaxCoefGrad);
  int *err = nullptr;
  if ((st = error_word(&err)) != GBS_OK) return st;
  const Layout L = make_layout(d);
  const Workspace w = workspace_of(d, L, checkpoint_every, slots);
  const AdjGeom g = geom_of(L);
  char *ws = static_cast<char *>(workspace);
  cudaStream_t s = (cudaStream_t)stream;
  const AdjKernels K = adj_kernels(d->stencil, d->dtype);
  const unsigned blocks = (unsigned)((g.cells + kAdjThreads - 1) / kAdjThreads);
  char *stash = ws + w.off_stash;
  char *lam[2] = {ws + w.off_lam, ws + w.off_lam + w.plane_bytes};
  char *hg = ws + w.off_hg;
  double *part = reinterpret_cast<double *>(ws + w.off_part);

  std::vector<double> coef, coefT;
  double div = 0.0, eps = 0.0;
  forward_coefficients(d, coef, div, eps);
  if (sd->divisor && div == 0.0) return fail(GBS_ERR_INVALID, "divisor must be nonzero");
  if (!gradient && !transposed_coefficients(sd, coef, coefT))
    return fail(GBS_ERR_UNSUPPORTED, "%s has an asymmetric offset set", sd->name);
  gbs_desc dT = *d;  // the transposed step: the forward kernels, FMA mode
  dT.fp_mode = GBS_FP_FMA;

  CK(cudaMemcpyAsync(lam[0], dev_lamT, w.plane_bytes, cudaMemcpyDeviceToDevice, s), "adjoint: lam_T");
  if (d->dtype == GBS_F64) zero_halo_kernel<double><<<blocks, kAdjThreads, 0, s>>>((double *)lam[0], g);
  else zero_halo_kernel<float><<<blocks, kAdjThreads, 0, s>>>((float *)lam[0], g);
  CK(cudaMemsetAsync(lam[1], 0, w.plane_bytes, s), "adjoint: memset");
  CK(cudaMemsetAsync(hg, 0, w.plane_bytes, s), "adjoint: memset");
  CK(cudaMemsetAsync(part, 0, (size_t)w.nblocks * w.nt * sizeof(double), s), "adjoint: memset");
  int cur = 0;
  const bool blocked = !gradient && g.dim == 2 && sd->nterms <= kMaxCoefGrad;  // adjoint2d.cu
  const AdjPicks2D P2 = blocked ? adj2d_picks(sd, d->dtype) : AdjPicks2D{};
  if (blocked && !P2.step[0][1]) return fail(GBS_ERR_UNSUPPORTED, "no 2-D adjoint step built for %s", sd->name);
  const int want = dev_coef_grad ? 1 : 0;
  // steps of one launch when `left` remain
  auto degree = [&](int left) {
    for (int b = std::min(left, kAdjMaxB); b > 1; --b)
      if (P2.step[want][b]) return b;
    return 1;
  };
  // b adjoint steps lam[cur] (= lam_{t+1}) -> lam[cur ^ 1] (= lam_{t+1-b}), u = the state u_t (u_{t-1} one plane
  // before it, ...); b > 1 for blocked stencils only
  auto steps = [&](const char *u, int b) -> gbs_status {
    AdjStep2D a{};
    a.g = &g;
    a.lam = lam[cur];
    a.u = u;
    a.lam_out = lam[cur ^ 1];
    a.hg = hg;
    a.part = part;
    a.coef = coef.data();
    a.div = sd->divisor ? div : 1.0;
    CK(P2.step[want][b](a, s), "adjoint: 2-D steps");
    cur ^= 1;
    return GBS_OK;
  };
  BlockPlan planT{};  // the transposed step of the stencils that the forward kernels serve
  // one adjoint step lam[cur] (= lam_{t+1}) -> lam[cur ^ 1] (= lam_t) on state u_t
  auto step = [&](const char *u) -> gbs_status {
    if (blocked) return steps(u, 1);
    if (gradient) {
      CK(K.grad(g, u, lam[cur], lam[cur ^ 1], hg, part, coef[0], eps, dev_coef_grad != nullptr, s),
         "adjoint: gradient2d step");
    } else {
      CK(K.halo(g, lam[cur], hg, coef, div, s), "adjoint: halo");
      if (dev_coef_grad) CK(K.coef(g, lam[cur], u, part, div, s), "adjoint: coefficients");
      gbs_status r = GBS_OK;
      if (planT.dim == 0) r = plan_block(&dT, L, coefT.data(), div, eps, 0, 1, false, err, &planT);
      if (r == GBS_OK) r = launch_plan(planT, lam[cur], lam[cur ^ 1], nullptr, s);
      if (r != GBS_OK) return r;
    }
    cur ^= 1;
    return GBS_OK;
  };

  if (!gradient && !dev_coef_grad) {
    // no forward state enters: T transposed steps from lam_T
    for (int left = d->timestep; left > 0;) {
      const int b = blocked ? degree(left) : 1;
      st = blocked ? steps(nullptr, b) : step(nullptr);
      if (st != GBS_OK) return st;
      left -= b;
    }
  } else if (w.revolve) {
    // Each chunk reversed by the binomial schedule over `slots` snapshot
    // planes and two work planes, all on `s`. The halo of every stash plane
    // is the fixed boundary (copied once; launches never write it).
    CK(copy_halo(d->dtype, g, ws + w.off_cp, stash, w.slots + 2, s), "adjoint: stash");
    char *work0 = stash + (size_t)w.slots * w.plane_bytes;  // ping-pong partner of an advance
    char *work1 = work0 + w.plane_bytes;                     // target of a recompute without slots
    gbs_plan_info pi{};
    {
      gbs_desc dp = *d;
      dp.timestep = std::max(1, w.C);
      if ((st = gbs_plan(&dp, &pi)) != GBS_OK) return st;
    }
    const int bfwd = std::max(1, pi.bt);
    // advance k >= 1 steps from plane src into plane dst (dst != work0)
    auto advance = [&](const char *src, char *dst, int k) -> gbs_status {
      const std::vector<int> blocks_k = split_steps(k, bfwd);
      const int n = (int)blocks_k.size();
      const char *from = src;
      for (int j = 0; j < n; ++j) {
        char *to = ((n - 1 - j) % 2 == 0) ? dst : work0;
        gbs_status r = launch_block(d, L, coef.data(), div, eps, 0, blocks_k[j], from, to, s, err);
        if (r != GBS_OK) return r;
        from = to;
      }
      return GBS_OK;
    };
    // reverse steps [a, b) given u_a in plane ua, with `nfree` snapshot slots
    // free from index `top` on
    std::function<gbs_status(int, int, const char *, int)> reverse = [&](int a, int b, const char *ua,
                                                                         int top) -> gbs_status {
      const int l = b - a, nfree = w.slots - top;
      if (l <= 0) return GBS_OK;
      if (l == 1) return step(ua);
      if (nfree == 0) {
        for (int t = b - 1; t > a; --t) {
          gbs_status r = advance(ua, work1, t - a);
          if (r == GBS_OK) r = step(work1);
          if (r != GBS_OK) return r;
        }
        return step(ua);
      }
      const int m = revolve_split(l, nfree);
      char *snap = stash + (size_t)top * w.plane_bytes;
      gbs_status r = advance(ua, snap, m);
      if (r == GBS_OK) r = reverse(a + m, b, snap, top + 1);
      if (r == GBS_OK) r = reverse(a, a + m, ua, top);
      return r;
    };
    for (int j = w.ncp - 1; j >= 0 && st == GBS_OK; --j) {
      const int t0 = j * w.C;
      const int c = std::min(w.C, d->timestep - t0);
      st = reverse(t0, t0 + c, ws + w.off_cp + (size_t)j * w.plane_bytes, 0);
    }
    if (st != GBS_OK) return st;
  } else {
    // Two stash buffers: while the adjoint steps of chunk j run on `s`, a
    // second stream recomputes the states of chunk j-1 into the other
    // buffer. Events order it: a buffer is refilled only after the adjoint
    // steps that read it (freed), and read only after its refill (ready).
    const size_t buf_bytes = (size_t)w.C * w.plane_bytes;
    cudaStream_t s2 = nullptr;
    cudaEvent_t setup = nullptr, done2 = nullptr, ready[2] = {}, freed[2] = {};
    auto release = [&]() {
      for (int b = 0; b < 2; ++b) {
        if (ready[b]) cudaEventDestroy(ready[b]);
        if (freed[b]) cudaEventDestroy(freed[b]);
      }
      if (setup) cudaEventDestroy(setup);
      if (done2) cudaEventDestroy(done2);
      if (s2) cudaStreamDestroy(s2);
    };
    cudaError_t e = cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&setup, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done2, cudaEventDisableTiming);
    for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
      e = cudaEventCreateWithFlags(&ready[b], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&freed[b], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
      release();
      return cuda_fail(e, "adjoint: streams");
    }
    // the halo of every stash slot of both buffers: the fixed boundary (never rewritten)
    if ((e = copy_halo(d->dtype, g, ws + w.off_cp, stash, 2 * w.C, s)) != cudaSuccess) {
      release();
      return cuda_fail(e, "adjoint: stash");
    }
    cudaEventRecord(setup, s);
    cudaStreamWaitEvent(s2, setup, 0);
    // recompute degree: 2-D grids in FMA mode use the forward's fused degree
    // (at most the largest stash-mode degree), each launch also storing its
    // intermediate states; otherwise one step per launch
    int bre = 1;
    if (g.dim == 2 && d->fp_mode == GBS_FP_FMA) {
      gbs_desc dp = *d;
      dp.timestep = std::max(1, w.C);
      gbs_plan_info pi{};
      if ((st = gbs_plan(&dp, &pi)) != GBS_OK) {
        release();
        return st;
      }
      bre = std::max(1, std::min(pi.bt, kMaxStashB));
    }
    BlockPlan planR[kMaxStashB + 1] = {};  // the recompute's launches, by degree
    // recompute u_{t0} .. u_{t0+c-1} of chunk j into buffer j % 2 on s2
    auto recompute = [&](int j) -> gbs_status {
      const int b = j & 1;
      char *buf = stash + (size_t)b * buf_bytes;
      const int c = std::min(w.C, d->timestep - j * w.C);
      cudaStreamWaitEvent(s2, freed[b], 0);  // no-op before the buffer's first use
      cudaError_t ce = cudaMemcpyAsync(buf, ws + w.off_cp + (size_t)j * w.plane_bytes, w.plane_bytes,
                                       cudaMemcpyDeviceToDevice, s2);
      if (ce != cudaSuccess) return cuda_fail(ce, "adjoint: restore");
      for (int k = 1; k < c;) {
        // one launch of bb steps from slot k-1: slots k .. k+bb-1
        const int bb = std::min(bre, c - k);
        BlockPlan &plan = planR[bb];
        gbs_status r = GBS_OK;
        if (plan.dim == 0)
          r = plan_block(d, L, coef.data(), div, eps, shared && L.dim == 2 ? instance_rows(d, L, bb) : 0, bb, bb > 1, err,
                         &plan);
        if (r == GBS_OK)
          r = launch_plan(plan, buf + (size_t)(k - 1) * w.plane_bytes, buf + (size_t)(k - 1 + bb) * w.plane_bytes,
                          bb > 1 ? buf + (size_t)k * w.plane_bytes : nullptr, s2);
        if (r != GBS_OK) return r;
        k += bb;
      }
      cudaEventRecord(ready[b], s2);
      return GBS_OK;
    };
    st = recompute(w.ncp - 1);
    for (int j = w.ncp - 1; j >= 0 && st == GBS_OK; --j) {
      const int b = j & 1;
      const int c = std::min(w.C, d->timestep - j * w.C);
      if (j > 0 && (st = recompute(j - 1)) != GBS_OK) break;  // overlaps the steps below
      cudaStreamWaitEvent(s, ready[b], 0);
      // lam_{t+1} -> lam_t for t = t0+c-1 .. t0
      char *buf = stash + (size_t)b * buf_bytes;
      for (int k = c - 1; k >= 0 && st == GBS_OK;) {
        const int bb = blocked ? degree(k + 1) : 1;
        const char *u = buf + (size_t)k * w.plane_bytes;
        st = blocked ? steps(u, bb) : step(u);
        k -= bb;
      }
      cudaEventRecord(freed[b], s);
    }
    // every piece of s2's work is ordered before s (the last ready event); join anyway
    cudaEventRecord(done2, s2);
    cudaStreamWaitEvent(s, done2, 0);
    release();
    if (st != GBS_OK) return st;
  }
  if (d->dtype == GBS_F64)
    combine_kernel<double><<<blocks, kAdjThreads, 0, s>>>((const double *)lam[cur], (const double *)hg,
                                                         (double *)dev_grad_u0, g);
  else
    combine_kernel<float><<<blocks, kAdjThreads, 0, s>>>((const float *)lam[cur], (const float *)hg,
                                                        (float *)dev_grad_u0, g);
  if (dev_coef_grad) sum_parts_kernel<<<w.nt, 256, 0, s>>>(part, w.nblocks, w.nt, dev_coef_grad);
  CK(cudaGetLastError(), "adjoint: combine");
  return GBS_OK;
}

}  // namespace
}  // namespace gbs

extern "C" {
gbs_status gbs_adjoint_backward(const gbs_desc *d, const void *dev_lamT, void *dev_grad_u0, double *dev_coef_grad,
                                int checkpoint_every, void *workspace, void *stream) {
  return adjoint_backward(d, dev_lamT, dev_grad_u0, dev_coef_grad, checkpoint_every, 2 * std::max(1, checkpoint_every),
                          workspace, stream, false);
}

gbs_status gbs_adjoint_backward_slots(const gbs_desc *d, const void *dev_lamT, void *dev_grad_u0,
                                      double *dev_coef_grad, int checkpoint_every, int slots, void *workspace,
                                      void *stream) {
  return adjoint_backward(d, dev_lamT, dev_grad_u0, dev_coef_grad, checkpoint_every, slots, workspace, stream, false);
}

gbs_status gbs_adjoint_forward_batch(const gbs_desc *descs, int n, void *const *dev_A, int checkpoint_every,
                                     void *const *workspaces, void *stream) {
  if (!descs || n < 1 || !dev_A || !workspaces) return fail(GBS_ERR_INVALID, "adjoint batch: no instances");
  for (int i = 0; i < n; ++i) {
    gbs_status st = check_adjoint_args(&descs[i], checkpoint_every, workspaces[i]);
    if (st != GBS_OK) return st;
    if (!dev_A[i]) return fail(GBS_ERR_INVALID, "adjoint batch: instance %d has no grid", i);
  }
  return on_branches(n, (cudaStream_t)stream, [&](int i, cudaStream_t bs) {
    return adjoint_forward(&descs[i], dev_A[i], checkpoint_every, workspaces[i], bs, n > 1);
  });
}

gbs_status gbs_adjoint_backward_batch(const gbs_desc *descs, int n, const void *const *dev_lamT,
                                      void *const *dev_grad_u0, double *const *dev_coef_grad, int checkpoint_every,
                                      void *const *workspaces, void *stream) {
  if (!descs || n < 1 || !dev_lamT || !dev_grad_u0 || !workspaces)
    return fail(GBS_ERR_INVALID, "adjoint batch: no instances");
  for (int i = 0; i < n; ++i) {
    gbs_status st = check_adjoint_args(&descs[i], checkpoint_every, workspaces[i]);
    if (st != GBS_OK) return st;
    if (!dev_lamT[i] || !dev_grad_u0[i]) return fail(GBS_ERR_INVALID, "adjoint batch: instance %d lacks a plane", i);
  }
  return on_branches(n, (cudaStream_t)stream, [&](int i, cudaStream_t bs) {
    return adjoint_backward(&descs[i], dev_lamT[i], dev_grad_u0[i], dev_coef_grad ? dev_coef_grad[i] : nullptr,
                            checkpoint_every, 2 * std::max(1, checkpoint_every), workspaces[i], bs, n > 1);
  });
}

}  // extern "C"
