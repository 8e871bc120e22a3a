// Adjoint step of the 2-D linear stencils, temporally blocked.
//
// For u_{t+1}(x) = sum_k c_k u_t(x + o_k) / d on the interior and lam = 0 on
// the halo, b steps back in one launch (level l = 0 .. b-1, lam^0 = the input):
//   v(y) = sum_k c_k/d lam^l(y - o_k) at every cell y of the grid;
//   lam^{l+1} = v on the interior; hg += v on the halo (its gradient);
//   and, for the coefficient gradients, acc_k += lam^l(y - o_k) u_{t-l}(y)
// over every cell y: sum_x lam(x) u(x + o_k) with the states' cells as the
// index of the sum, so that the products use the very operands of the step
// and read one row of the state, with no neighbours. Where y - o_k is not
// interior lam is 0, and so is the product, unless the state there is infinite
// or NaN: a warp at the grid's rim whose sums are not finite forms them again
// without those products (recount; tests of every product in the row loops
// cost 10 to 13%, j2d5pt and j2d9pt f32 2048^2).
//
// A warp owns a strip of columns and a block of rows and streams the rows as
// the forward kernels do (kernel2d.cuh): lane-private cp.async copies of lam's
// row and of the state rows that the step needs into a ring, groups of rows in
// flight ahead, a register window of 2r+1 rows of lam per level, in-row
// neighbours by shuffles, overlapped tiling. The edge strips own the halo
// columns beside them, the first and last blocks the halo rows; the halo's
// gradient is accumulated by reductions to memory (each cell by one lane of
// one warp, in order), so that no warp waits for it.
//
// Products are summed per lane and level in T; every kFlushRows rows a float
// sum is folded into a compensated pair, and the pairs are reduced over the
// CTA, so that a long block loses no precision; the warps' sums are added in
// double. The decomposition does not depend on b and the levels' sums enter
// the result one after the other, so b steps in one launch give the bits of b
// launches (a chunk reversed by the binomial schedule takes single steps).
//
// Bound: memory latency and instruction issue (a step of a 2048^2 grid moves
// 50 MB, mostly within the L2; issue 52% busy at 0.73 waves). Measured (GB300,
// j2d5pt f32 2048^2, cold L2): with products 21.3 us a launch of two steps; the
// kernel of one step this replaced took 13.0.
//
// Built per stencil and element type with -DGBS_SID=<table id>
// -DGBS_T=<float|double> -DGBS_PICK=<exported name>; a divisor is folded into
// the coefficients, so stencils with the same offsets share one.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "adjoint_internal.h"
#include "gbs_device.cuh"

#if !defined(GBS_SID) || !defined(GBS_T) || !defined(GBS_PICK)
#error "GBS_SID, GBS_T and GBS_PICK must be defined"
#endif

namespace gbs {
namespace {

using T = GBS_T;
using S = typename StencilById<GBS_SID>::type;
constexpr int kWarps = 4;

template <int NT> struct AdjParams2D {
  const T *lam, *u;          // lam_{t+1}; u_t (u_{t-l} is l planes before it)
  T *lam_out, *hg;
  double *part;
  long long pitch, u_stride; // elements per row; between successive states
  int d0, d1, shift, nstrips;
  int nblocks, sl;           // stream blocks of the inner strips, their rows
  int nblocks_e, sl_e;       // of the edge strips
  long long item0;           // the launch's first item
  T inv_div;
  T coef[NT];                // c_k / d
};

template <class ST, int B, bool COEF> struct AdjPipe2D {
  static constexpr int R = ST::kRad, W = 2 * R + 1;
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int COLS = 32 * V;
  // rows of lam with in-row neighbours at every offset (boxes): the window
  // holds them extended, from their arrival on
  static constexpr bool BOX = ST::kAssoc;
  static constexpr int XW = BOX ? V + 2 * R : V;
  static constexpr int NROW = 1 + (COEF ? B : 0);            // rows per step: lam, u_{t-l}
  static constexpr unsigned ROWB = 512u * NROW;
  static constexpr int ROW_INSTR = B * (ST::kTerms * V * (COEF ? 2 : 1) + 14) + 20;
  static constexpr bool ROT = W * ROW_INSTR <= 1300;
  static constexpr int SLIDE = 800 / ROW_INSTR;
  static constexpr int NPH = ROT ? W : (SLIDE < 1 ? 1 : (SLIDE > W - 1 ? W - 1 : SLIDE));
  static constexpr int WSLOTS = ROT ? W : W + NPH - 1;
  static constexpr int PG = (6 + NPH - 1) / NPH;
  static constexpr unsigned GROUP = NPH * ROWB, RING = (PG + 1) * GROUP;
  // shared memory of a CTA: the warps' rings, then the lanes' sums
  static constexpr size_t RINGS = (size_t)kWarps * RING,
                          SUMS = COEF ? 2 * sizeof(T) * B * ST::kTerms * kWarps * 32 : 0,
                          SMEM = RINGS > SUMS ? RINGS : SUMS;
  static constexpr int ML = (B * R + V - 1) / V * V;
  static constexpr int WOUT = (COLS - ML - B * R) / V * V;
  // Single steps in double: the FP64 pipe bounds them, so the rows before a
  // block's first are not computed: whole groups that only fill the window come
  // first, and the rows after them need no branch (a branch per row instead kept
  // the compiler from overlapping rows: box2d2r 1500^2 6494 us against 5266)
  static constexpr bool FILL = B == 1 && sizeof(T) == 8;
  static constexpr int NFILL = FILL ? (2 * R + NPH - 1) / NPH : 0;
  static constexpr int slot(int ph, int j) { return ROT ? (ph + 1 + j) % W : ph + j; }
};

constexpr int kFlushRows = 16;  // 64 products per float partial sum

enum : int { kIn = 0, kCols = 1, kEverything = 2 };

// (hi, lo) += v, the rounding error of the sum kept in lo (Knuth's TwoSum)
template <typename U> __device__ __forceinline__ void pair_add(U &hi, U &lo, U v) {
  using A = Arith<U>;
  const U s = A::add(hi, v), b = A::sub(s, hi);
  lo = A::add(lo, A::add(A::sub(hi, A::sub(s, b)), A::sub(v, b)));
  hi = s;
}

// A warp's work item: a strip of columns and a block of rows.
struct AdjItem {
  int cs, ce;          // columns stored
  int own_lo, own_hi;  // and those summed over (a grid's edge strips own the halo beside them)
  int i0, i1, o0, o1;  // the same for the rows
  bool rim;            // owns halo cells
};
// the edge strips' items come first, in shorter blocks (see launch)
template <class ST, class AP> __device__ __forceinline__ AdjItem adj_item(const AdjParams2D<ST::kTerms> &p, long long gw) {
  constexpr int R = ST::kRad;
  const int edges = p.nstrips > 1 ? 2 : 1;
  const long long edge_items = (long long)edges * p.nblocks_e;
  const bool first = gw < edge_items;
  const int strip = first ? (gw % edges ? p.nstrips - 1 : 0) : 1 + (int)((gw - edge_items) % (p.nstrips - edges));
  const int blk = first ? (int)(gw / edges) : (int)((gw - edge_items) / (p.nstrips - edges));
  const int sl = first ? p.sl_e : p.sl, nblocks = first ? p.nblocks_e : p.nblocks;
  AdjItem it;
  it.cs = R + strip * AP::WOUT;
  it.ce = min(it.cs + AP::WOUT, p.d1 - R);
  it.own_lo = strip == 0 ? 0 : it.cs;
  it.own_hi = strip == p.nstrips - 1 ? p.d1 : it.ce;
  it.i0 = R + blk * sl;
  it.i1 = min(it.i0 + sl, p.d0 - R);
  it.o0 = blk == 0 ? 0 : it.i0;
  it.o1 = blk == nblocks - 1 ? p.d0 : it.i1;
  it.rim = first || blk == 0 || blk == nblocks - 1;
  return it;
}

// One lane's sum (hi, lo) for term t of level l, in the order of the row loops
// and with lam^l as the step forms it, over the cells y whose y - o_t is
// interior. Plain loads and loops: for states that are not finite.
template <class ST, class AP>
__device__ __noinline__ void recount(const AdjParams2D<ST::kTerms> &p, long long gw, int l, int t, T &hi, T &lo) {
  constexpr int R = ST::kRad, V = AP::V;
  const AdjItem it = adj_item<ST, AP>(p, gw);
  const int col0 = it.cs - AP::ML + (int)(threadIdx.x & 31) * V;
  auto offset = [](int k, int &di, int &dj) GBS_INL {
    static_for<ST::kTerms>([&](auto TI) GBS_INL {
      constexpr int kk = decltype(TI)::value, ki = ST::kOff[kk][0], kj = ST::kOff[kk][1];
      if (kk == k) {
        di = ki;
        dj = kj;
      }
    });
  };
  auto inner = [&](int i, int j) GBS_INL { return i >= R && i < p.d0 - R && j >= R && j < p.d1 - R; };
  auto lam = [&](int i, int j) GBS_INL { return inner(i, j) ? __ldcg(p.lam + (long long)i * p.pitch + p.shift + j) : T(0); };
  int di = 0, dj = 0;
  offset(t, di, dj);
  T acc = T(0);
  hi = lo = T(0);
#pragma unroll 1
  for (int q = it.o0; q < it.o1; ++q) {
#pragma unroll 1
    for (int c = max(col0, it.own_lo); c < min(col0 + V, it.own_hi); ++c) {
      const int i = q - di, j = c - dj;
      if (!inner(i, j)) continue;
      T v = lam(i, j);
      if (l == 1) {
#pragma unroll 1
        for (int k = 0; k < ST::kTerms; ++k) {
          int ki = 0, kj = 0;
          offset(k, ki, kj);
          const T a = lam(i - ki, j - kj);
          v = k == 0 ? Arith<T>::mul(p.coef[0], a) : Arith<T>::fma(p.coef[k], a, v);
        }
      }
      acc = Arith<T>::fma(v, __ldcg(p.u - (long long)l * p.u_stride + (long long)q * p.pitch + p.shift + c), acc);
    }
    if (sizeof(T) == 4 && (q - it.o0) % kFlushRows == kFlushRows - 1) {
      pair_add(hi, lo, acc);
      acc = T(0);
    }
  }
  pair_add(hi, lo, acc);
}

// A row extended by its in-row neighbours. Beyond the window they are 0 (only
// a halo column's own neighbours off the grid are ever that far).
template <int V, int R, bool ZERO>
__device__ __forceinline__ void extend(T (&ext)[V + 2 * R], const T (&row)[V], int lane) {
  static_for<V + 2 * R>([&](auto XI) GBS_INL {
    constexpr int x = decltype(XI)::value - R;
    T v = row_elem<V, x>(row);
    if constexpr (ZERO && x < 0) v = lane < (-x + V - 1) / V ? T(0) : v;
    if constexpr (ZERO && x >= V) v = lane >= 32 - x / V ? T(0) : v;
    ext[R + x] = v;
  });
}

// In double two CTAs on an SM fill the FP64 pipe; asking for no more keeps the
// box of radius 2 from spilling its coefficient sums (560 bytes of 168 registers)
template <class ST, int B, bool COEF>
__global__ void __launch_bounds__(kWarps * 32, (AdjPipe2D<ST, B, COEF>::FILL ? 2 : 0))
    adj2d_kernel(const __grid_constant__ AdjParams2D<ST::kTerms> p) {
  using AP = AdjPipe2D<ST, B, COEF>;
  constexpr int V = AP::V, R = AP::R, NPH = AP::NPH, PG = AP::PG, NT = ST::kTerms;
  constexpr int NP = COEF ? NT : 1, NL = COEF ? B : 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ double sums[NL * NP];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long gw = p.item0 + (long long)blockIdx.x * kWarps + wid;
  // this CTA's row of the partial sums, read ahead of its update
  double total = 0.0;
  if (COEF && (int)threadIdx.x < NT) total = p.part[(size_t)blockIdx.x * NT + threadIdx.x];
  const int edges = p.nstrips > 1 ? 2 : 1;
  const bool busy = gw < (long long)edges * p.nblocks_e + (long long)(p.nstrips - edges) * p.nblocks;
  [[maybe_unused]] bool redo = false;  // the warp's sums are not finite, and it owns halo cells
  T acc[NL][NP], hi[NL][NP], lo[NL][NP];
#pragma unroll
  for (int l = 0; l < NL; ++l)
#pragma unroll
    for (int t = 0; t < NP; ++t) acc[l][t] = hi[l][t] = lo[l][t] = T(0);

  if (busy) {
    const AdjItem it = adj_item<ST, AP>(p, gw);
    const int cs = it.cs, ce = it.ce, own_lo = it.own_lo, own_hi = it.own_hi;
    const int i0 = it.i0, i1 = it.i1, o0 = it.o0, o1 = it.o1;
    const int el = cs + p.shift - AP::ML + lane * V;
    const int col0 = el - p.shift;
    const int w0 = cs - AP::ML;                   // column of the window's element 0
    const bool edge = (w0 < R) || (w0 + AP::COLS > p.d1 - R);
    const bool in_row = el >= 0 && el + V <= p.pitch;
    const bool whole = col0 >= cs && col0 + V <= ce;
    bool inner[V], own[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      inner[e] = col0 + e >= R && col0 + e < p.d1 - R;
      own[e] = col0 + e >= own_lo && col0 + e < own_hi;
    }
    const int pstart = AP::FILL ? o0 + R - AP::NFILL * NPH : max(0, o0 - B * R), pend = min(p.d0, o1 + B * R);
    const int ng = (o1 + B * R - pstart + NPH - 1) / NPH;
    // rows [fast_lo, fast_hi): every row that enters or leaves a level is interior
    const int fast_lo = pstart >= R ? pstart : (B + 1) * R;
    const int fast_hi = o1 + B * R <= p.d0 - R ? 0x7fffffff : p.d0 - R;
    const unsigned nown = (unsigned)(o1 - o0), nout = (unsigned)(i1 - i0);

    unsigned char *my = smem_raw + (size_t)wid * AP::RING + lane * 16;
    const uint32_t my_s = smem_u32(my);
    const T *lam_next = p.lam + (long long)pstart * p.pitch + el;  // next rows to request
    const T *u_next[COEF ? B : 1];
    if constexpr (COEF) {
#pragma unroll
      for (int l = 0; l < B; ++l)
        u_next[l] = p.u + ((long long)(pstart - (l + 1) * R) * p.pitch + el - (long long)l * p.u_stride);
    }
    int req = pstart;                             // row of the next group's phase 0
    unsigned wr = 0, rd = 0;
    auto request_group = [&]() GBS_INL {
#pragma unroll
      for (int ph = 0; ph < NPH; ++ph) {
        if (in_row && (AP::FILL ? (unsigned)(req + ph) < (unsigned)pend : req + ph < pend)) cp_async16(my_s + wr + ph * AP::ROWB, lam_next);
        lam_next += p.pitch;
        if constexpr (COEF) {
#pragma unroll
          for (int l = 0; l < B; ++l) {
            if (in_row && (unsigned)(req + ph - (l + 1) * R - o0) < nown)
              cp_async16(my_s + wr + ph * AP::ROWB + 512 * (1 + l), u_next[l]);
            u_next[l] += p.pitch;
          }
        }
      }
      cp_async_commit();
      req += NPH;
      wr = wr + AP::GROUP == AP::RING ? 0u : wr + AP::GROUP;
    };
#pragma unroll 1
    for (int k = 0; k < PG; ++k) request_group();

    T win[B][AP::WSLOTS][AP::XW];
#pragma unroll
    for (int l = 0; l < B; ++l)
#pragma unroll
      for (int w = 0; w < AP::WSLOTS; ++w)
#pragma unroll
        for (int e = 0; e < AP::XW; ++e) win[l][w][e] = T(0);

    int pb = pstart;
    T *out = p.lam_out + ((long long)(pstart - B * R) * p.pitch + el);  // the row the last level completes

    auto rows = [&](auto CAREI, auto FILLI) GBS_INL {
      constexpr int care = decltype(CAREI)::value;
      constexpr bool fill = decltype(FILLI)::value;
      static_for<NPH>([&](auto PHI) GBS_INL {
        constexpr int ph = decltype(PHI)::value;
        const int pp = pb + ph;
        T x[V];
        ld_vec<T, V>(x, reinterpret_cast<const T *>(my + rd + ph * AP::ROWB));
        if constexpr (care != kIn) {  // lam is 0 off the interior, whatever memory holds there
          const bool row_in = care == kCols || (pp >= R && pp < p.d0 - R);
#pragma unroll
          for (int e = 0; e < V; ++e) x[e] = row_in && inner[e] ? x[e] : T(0);
        }
        static_for<B>([&](auto LI) GBS_INL {
          constexpr int l = decltype(LI)::value;
          [[maybe_unused]] const int q = pp - (l + 1) * R;
          T ext[V + 2 * R];
          if constexpr (AP::BOX) {
            extend<V, R, care != kIn>(ext, x, lane);
#pragma unroll
            for (int e = 0; e < AP::XW; ++e) win[l][AP::slot(ph, 2 * R)][e] = ext[e];
          } else {
#pragma unroll
            for (int e = 0; e < V; ++e) win[l][AP::slot(ph, 2 * R)][e] = x[e];
            T row[V];
#pragma unroll
            for (int e = 0; e < V; ++e) row[e] = win[l][AP::slot(ph, R)][e];
            if constexpr (!fill) extend<V, R, care != kIn>(ext, row, lane);
          }
          if constexpr (fill) return;
          if constexpr (AP::FILL && care == kEverything) {  // rows past the block's last
            if ((unsigned)(q - o0) >= nown) return;
          }
          // lam^l(y - o_t) for the lane's element e of row q
          auto operand = [&](auto TI, auto EI) GBS_INL -> T {
            constexpr int di = ST::kOff[decltype(TI)::value][0], dj = ST::kOff[decltype(TI)::value][1];
            constexpr int e = decltype(EI)::value;
            if constexpr (AP::BOX) return win[l][AP::slot(ph, R - di)][R + e - dj];
            else if constexpr (dj == 0) return win[l][AP::slot(ph, R - di)][e];
            else return ext[R + e - dj];
          };
          T y[V];
          static_for<NT>([&](auto TI) GBS_INL {
            static_for<V>([&](auto EI) GBS_INL {
              constexpr int t = decltype(TI)::value, e = decltype(EI)::value;
              if constexpr (t == 0) y[e] = Arith<T>::mul(p.coef[t], operand(TI, EI));
              else y[e] = Arith<T>::fma(p.coef[t], operand(TI, EI), y[e]);
            });
          });
          if constexpr (COEF) {
            if ((unsigned)(q - o0) < nown) {
              T uv[V];
              ld_vec<T, V>(uv, reinterpret_cast<const T *>(my + rd + ph * AP::ROWB + 512 * (1 + l)));
              if constexpr (care != kIn) {
#pragma unroll
                for (int e = 0; e < V; ++e) uv[e] = own[e] ? uv[e] : T(0);
              }
              static_for<NT>([&](auto TI) GBS_INL {
                static_for<V>([&](auto EI) GBS_INL {
                  constexpr int t = decltype(TI)::value, e = decltype(EI)::value;
                  acc[l][t] = Arith<T>::fma(operand(TI, EI), uv[e], acc[l][t]);
                });
              });
              if (sizeof(T) == 4 && (q - o0) % kFlushRows == kFlushRows - 1) {
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                  pair_add(hi[l][t], lo[l][t], acc[l][t]);
                  acc[l][t] = T(0);
                }
              }
            }
          }
          if constexpr (care != kIn) {
            const bool row_in = care == kCols || (q >= R && q < p.d0 - R);
            const bool owned = (unsigned)(q - o0) < nown;
            T *h = p.hg + (long long)q * p.pitch + el;
#pragma unroll
            for (int e = 0; e < V; ++e) red_add_if(h + e, y[e], owned && own[e] && !(row_in && inner[e]));
#pragma unroll
            for (int e = 0; e < V; ++e) y[e] = row_in && inner[e] ? y[e] : T(0);
          }
#pragma unroll
          for (int e = 0; e < V; ++e) x[e] = y[e];
        });
        [[maybe_unused]] const bool keep = (unsigned)(pp - B * R - i0) < nout;
        if constexpr (!fill) st_vec_global_if<V>(out, x, keep && whole);
        if constexpr (care != kIn && !fill) {
#pragma unroll
          for (int e = 0; e < V; ++e) st_global_if(out + e, x[e], keep && !whole && col0 + e >= cs && col0 + e < ce);
        }
        out += p.pitch;
      });
      if constexpr (!AP::ROT) {
#pragma unroll
        for (int l = 0; l < B; ++l)
#pragma unroll
          for (int j = 0; j < 2 * R; ++j)
#pragma unroll
            for (int e = 0; e < AP::XW; ++e) win[l][j][e] = win[l][j + NPH][e];
      }
    };

#pragma unroll 1
    for (int k = 0; k < ng; ++k) {
      request_group();
      cp_async_wait<PG>();
      if (k < AP::NFILL) rows(IC<kEverything>(), IC<1>());
      else if (pb < fast_lo || pb + NPH > fast_hi || (AP::FILL && pb + NPH > o1 + R)) rows(IC<kEverything>(), IC<0>());
      else if (edge) rows(IC<kCols>(), IC<0>());
      else rows(IC<kIn>(), IC<0>());
      pb += NPH;
      rd = rd + AP::GROUP == AP::RING ? 0u : rd + AP::GROUP;
    }
    cp_async_wait<0>();
    if constexpr (COEF) {
      // lanes outside the strip's own columns summed their neighbours' products
      const bool mine = own[0] || own[V - 1];
#pragma unroll
      for (int l = 0; l < NL; ++l)
#pragma unroll
        for (int t = 0; t < NP; ++t) {
          pair_add(hi[l][t], lo[l][t], acc[l][t]);
          hi[l][t] = mine ? hi[l][t] : T(0);
          lo[l][t] = mine ? lo[l][t] : T(0);
          redo = redo || !(hi[l][t] - hi[l][t] == T(0));
        }
      redo = __any_sync(0xffffffffu, redo) && it.rim;
    }
  }
  if constexpr (COEF) {
    // every lane's pairs through shared memory (the rings' room); each warp
    // then reduces some of them
    auto part_hi = reinterpret_cast<T(*)[kWarps * 32]>(smem_raw), part_lo = part_hi + NL * NT;
    __syncthreads();
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        part_hi[l * NT + t][threadIdx.x] = hi[l][t];
        part_lo[l * NT + t][threadIdx.x] = lo[l][t];
      }
    if (redo) {
      static_assert(NL <= 2, "recount forms lam^0 and lam^1");
#pragma unroll 1
      for (int k = 0; k < NL * NT; ++k)
        recount<ST, AP>(p, gw, k / NT, k % NT, part_hi[k][threadIdx.x], part_lo[k][threadIdx.x]);
    }
    __syncthreads();
    for (int k = wid; k < NL * NT; k += kWarps) {
      T h = part_hi[k][lane], c = part_lo[k][lane];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) {
        pair_add(h, c, part_hi[k][w * 32 + lane]);
        c = Arith<T>::add(c, part_lo[k][w * 32 + lane]);
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const T h2 = __shfl_down_sync(0xffffffffu, h, s), c2 = __shfl_down_sync(0xffffffffu, c, s);
        pair_add(h, c, h2);
        c = Arith<T>::add(c, c2);
      }
      if (lane == 0) sums[k] = (double)h + (h - h == T(0) ? (double)c : 0.0);  // c is NaN beside an infinite h
    }
    __syncthreads();
    static_assert(NT <= kWarps * 32, "a thread per term");
    if ((int)threadIdx.x < NT) {
#pragma unroll
      for (int l = 0; l < NL; ++l) total += sums[l * NT + threadIdx.x] * (double)p.inv_div;
      p.part[(size_t)blockIdx.x * NT + threadIdx.x] = total;
    }
  }
}

// Degrees built. Float: four steps for radius 1, two with coefficient
// gradients (each level keeps its own sums) and for stars of radius 2. Double
// is bound by the FP64 pipe, where the overlap's recomputation only adds.
template <class ST, bool COEF> constexpr int max_degree() {
  if (sizeof(T) == 8) return 1;
  if (ST::kRad == 1) return COEF ? 2 : 4;
  if (ST::kRad == 2 && !ST::kAssoc) return 2;
  return 1;
}

// Rows per block of a step in double: the FP64 pipe is shared by the warps of an
// SM quarter. extra: what a block costs beside its rows, in rows.
inline int fill_rows(int nstrips, int ni, int extra) {
  const int sms = sm_count();
  double best = 1e300;
  int best_sl = ni;
  for (int k = 1; k <= 32; ++k) {
    const long long nb = std::max<long long>(1, std::min<long long>(ni, (long long)k * sms * kWarps / nstrips));
    const int sl = (int)((ni + nb - 1) / nb);
    const long long ctas = (((long long)ni + sl - 1) / sl * nstrips + kWarps - 1) / kWarps;
    const double per_sm = (double)((ctas + sms - 1) / sms);
    const double cost = (sl + extra) * std::max(1.3, per_sm);  // a warp alone does not fill the pipe
    if (cost < best) {
      best = cost;
      best_sl = sl;
    }
    if (nb == ni) break;
  }
  return best_sl;
}

template <class ST, int B, bool COEF> cudaError_t launch(const AdjStep2D &a, cudaStream_t stream) {
  using AP = AdjPipe2D<ST, B, COEF>;
  auto kern = adj2d_kernel<ST, B, COEF>;
  constexpr size_t smem = AP::SMEM;
  if (smem > kOptInSmem) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return e;
    }
  }
  const AdjGeom &g = *a.g;
  AdjParams2D<ST::kTerms> p;
  p.lam = static_cast<const T *>(a.lam);
  p.u = static_cast<const T *>(a.u);
  p.lam_out = static_cast<T *>(a.lam_out);
  p.hg = static_cast<T *>(a.hg);
  p.part = a.part;
  p.pitch = g.pitch;
  p.u_stride = g.plane;
  p.d0 = g.d0;
  p.d1 = g.d1;
  p.shift = g.shift;
  for (int t = 0; t < ST::kTerms; ++t) p.coef[t] = (T)(a.coef[t] / a.div);
  p.inv_div = (T)(1.0 / a.div);
  const int ni = g.d0 - 2 * ST::kRad, nj = g.d1 - 2 * ST::kRad;
  p.nstrips = (nj + AP::WOUT - 1) / AP::WOUT;
  // the blocks of the largest degree, for every degree (see above)
  constexpr int M = max_degree<ST, COEF>();
  static_assert(AdjPipe2D<ST, M, COEF>::WOUT == AP::WOUT || !COEF, "one decomposition for every degree");
  const int wave = adj_wave(reinterpret_cast<const void *>(adj2d_kernel<ST, M, COEF>), kWarps * 32,
                            AdjPipe2D<ST, M, COEF>::SMEM);
  // a block's sums cost about as much as a dozen rows (radius 1)
  int sl = AP::FILL ? fill_rows(p.nstrips, ni, COEF ? 9 : 3)
                    : stream_rows_2d(p.nstrips, ni, M * ST::kRad + (COEF ? 6 : 0), false, (long long)wave * kWarps);
  // The edge strips' rows cost more (masks, halo gradient), and all warps start
  // together: without products, a third of the rows per block there (four
  // steps of a 2048^2 grid 21.8 us with the same rows, 18.6 with half, 14.8
  // with a third); with products, which every row has, the same (two steps
  // 19.3, 20.1, 21.0 us). In double, bound by the FP64 pipe, the same as well
  // (star2d1r 1500^2, 20 steps with the forward pass: 1512 us with a third, 1301).
  const int edges = p.nstrips > 1 ? 2 : 1;
  // With products every CTA of a launch has its own row of the partial-sum
  // table: blocks as long as that takes, and where one block per strip is
  // still too many (more than 4096 strips), several launches over the items.
  constexpr long long kMost = (long long)kAdjPartRows * kWarps;
  long long items = 0;
  for (;; ++sl) {
    p.sl = sl;
    p.nblocks = (ni + sl - 1) / sl;
    p.sl_e = COEF || AP::FILL ? sl : (sl + 2) / 3;
    p.nblocks_e = (ni + p.sl_e - 1) / p.sl_e;
    items = (long long)edges * p.nblocks_e + (long long)(p.nstrips - edges) * p.nblocks;
    if (items <= kMost || sl >= ni) break;
  }
  const long long most = COEF ? kMost : items;
  for (p.item0 = 0; p.item0 < items; p.item0 += most) {
    const unsigned grid = (unsigned)((std::min(most, items - p.item0) + kWarps - 1) / kWarps);
    const cudaError_t e = launch_kernel(kern, grid, kWarps * 32, smem, stream, p);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <class ST, bool COEF> void fill(AdjStep2DFn (&f)[kAdjMaxB + 1]) {
  constexpr int m = max_degree<ST, COEF>();
  f[1] = &launch<ST, 1, COEF>;
  if constexpr (m >= 2) f[2] = &launch<ST, 2, COEF>;
  if constexpr (m >= 4) f[4] = &launch<ST, 4, COEF>;

}

}  // namespace

AdjPicks2D GBS_PICK() {
  static_assert(S::kDim == 2 && S::kKind == KIND_LINEAR && S::kTerms <= kMaxCoefGrad, "2-D linear stencils");
  AdjPicks2D p{};
  fill<S, false>(p.step[0]);
  fill<S, true>(p.step[1]);
  return p;
}
}  // namespace gbs
