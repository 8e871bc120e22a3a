// 2-D temporally-blocked stencil kernel family (sm_103a).
//
// Replaces the AN5D-generated 2-D kernels kernel0_<b> (e.g.
// compiled/float/star2d1r-256-10-256_kernel.cu:4..3488) and computes what
// the artifact's scop loop computes (star2d1r.c:14-24 and the other 2-D
// sources): b Jacobi steps of A[(t+1)%2][i][j] = f(A[t%2][neighbourhood]) on
// the interior, the halo held fixed.
//
// Work decomposition. One WARP is the unit of work; warps never wait on each
// other. A warp owns a strip of output columns [cs, ce) (wout wide) and a
// block of output rows [i0, i1) (sl long). Lane l holds the V columns
// [l*V, l*V+V) of the strip's 32*V-column window, one 16-byte vector per row
// (V = 4 for float, 2 for double).
//
// Row pipeline. Level-0 rows i0-b*r .. i1-1+b*r stream through a ring of
// row buffers in shared memory, filled by 16-byte cp.async copies: every
// lane copies its own columns and reads back only what it copied, so a row
// needs no barrier, no vote and no elected lane. Rows are handled in groups
// of kNph (the unroll of the row loop): one commit and one wait per group,
// kPrefetch groups in flight ahead of the one being computed.
//
// Per fused time level l (1..b) the warp keeps a (2r+1)-row register window.
// At pipeline step p (level-0 row p arrives) level l produces row p - l*r,
// which feeds level l+1 in the same step; level b's row p - b*r is stored if
// it lies in [i0, i1). Row neighbours at other column offsets come from the
// neighbouring lanes by shuffles. The window's edge lanes (b*r columns at
// each side) lose accuracy level by level; they are the overlap that
// neighbouring strips compute for real (overlapped tiling), so no warp ever
// needs another warp's result.
//
// Two evaluation forms, chosen per stencil by the tap-table generator:
//  * direct: the window holds the input rows; each output is one chain over
//    the terms in source order. Used for stars, gradient2d and star2d4r.
//  * assoc:  the window holds partial sums of the 2r+1 outputs in flight;
//    each arriving row adds its terms to every output it touches. Used for
//    stencils whose source groups the terms by ascending row (the boxes,
//    j2d9pt-gol), where the partial sums are built in exactly the source
//    order, so both forms give the same bits.
//
// Halo cells (rows/columns within r of the grid edge) carry their input
// value through every level, like the reference's untouched halo.
#pragma once
#include "gbs_device.cuh"
#include "gbs_launch.h"
#include "stencil_table.cuh"

namespace gbs {

template <typename T, int NT> struct Params2D {
  const T *src;        // plane read (row 0, element 0 of the padded row)
  T *dst;              // plane written
  long long pitch;     // elements per padded row
  int d0, d1;          // dimsize: rows, columns (interior + 2r)
  int shift;           // column c is stored at element shift + c
  int nstrips, nblocks, sl;  // strips of Pipe2D::WOUT columns, stream blocks of sl rows
  T coef[NT];
  T div, rdiv, eps;    // divisor, RN(1/divisor), gradient epsilon
  int divmode;         // 0: no division (folded into coef), 1: checked, 2: proven fast path
  T *stash;            // stash-mode kernels: level l < b also stores its interior cells to
  long long stash_stride;  // stash + (l-1)*stash_stride (the states between)
};

// y / div for a lane's elements, as the params ask (see div_by / div_by_fast)
template <typename T, int V, int NT>
__device__ __forceinline__ void apply_div(T (&y)[V], const Params2D<T, NT> &p) {
  if constexpr (sizeof(T) == 4) {
    if (p.divmode == 2) {
      div_by_fast(y, p.div, p.rdiv);
      return;
    }
  }
  if (p.divmode == 0) return;
#pragma unroll
  for (int e = 0; e < V; ++e) y[e] = div_by(y[e], p.div, p.rdiv);
}

// Compile-time facts about a stencil's term list.
template <class ST, int V> struct Tap2 {
  static constexpr int R = ST::kRad;
  static constexpr int NT = ST::kTerms;
  // does some term read row offset di at element x (x relative to the lane's
  // first element, x in [-R, V+R))?
  __host__ __device__ static constexpr bool need(int di, int x) {
    if (ST::kKind == KIND_GRADIENT && di == 0 && x >= 0 && x < V) return true;
    for (int t = 0; t < NT; ++t)
      if (ST::kOff[t][0] == di) {
        const int e = x - ST::kOff[t][1];
        if (e >= 0 && e < V) return true;
      }
    return false;
  }
  __host__ __device__ static constexpr bool row_has_dj(int di) {
    for (int t = 0; t < NT; ++t)
      if (ST::kOff[t][0] == di && ST::kOff[t][1] != 0) return true;
    if (ST::kKind == KIND_GRADIENT) return false;
    return false;
  }
};

// ext[R + x] = row element x, x in [-R, V+R), for the x some term needs.
template <class ST, int V, int DI, typename T>
__device__ __forceinline__ void extend_row(T (&ext)[V + 2 * ST::kRad], const T (&row)[V]) {
  constexpr int R = ST::kRad;
  static_for<V + 2 * R>([&](auto XI) {
    constexpr int x = decltype(XI)::value - R;
    if constexpr (Tap2<ST, V>::need(DI, x)) ext[R + x] = row_elem<V, x>(row);
  });
}


// Shape of a warp's row pipeline for (stencil, element type, degree).
template <class ST, typename T, int B, bool FMA> struct Pipe2D {
  static constexpr int R = ST::kRad;
  static constexpr int W = 2 * R + 1;
  // One 16-byte vector per lane. (Two for double, whose 128-column window
  // would lose half as large a share of its lanes to the overlap, measured
  // 3% to 14% slower at degree 1: j2d9pt f64 8192^2 1272 us a step against
  // 1240, box2d1r 4096^2 326 against 286.)
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int COLS = 32 * V;
  static constexpr unsigned ROWB = 512;           // bytes of one ring row
  // The row loop is unrolled over the window's W positions, which rotates the
  // window by renaming, where that body stays within about 1300 instructions
  // (20 KB; it exists once per Care2D). Larger ones slide a window of
  // W + kNph - 1 rows and move it once per kNph rows, as many as about 800
  // instructions hold: box2d4r f32 at 4096^2 took 79 us a step unrolled by
  // three and 69 us by one or two, box2d2r at degree 2 within 3% either way,
  // star2d3r at degree 3 22 us by four and 20 us by seven. (Instructions of
  // one row: the sums, a dozen for shuffles and window per level, the copy
  // and the store.)
  static constexpr int ROW_INSTR = B * (ST::kTerms * V * (FMA ? 1 : 2) + (ST::kHasDiv && !FMA ? 36 : 0) + 12) + 14;
  static constexpr bool ROT = sizeof(T) == 8 || W * ROW_INSTR <= 1300;
  static constexpr int SLIDE = 800 / ROW_INSTR;
  static constexpr int NPH = ROT ? W : (SLIDE < 1 ? 1 : (SLIDE > W - 1 ? W - 1 : SLIDE));
  static constexpr int WSLOTS = ROT ? W : W + NPH - 1;
  // groups in flight ahead of the one being computed: at least 8 rows for
  // float; 4 for double, whose larger ring would cost resident CTAs
  static constexpr int PG = ((sizeof(T) == 8 ? 4 : 8) + NPH - 1) / NPH;
  // level-0 rows kept after they arrive: the assoc form's halo cells take
  // their fixed values (of rows up to b*r back) from the ring
  static constexpr int KEEP = ST::kAssoc ? B * R : 0;
  static constexpr int KG = (KEEP + NPH - 1) / NPH;
  static constexpr int NROWS = (PG + 1 + KG) * NPH;  // rows of the ring
  static constexpr unsigned RING = NROWS * ROWB;     // bytes per warp
  // columns of the window left of the first output column: the overlap b*r
  // rounded up to whole lanes, so that a lane's vector is stored whole
  static constexpr int ML = (B * R + V - 1) / V * V;
  static constexpr int WOUT = (COLS - ML - B * R) / V * V;
};

// the lane's elements of a ring row (p: the row + lane * 16)
template <class PP, typename T>
__device__ __forceinline__ void ld_ring(T (&x)[PP::V], const unsigned char *p) {
  ld_vec<T, PP::V>(x, reinterpret_cast<const T *>(p));
}

// window slot of logical position j (0 = oldest row) in phase ph
template <class PP> __host__ __device__ constexpr int slot2d(int ph, int j) {
  return PP::ROT ? (ph + 1 + j) % PP::W : ph + j;
}

// Halo values for the assoc form: the level-0 row q of the lane, in the ring
// for b*r rows after it arrived. Read unconditionally, ahead of the sums that
// hide its latency; for a row that was never loaded the ring's stale contents
// reach only rows and columns that no output needs.
template <class PP> struct CarryRing {
  const unsigned char *ring;  // the warp's ring + lane * 16
  int cur, cur_row;           // ring row index and grid row of the group's first row
  template <typename T> __device__ __forceinline__ void row(T (&x)[PP::V], int q) const {
    int s = cur + (q - cur_row);
    if (s < 0) s += PP::NROWS;
    ld_ring<PP>(x, ring + (unsigned)s * PP::ROWB);
  }
};

// What a group of rows may meet. Three copies of the row code: all warps of a
// launch start together, so the strips at the grid's left and right edge set
// its end if their rows cost much more than the others' (with the halo-row
// tests in every edge row, branches and late ring reads, box2d1r f32 at
// 4096^2, degree 4, took 13.8 us a step; 10.0 now).
enum Care2D : int {
  kInterior = 0,  // interior rows and columns only
  kColumns = 1,   // halo columns (a strip at the grid's left or right edge), interior rows
  kAll = 2        // halo rows as well
};

// One fused time level: the level-(l) row x arrives, the level-(l+1) row q
// leaves in x. up (gradient2d): the squared differences between rows q-1 and q,
// which the step of row q-1 formed.
// The sums of the few overlap rows that no output needs are computed all the
// same: a test per row and level costs more than it saves, on the FP64 pipe
// too (star2d1r f64 16384^2 2755 us a step with it, 2444 without).
template <class ST, class PP, typename T, bool FMA, int CARE, int PH>
__device__ __forceinline__ void level2d(T (&win)[PP::WSLOTS][PP::V], T (&up)[PP::V], T (&x)[PP::V], int q,
                                        const bool (&fixed)[PP::V], const CarryRing<PP> &carry,
                                        const Params2D<T, ST::kTerms> &p) {
  constexpr int R = ST::kRad;
  constexpr int V = PP::V;
  using A = Arith<T>;
  T y[V];
  bool halo_row = false;
  if constexpr (CARE == kAll) halo_row = (q < R) || (q >= p.d0 - R);
  // the constant divisor (FMA mode folds it into the coefficients). Columns
  // that keep their halo value are off the grid too, where memory or the ring
  // holds anything: a 1 there, or one zero or denormal sends its warp through
  // the rare path of the division in every row (j2d9pt-gol f32 1500^2, degree
  // 4: 9.9 us a step, 5.8 now)
  auto divide = [&]() GBS_INL {
    if constexpr (ST::kHasDiv && !FMA) {
      if constexpr (CARE != kInterior) {
#pragma unroll
        for (int e = 0; e < V; ++e) y[e] = halo_row || fixed[e] ? T(1) : y[e];
      }
      apply_div(y, p);
    }
  };
  if constexpr (!ST::kAssoc) {
#pragma unroll
    for (int e = 0; e < V; ++e) win[slot2d<PP>(PH, 2 * R)][e] = x[e];
    constexpr int cslot = slot2d<PP>(PH, R);
    if constexpr (ST::kKind == KIND_GRADIENT) {
      // the squared differences in source order (up, down, right, left). Each
      // is one of two cells' (u - u_n and u_n - u are exact negatives, so the
      // squares are equal): the upper one was the row above's lower one, the
      // left one is the left neighbour's right one. 14 FP64 operations a
      // cell instead of 25.
      static_assert(ST::kTerms == 4 && R == 1 && ST::kOff[0][0] == -1 && ST::kOff[1][0] == 1 &&
                        ST::kOff[2][1] == 1 && ST::kOff[3][1] == -1, "neighbours: up, down, right, left");
      const T(&c)[V] = win[cslot];
      const T(&below)[V] = win[slot2d<PP>(PH, 2)];
      const T after = row_elem<V, V>(c);
      T sr[V];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const T d = A::sub(c[e], e + 1 < V ? c[e + 1 < V ? e + 1 : e] : after);
        sr[e] = A::mul(d, d);
      }
      const T sl = shfl_up(sr[V - 1], 1);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const T d = A::sub(c[e], below[e]);
        const T sd = A::mul(d, d);
        T s = A::add(A::add(A::add(A::add(p.eps, up[e]), sd), sr[e]), e > 0 ? sr[e > 0 ? e - 1 : 0] : sl);
        if constexpr (CARE != kInterior) s = halo_row || fixed[e] ? T(1) : s;  // as for the quotients below
        up[e] = sd;
        y[e] = gradient_finish<T, FMA>(c[e], s, p.coef[0]);
      }
    } else {
      // the direct form serves stencils whose off-centre rows are read at
      // the centre column only (stars, star2d4r): one extended row
      T ext[V + 2 * R];
      extend_row<ST, V, 0>(ext, win[cslot]);
      static_for<ST::kTerms>([&](auto TI) GBS_INL {
        constexpr int t = decltype(TI)::value;
        constexpr int di = ST::kOff[t][0], dj = ST::kOff[t][1];
        static_assert(di == 0 || dj == 0, "direct 2-D form expects off-centre rows at dj == 0");
        constexpr int slot = slot2d<PP>(PH, R + di);
        static_for<V>([&](auto EI) GBS_INL {
          constexpr int e = decltype(EI)::value;
          T a;
          if constexpr (dj == 0) a = win[slot][e];
          else a = ext[R + e + dj];
          if constexpr (t == 0) y[e] = A::mul(p.coef[t], a);
          else y[e] = term_next<T, FMA>(y[e], p.coef[t], a);
        });
      });
      divide();
    }
    if constexpr (CARE != kInterior) {
#pragma unroll
      for (int e = 0; e < V; ++e) y[e] = (halo_row || fixed[e]) ? win[cslot][e] : y[e];
    }
  } else {
    // assoc: the arriving row m = q + R adds its terms to outputs q..q+2R
    T cv[V];
    if constexpr (CARE != kInterior) carry.row(cv, q);
    T ext[V + 2 * R];
    static_for<V + 2 * R>([&](auto XI) GBS_INL {
      constexpr int xx = decltype(XI)::value - R;
      constexpr bool any = [] {
        for (int di = -R; di <= R; ++di)
          if (Tap2<ST, V>::need(di, xx)) return true;
        return false;
      }();
      if constexpr (any) ext[R + xx] = row_elem<V, xx>(x);
    });
    // term by term in source order, one row offset after the other
    static_for<PP::W>([&](auto DI) GBS_INL {
      constexpr int di = decltype(DI)::value - R;
      static_for<ST::kTerms>([&](auto TI) GBS_INL {
        constexpr int t = decltype(TI)::value;
        if constexpr (ST::kOff[t][0] == di) {
          constexpr int dj = ST::kOff[t][1];
          constexpr int slot = slot2d<PP>(PH, R - di);
          static_for<V>([&](auto EI) GBS_INL {
            constexpr int e = decltype(EI)::value;
            const T a = ext[R + e + dj];
            if constexpr (t == 0) win[slot][e] = A::mul(p.coef[t], a);
            else win[slot][e] = term_next<T, FMA>(win[slot][e], p.coef[t], a);
          });
        }
      });
    });
    constexpr int oslot = slot2d<PP>(PH, 0);
#pragma unroll
    for (int e = 0; e < V; ++e) y[e] = win[oslot][e];
    divide();
    if constexpr (CARE != kInterior) {
#pragma unroll
      for (int e = 0; e < V; ++e) y[e] = (halo_row || fixed[e]) ? cv[e] : y[e];
    }
  }
#pragma unroll
  for (int e = 0; e < V; ++e) x[e] = y[e];
}

// One work item of a warp: output columns [cs, ce) of strip `strip` and
// output rows [i0, i1) of stream block `blk`, advanced by B levels from p.src
// into p.dst. `ring` is the warp's Pipe2D::RING bytes of shared memory
// (16-byte aligned), owned by this warp.
// STASH: the intermediate levels also store their rows (the states after 1
// .. B-1 steps) in the item's output rows and columns, where every level is
// valid, to p.stash; a separate instantiation, so that the plain kernels
// carry none of it.
//
// What bounds it and what it measured: see stencil2d_kernel.
template <class ST, typename T, int B, bool FMA, bool STASH = false>
__device__ __forceinline__ void warp_item2d(const Params2D<T, ST::kTerms> &p, int strip, int blk,
                                            unsigned char *ring) {
  using PP = Pipe2D<ST, T, B, FMA>;
  constexpr int V = PP::V, R = PP::R, NPH = PP::NPH, PG = PP::PG;
  const int lane = threadIdx.x & 31;

  // ---- columns (column space c; element space c + shift) ----
  const int cs = R + strip * PP::WOUT;
  const int ce = min(cs + PP::WOUT, p.d1 - R);
  const int ws = cs + p.shift - PP::ML;          // element of the window's column 0 (may be negative)
  const int el = ws + lane * V;                  // this lane's first element
  const int col0 = el - p.shift;                 // and its column
  const bool edge = (ws - p.shift < R) || (ws - p.shift + PP::COLS > p.d1 - R);
  const bool store_all = (col0 >= cs && col0 + V <= ce);
  bool fixed[V];                                 // halo columns (and columns off the grid)
#pragma unroll
  for (int e = 0; e < V; ++e) fixed[e] = (col0 + e < R || col0 + e >= p.d1 - R);

  // ---- rows ----
  const int i0 = R + blk * p.sl;
  const int i1 = min(i0 + p.sl, p.d0 - R);
  const int pstart = max(0, i0 - B * R);
  const int pend = min(p.d0, i1 + B * R);        // rows loaded: [pstart, pend)
  const int ng = (i1 + B * R - pstart + NPH - 1) / NPH;
  // rows [fast_lo, fast_hi): every level's row is interior (or not needed)
  const int fast_lo = i0 >= B * R ? pstart : (B + 1) * R;
  const int fast_hi = i1 + B * R <= p.d0 ? 0x7fffffff : p.d0;

  // ---- copies: lane-private, one vector per row ----
  unsigned char *my = ring + lane * 16;
  const uint32_t my_s = smem_u32(my);
  const bool in_row = el >= 0 && el + V <= p.pitch;
  const T *ld = p.src + (long long)pstart * p.pitch + el;
  int ld_left = pend - pstart;                   // rows not yet requested
  unsigned wr = 0;                               // byte offset of the next group's first row
  auto request_group = [&]() GBS_INL {
#pragma unroll
    for (int ph = 0; ph < NPH; ++ph) {
      if (in_row && ph < ld_left) cp_async16(my_s + wr + (unsigned)ph * PP::ROWB, ld);
      ld += p.pitch;
    }
    cp_async_commit();
    ld_left -= NPH;
    wr = wr + NPH * PP::ROWB == PP::RING ? 0u : wr + NPH * PP::ROWB;
  };
#pragma unroll 1
  for (int g = 0; g < PG; ++g) request_group();

  T win[B][PP::WSLOTS][V];
#pragma unroll
  for (int l = 0; l < B; ++l)
#pragma unroll
    for (int w = 0; w < PP::WSLOTS; ++w)
#pragma unroll
      for (int e = 0; e < V; ++e) win[l][w][e] = T(0);

  T up[B][V];  // see level2d
#pragma unroll
  for (int l = 0; l < B; ++l)
#pragma unroll
    for (int e = 0; e < V; ++e) up[l][e] = T(0);

  unsigned rd = 0;                               // byte offset of the group being computed
  T *st = p.dst + (long long)(pstart - B * R) * p.pitch + el;  // row the last level stores in the first step
  T *ss = STASH ? p.stash + (long long)pstart * p.pitch + el : nullptr;
  const unsigned nout = (unsigned)(i1 - i0);
  int pb = pstart;                               // row of the group's phase 0

  // rows pb .. pb+NPH-1, with what CAREI (Care2D) says they meet. Rows past the item's last are computed from
  // whatever the ring holds and never stored; in double, where the FP64 pipe bounds the loop, the last group takes
  // the copy of all cases and leaves them out (box2d2r f64 500x900, 7 rows and 4 of overlap in groups of 5: 49.9 us
  // a step with them, 37.9 without; j2d9pt f64 200x300 13.0, 11.7; star2d1r f64 16384^2 2458, 2460).
  auto rows = [&](auto CAREI) GBS_INL {
    constexpr int care = decltype(CAREI)::value;
    const CarryRing<PP> carry{my, (int)(rd / PP::ROWB), pb};
    static_for<NPH>([&](auto PHI) GBS_INL {
      constexpr int ph = decltype(PHI)::value;
      const int pp = pb + ph;
      if constexpr (sizeof(T) == 8 && care == kAll) {
        if (pp >= i1 + B * R) return;
      }
      T x[V];
      ld_ring<PP>(x, my + rd + (unsigned)ph * PP::ROWB);
      // the lane's columns of an output row; outside the edge strips a lane is
      // stored whole or not at all
      auto store = [&](T *d, bool on) GBS_INL {
        st_vec_global_if<V>(d, x, on && store_all);
        if constexpr (care != kInterior) {
#pragma unroll
          for (int e = 0; e < V; ++e) st_global_if(d + e, x[e], on && !store_all && col0 + e >= cs && col0 + e < ce);
        }
      };
      static_for<B>([&](auto LI) GBS_INL {
        constexpr int l = decltype(LI)::value;
        level2d<ST, PP, T, FMA, care, ph>(win[l], up[l], x, pp - (l + 1) * R, fixed, carry, p);
        if constexpr (STASH && l + 1 < B) {
          store(ss + (long long)l * p.stash_stride - (long long)((l + 1) * R) * p.pitch,
                (unsigned)(pp - (l + 1) * R - i0) < nout);
        }
      });
      store(st, (unsigned)(pp - B * R - i0) < nout);
      st += p.pitch;
      if constexpr (STASH) ss += p.pitch;
    });
    if constexpr (!PP::ROT) {
#pragma unroll
      for (int l = 0; l < B; ++l)
#pragma unroll
        for (int j = 0; j < 2 * R; ++j)
#pragma unroll
          for (int e = 0; e < V; ++e) win[l][j][e] = win[l][j + NPH][e];
    }
  };

#pragma unroll 1
  for (int g = 0; g < ng; ++g) {
    request_group();           // group g + PG, into the slot freed by the group before the kept ones
    cp_async_wait<PG>();       // group g has landed (this lane's own copies)
    if (pb < fast_lo || pb + NPH > fast_hi || (sizeof(T) == 8 && pb + NPH > i1 + B * R)) rows(IC<kAll>());
    else if (edge) rows(IC<kColumns>());
    else rows(IC<kInterior>());
    pb += NPH;
    rd = rd + NPH * PP::ROWB == PP::RING ? 0u : rd + NPH * PP::ROWB;
  }
  cp_async_wait<0>();          // nothing in flight into the ring when the next item starts
}

constexpr int kWpc2D = kWarpsPerCta2D;

template <class ST, typename T, int B, bool FMA> constexpr size_t smem_bytes2d() {
  return (size_t)kWpc2D * Pipe2D<ST, T, B, FMA>::RING;
}

// Bound: instruction issue at degree 2 and above for float (HBM at degree 1),
// the FP64 pipe for double. A row of star2d1r at degree 4 takes 123 warp
// instructions for its 80 multiplies and FMAs (degree 7: 202 for 140), issued
// 73% of the time; with one bulk copy per row, its mbarrier wait, vote and
// elected refill it took 191. Measured (GB300, time per step at the tuned
// degree, with those copies -> here): star2d1r f32 4096^2 13.2 us (degree 4) ->
// 6.7 (8); j2d5pt f32 16384^2 125 -> 80; box2d2r f32 3001x2217 24.5 -> 11.7;
// j2d9pt f64 1777x2500 132 (2) -> 84 (1; its FP64 pipe 92% busy); j2d9pt-gol
// f32 2048^2, exact mode, 22.4 (1) -> 8.8 (4).
template <class ST, typename T, int B, bool FMA, bool STASH = false>
__global__ void __launch_bounds__(kWpc2D * 32, gbs_min_ctas(kWpc2D * 32))
    stencil2d_kernel(const __grid_constant__ Params2D<T, ST::kTerms> p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int w = threadIdx.x >> 5;
  const long long gw = (long long)blockIdx.x * kWpc2D + w;
  if (gw >= (long long)p.nstrips * p.nblocks) return;
  warp_item2d<ST, T, B, FMA, STASH>(p, (int)(gw % p.nstrips), (int)(gw / p.nstrips),
                                    smem_raw + (size_t)w * Pipe2D<ST, T, B, FMA>::RING);
}

// opts the kernel in to its shared memory (above 48 KB the default refuses the launch)
template <class K> cudaError_t allow_smem2d(K kern, size_t smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

template <class ST, typename T, int B, bool FMA>
int occupancy2d() {
  constexpr size_t smem = smem_bytes2d<ST, T, B, FMA>();
  auto kern = stencil2d_kernel<ST, T, B, FMA>;
  int nb = 0;
  if (allow_smem2d(kern, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kWpc2D * 32, smem) != cudaSuccess)
    return 0;
  return nb * kWpc2D;
}

template <class ST, typename T, int B, bool FMA, bool STASH = false>
cudaError_t launch2d(const Launch2D &a, cudaStream_t stream) {
  constexpr size_t smem = smem_bytes2d<ST, T, B, FMA>();
  auto kern = stencil2d_kernel<ST, T, B, FMA, STASH>;
  if (STASH != (a.stash != nullptr) || a.wout != Pipe2D<ST, T, B, FMA>::WOUT) return cudaErrorInvalidValue;
  if (const cudaError_t e = allow_smem2d(kern, smem); e != cudaSuccess) return e;
  Params2D<T, ST::kTerms> p;
  p.src = static_cast<const T *>(a.src);
  p.dst = static_cast<T *>(a.dst);
  p.pitch = a.pitch;
  p.d0 = a.d0;
  p.d1 = a.d1;
  p.shift = a.shift;
  p.nstrips = a.nstrips;
  p.nblocks = a.nblocks;
  p.sl = a.sl;
  // FMA mode is tolerance-bound: a divisor (nonzero, checked by the planner)
  // is folded into the coefficients, and the kernel has no division at all
  const bool fold = FMA && ST::kHasDiv;
  for (int t = 0; t < ST::kTerms; ++t) p.coef[t] = fold ? (T)(a.coef[t] / a.div) : (T)a.coef[t];
  p.divmode = !ST::kHasDiv || fold ? 0 : (a.div_proven ? 2 : 1);
  p.div = (T)a.div;
  p.rdiv = div_reciprocal<T>(a.div);
  p.eps = (T)a.eps;
  p.stash = static_cast<T *>(a.stash);
  p.stash_stride = a.stash_stride;
  const long long warps = (long long)a.nstrips * a.nblocks;
  const long long grid = (warps + kWpc2D - 1) / kWpc2D;
  return launch_kernel(kern, (unsigned)grid, kWpc2D * 32, smem, stream, p);
}

// Parameters of one item, from its grid's table entry into p (coefficients by
// the whole warp; every lane must call it, and p is either every lane's own or
// shared by the warp).
template <class ST>
__device__ __forceinline__ void batch_params(Params2D<float, ST::kTerms> &p, const BatchGridDev &g, int k, int sl) {
  p.src = g.base + (long long)(k % 2) * g.plane;
  p.dst = g.base + (long long)((k + 1) % 2) * g.plane;
  p.pitch = g.pitch;
  p.d0 = g.d0;
  p.d1 = g.d1;
  p.shift = g.shift;
  p.nstrips = 0;
  p.nblocks = 0;
  p.sl = sl;
  p.div = g.div;
  p.rdiv = g.rdiv;
  p.eps = g.eps;
  p.divmode = g.divmode;
  p.stash = nullptr;
  p.stash_stride = 0;
}
// bytes of the per-warp shared-memory slot that holds an item's parameters
// where they do not fit in registers
constexpr int kParamSlot = 512;
static_assert(sizeof(Params2D<float, kBatchMaxTerms>) <= kParamSlot, "parameter slot too small");

// Layered batched schedule: one time block of the grids of one stencil at one
// degree, warp w running item first + w. One kernel per (stencil, degree), so
// that each gets its own registers and a layer's launches of different
// stencils need not wait for each other; one kernel that dispatched on the
// stencil ran every variant at 128 registers and each layer as long as its
// slowest item: 48 grids of 128..2048 cells a side, up to 128 steps,
// 9.0 ms -> 4.1 (GB300); the 512-grid mix of the benchmark 370 -> 690 GCells/s.
template <class ST, int B, bool FMA>
__global__ void __launch_bounds__(kWpc2D * 32)
    batch_family_kernel(const BatchGridDev *__restrict__ grids, const BatchItem *__restrict__ items, int count) {
  constexpr bool SLOT = ST::kTerms > 25;  // more coefficients than registers to spare
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int w = threadIdx.x >> 5;
  const long long gw = (long long)blockIdx.x * kWpc2D + w;
  if (gw >= count) return;
  const BatchItem it = items[gw];
  const BatchGridDev &g = grids[it.grid];
  unsigned char *ring = smem_raw + (size_t)w * Pipe2D<ST, float, B, FMA>::RING;
  if constexpr (SLOT) {
    auto &p = *reinterpret_cast<Params2D<float, ST::kTerms> *>(
        smem_raw + (size_t)kWpc2D * Pipe2D<ST, float, B, FMA>::RING + (size_t)w * kParamSlot);
    for (int t = threadIdx.x & 31; t < ST::kTerms; t += 32) p.coef[t] = g.coef[t];
    if ((threadIdx.x & 31) == 0) batch_params<ST>(p, g, it.k, it.sl);
    __syncwarp();
    warp_item2d<ST, float, B, FMA>(p, it.strip, it.blk, ring);
  } else {
    Params2D<float, ST::kTerms> p;
    batch_params<ST>(p, g, it.k, it.sl);
#pragma unroll
    for (int t = 0; t < ST::kTerms; ++t) p.coef[t] = g.coef[t];
    warp_item2d<ST, float, B, FMA>(p, it.strip, it.blk, ring);
  }
}

template <class ST, int B, bool FMA>
cudaError_t batch_launch(const BatchGridDev *grids, const BatchItem *items, int first, int count, cudaStream_t stream) {
  constexpr size_t smem = smem_bytes2d<ST, float, B, FMA>() + (ST::kTerms > 25 ? kWpc2D * kParamSlot : 0);
  auto kern = batch_family_kernel<ST, B, FMA>;
  if (const cudaError_t e = allow_smem2d(kern, smem); e != cudaSuccess) return e;
  return launch_kernel(kern, (unsigned)((count + kWpc2D - 1) / kWpc2D), kWpc2D * 32, smem, stream, grids,
                       items + first, count);
}

}  // namespace gbs
