// Device-side building blocks shared by the stencil kernels: bulk-async
// (TMA) copies with mbarrier completion, bounded waits, lane shuffles,
// 16-byte vector access and the two floating-point evaluation modes.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>
#include <utility>

// Register cap of a build variant (0: none). A kernel of `threads` threads
// asks for at least 65536 / (threads * cap) resident CTAs per SM, which
// limits it to about `cap` registers per thread.
#ifndef GBS_REGCAP
#define GBS_REGCAP 0
#endif
constexpr int gbs_min_ctas(int threads) {
  return GBS_REGCAP > 0 && 65536 / (threads * GBS_REGCAP) > 1 ? 65536 / (threads * GBS_REGCAP) : 1;
}

namespace gbs {

// Error bits a kernel ORs into the launch's error word.
enum : int {
  ERR_WAIT_TIMEOUT = 1,   // an mbarrier wait exceeded its time limit
  ERR_DRAIN_TIMEOUT = 2,  // draining in-flight copies after a timeout gave up
  ERR_DEP_TIMEOUT = 4,    // a dependency wait (batched scheduler) gave up
};

// Wall-clock limit of every spin-wait, in nanoseconds (about one second).
constexpr unsigned long long kWaitLimitNs = 1000ull * 1000ull * 1000ull;

template <int N> using IC = std::integral_constant<int, N>;

// Forces a lambda inline. A lambda the compiler keeps as a call (it did so
// for the row loop of a kernel variant inside the batched dispatcher) has
// its captured locals, the register windows among them, in local memory.
#define GBS_INL __attribute__((always_inline))

// Compile-time loop: f(IC<0>), ..., f(IC<N-1>).
template <int N, class F, int... Is>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, Is...>) {
  (f(IC<Is>()), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
  static_for_impl<N>(std::forward<F>(f), std::make_integer_sequence<int, N>());
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for phase `parity` of `bar` to complete, for at most kWaitLimitNs.
// Returns false (and sets `code` in *err) when the limit is reached.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, int *err, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > kWaitLimitNs) {
      if (err) atomicOr(err, code);
      return false;
    }
  }
}

// ---- bulk async copies (TMA, non-tensor form) --------------------------------
// global -> shared, completion counted in bytes on `bar`. Both addresses must
// be 16-byte aligned and `bytes` a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// ---- per-thread async copies (16 bytes, L2 only) ------------------------------
// global -> shared, completed per thread: a thread that waits for its own
// groups may read what it copied itself, with no barrier.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most N of this thread's newest groups are still in flight
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- vectors of V elements (16 bytes) ----------------------------------------
template <typename T, int V> struct alignas(16) Vec { T v[V]; };

template <typename T, int V>
__device__ __forceinline__ void ld_vec(T (&x)[V], const T *p) {
  const Vec<T, V> t = *reinterpret_cast<const Vec<T, V> *>(p);
#pragma unroll
  for (int e = 0; e < V; ++e) x[e] = t.v[e];
}
template <typename T, int V>
__device__ __forceinline__ void ld_vec_global(T (&x)[V], const T *p) {
  Vec<T, V> t;
  if constexpr (sizeof(T) * V == 16) {
    // cached in L2 only: a batched launch rewrites grids it reads
    if constexpr (std::is_same<T, float>::value) {
      float4 f = __ldcg(reinterpret_cast<const float4 *>(p));
      t.v[0] = f.x; t.v[1] = f.y; t.v[2] = f.z; t.v[3] = f.w;
    } else {
      double2 f = __ldcg(reinterpret_cast<const double2 *>(p));
      t.v[0] = f.x; t.v[1] = f.y;
    }
  } else {
    t = *reinterpret_cast<const Vec<T, V> *>(p);
  }
#pragma unroll
  for (int e = 0; e < V; ++e) x[e] = t.v[e];
}
template <typename T, int V>
__device__ __forceinline__ void st_vec(T *p, const T (&x)[V]) {
  Vec<T, V> t;
#pragma unroll
  for (int e = 0; e < V; ++e) t.v[e] = x[e];
  *reinterpret_cast<Vec<T, V> *>(p) = t;
}
// 16-byte store to global memory, marked as such so that the compiler knows
// it cannot alias shared memory.
template <typename T, int V>
__device__ __forceinline__ void st_vec_global(T *p, const T (&x)[V]) {
  static_assert(sizeof(T) * V == 16, "16-byte vectors only");
  if constexpr (std::is_same<T, float>::value) __stcg(reinterpret_cast<float4 *>(p), make_float4(x[0], x[1], x[2], x[3]));
  else __stcg(reinterpret_cast<double2 *>(p), make_double2(x[0], x[1]));
}
template <typename T>
__device__ __forceinline__ void st_global(T *p, T v) { __stcg(p, v); }

// Predicated forms, for stores that a few lanes make in straight-line code: as
// branches they split a row into divergent pieces that cannot be scheduled
// across.
__device__ __forceinline__ void st_global_if(float *p, float v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q st.global.cg.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v),
               "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void st_global_if(double *p, double v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q st.global.cg.f64 [%0], %1;\n\t}" ::"l"(p), "d"(v),
               "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void red_add_if(float *p, float v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q red.global.add.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v),
               "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void red_add_if(double *p, double v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q red.global.add.f64 [%0], %1;\n\t}" ::"l"(p), "d"(v),
               "r"((int)on)
               : "memory");
}
template <int V> __device__ __forceinline__ void st_vec_global_if(float *p, const float (&x)[V], bool on) {
  static_assert(V == 4, "16-byte vectors only");
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t@q st.global.cg.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(p),
      "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "r"((int)on)
      : "memory");
}
template <int V> __device__ __forceinline__ void st_vec_global_if(double *p, const double (&x)[V], bool on) {
  static_assert(V == 2, "16-byte vectors only");
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q st.global.cg.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(p),
               "d"(x[0]), "d"(x[1]), "r"((int)on)
               : "memory");
}

// ---- lane shuffles -----------------------------------------------------------
template <typename T>
__device__ __forceinline__ T shfl_up(T v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
template <typename T>
__device__ __forceinline__ T shfl_down(T v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }

// Value at element x (x in [-R, V+R)) of a row whose lane-local part is
// row[0..V): x < 0 or x >= V come from the lanes to the left/right.
template <int V, int X, typename T>
__device__ __forceinline__ T row_elem(const T (&row)[V]) {
  if constexpr (X >= 0 && X < V) {
    return row[X];
  } else if constexpr (X < 0) {
    constexpr int dl = (-X + V - 1) / V;  // lanes to the left
    constexpr int m = X + dl * V;         // element index in that lane
    return shfl_up(row[m], dl);
  } else {
    constexpr int dl = X / V;             // lanes to the right
    constexpr int m = X - dl * V;
    return shfl_down(row[m], dl);
  }
}

// Window slots: with UNR the loop over pipeline steps is unrolled W times and
// the logical window position j (0 = oldest row/plane) of phase ph lives in
// slot (ph + 1 + j) % W, so the window rotates by renaming; without UNR
// (to keep the code small) slot == j and the window shifts by moves.
template <bool UNR, int W>
__host__ __device__ constexpr int wslot(int ph, int j) { return UNR ? (ph + 1 + j) % W : j; }

// ---- arithmetic modes ---------------------------------------------------------
// Exact mode: products and sums rounded separately (never contracted).
// FMA mode: acc + c*a as one fused operation.
template <typename T> struct Arith;
template <> struct Arith<float> {
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};
template <> struct Arith<double> {
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
  static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};

// acc + c*a in the requested mode (the first term of a sum is c*a alone)
template <typename T, bool FMA>
__device__ __forceinline__ T term_next(T acc, T c, T a) {
  using A = Arith<T>;
  if constexpr (FMA) return A::fma(c, a, acc);
  else return A::add(acc, A::mul(c, a));
}

// 1/sqrt(s) for double on few FP64 operations: the hardware's approximation
// (rsqrt.approx.ftz.f64, from the upper word of s) and one third-order step of
// Householder's iteration, y (1 + e/2 + 3 e^2/8) with e = 1 - s y^2, which
// cubes its relative error. For s in [2^-100, 2^100]; 5 FP64 operations
// (two Newton steps from a float estimate: 8, two conversions and two
// comparisons, all on the FP64 pipe).
__device__ __forceinline__ double rsqrt_core(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  const double e = __fma_rn(-__dmul_rn(s, y), y, 1.0);
  return __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
}
// s in [2^-100, 2^100): one integer comparison of its upper word
__device__ __forceinline__ bool rsqrt_range(double s) {
  return (unsigned)(__double2hiint(s) - ((1023 - 100) << 20)) < (200u << 20);
}
__device__ __noinline__ inline double rsqrt_rare(double s) { return 1.0 / sqrt(s); }
// 1/sqrt(s) to about one rounding
__device__ __forceinline__ double rsqrt_near(double s) { return rsqrt_range(s) ? rsqrt_core(s) : rsqrt_rare(s); }

// The same as a root y and its residual e = 1 - s y^2, for results that use it
// more than once: 1/sqrt(s) = y (1 - e)^(-1/2). In double y is the root above
// and e is left at 0; in float y is the hardware's estimate and e, about 2^-22,
// is exact to first order (the product s y is kept whole).
__device__ __forceinline__ void rsqrt_split(double s, double &y, double &e) {
  y = rsqrt_near(s);
  e = 0.0;
}
__device__ __forceinline__ void rsqrt_split(float s, float &y, float &e) {
  y = rsqrtf(s);
  const float p = __fmul_rn(s, y);
  e = __fmaf_rn(-p, y, 1.0f);
  e = __fmaf_rn(-__fmaf_rn(s, y, -p), y, e);
  if (!(s > 0.0f && s < 3e38f)) e = 0.0f;
}
// the root itself
__device__ __forceinline__ double rsqrt_of(double y, double) { return y; }
__device__ __forceinline__ float rsqrt_of(float y, float e) { return __fmaf_rn(__fmul_rn(0.5f, y), e, y); }
// x times the root's cube, x y^3 (1 - e)^(-3/2). In float the rounded root's
// error would enter three times: the gradient of gradient2d, one step, against
// 64 bits, as a share of the error with the root in double and rounded, 0.80
// to 0.93 (with the rounded root 1.12 on smooth grids). In double the residual
// would have to leave the range test's branch as well: 8% of the step.
__device__ __forceinline__ double rsqrt_cube(double x, double y, double) {
  return __dmul_rn(__dmul_rn(x, y), __dmul_rn(y, y));
}
__device__ __forceinline__ float rsqrt_cube(float x, float y, float e) {
  const float t = __fmul_rn(__fmul_rn(x, y), __fmul_rn(y, y));
  return __fmaf_rn(t, __fmul_rn(1.5f, e), t);
}

// gradient2d.c:17-21: u + num / sqrt(s), s = eps + sum_n (u - u_n)^2 (formed by
// the caller, every difference, square and sum rounded separately in both
// modes: the update amplifies rounding where neighbours agree, so even fusing
// the squares drifts past the 1e-5 parity bound within ten steps), evaluated
// as C evaluates it in exact mode: since `1.0f / sqrt(x)` calls the double
// sqrt, the root, the quotient and the final sum in double, rounded once to T.
// FMA mode (FAST) replaces the double root and quotient, which run on the
// FP64 pipe at 1/64 of the FP32 rate.
template <typename T, bool FAST>
__device__ __forceinline__ T gradient_finish(T u, T s, T num) {
  if constexpr (FAST && std::is_same<T, float>::value) {
    // FMA mode, float, all on the FP32 pipe. q = num / sqrt(s) as an
    // unevaluated pair qh + ql: y0 = an estimate of 1/sqrt(s), then one Newton
    // correction 1/sqrt(s) ~ y0 (1 + e/2) whose residual e = 1 - s y0^2 is
    // formed exactly with FMA (s y0 = p + pe). u + qh + ql is then rounded
    // once through Knuth's TwoSum, like exact mode's single rounding of the
    // double sum (they differ only within ~2^-20 ulp of a rounding midpoint).
    const float y0 = rsqrtf(s);
    const float p = __fmul_rn(s, y0);
    const float pe = __fmaf_rn(s, y0, -p);
    float e = __fmaf_rn(-p, y0, 1.0f);
    e = __fmaf_rn(-pe, y0, e);
    const float qh = __fmul_rn(num, y0);
    const float qe = __fmaf_rn(num, y0, -qh);
    const float ql = __fmaf_rn(qh, __fmul_rn(0.5f, e), qe);
    const float t = __fadd_rn(u, qh);
    const float bv = __fsub_rn(t, u);
    const float err = __fadd_rn(__fsub_rn(u, __fsub_rn(t, bv)), __fsub_rn(qh, bv));
    return __fadd_rn(t, __fadd_rn(err, ql));
  } else if constexpr (FAST) {
    return __fma_rn(num, rsqrt_near(s), u);
  } else {
    const double q = __ddiv_rn((double)num, __dsqrt_rn((double)s));
    const double r = __dadd_rn((double)u, q);
    if constexpr (std::is_same<T, float>::value) return __double2float_rn(r);
    else return r;
  }
}

// x / d, correctly rounded, for a divisor d known in advance with y =
// RN(1/d) (y == 0 marks a divisor outside [2^-16, 2^16] (float) or
// [2^-50, 2^50] (double): IEEE division only). A reciprocal product with one
// FMA correction (Markstein's scheme) gives q1; q1 is returned only when the
// exact remainder r1 = x - q1*d shows that x/d lies strictly between the two
// rounding midpoints around q1, which makes q1 = RN(x/d). In the guarded
// range r1 is exact (the remainder of a faithful quotient is representable)
// and so are the midpoint bounds |d|*ulp/2 (power-of-two scalings); outside
// it, or when the test fails (x/d within an ulp fraction of a midpoint), the
// IEEE division is used. gbs_check_division compares this with IEEE division.
__device__ __forceinline__ float div_by(float x, float d, float y) {
  if (y != 0.0f) {
    const float q0 = __fmul_rn(x, y);
    const float r = __fmaf_rn(-q0, d, x);
    const float q1 = __fmaf_rn(r, y, q0);
    const float a = fabsf(q1);
    if (a >= 0x1p-80f && a <= 0x1p+100f) {
      const float r1 = __fmaf_rn(-q1, d, x);
      const int ab = __float_as_int(a);
      const float u = __int_as_float((ab & 0x7f800000) - (23 << 23));  // ulp(q1)
      const bool pow2 = (ab & 0x007fffff) == 0;
      // offset of x/d from q1, times |d|, signed positive away from zero
      const float om = ((d < 0.0f) != (q1 < 0.0f)) ? -r1 : r1;
      const float ad = fabsf(d);
      const float lim = (om >= 0.0f || !pow2) ? __fmul_rn(ad, __fmul_rn(u, 0.5f))
                                              : __fmul_rn(ad, __fmul_rn(u, 0.25f));
      if (fabsf(om) < lim) return q1;
    }
  }
  if (x == 0.0f && y != 0.0f) return __fmul_rn(x, y);
  return __fdiv_rn(x, d);
}
__device__ __forceinline__ double div_by(double x, double d, double y) {
  if (y != 0.0) {
    const double q0 = __dmul_rn(x, y);
    const double r = __fma_rn(-q0, d, x);
    const double q1 = __fma_rn(r, y, q0);
    const double a = fabs(q1);
    if (a >= 0x1p-900 && a <= 0x1p+900) {
      const double r1 = __fma_rn(-q1, d, x);
      const long long ab = __double_as_longlong(a);
      const double u = __longlong_as_double((ab & 0x7ff0000000000000ll) - (52ll << 52));
      const bool pow2 = (ab & 0x000fffffffffffffll) == 0;
      const double om = ((d < 0.0) != (q1 < 0.0)) ? -r1 : r1;
      const double ad = fabs(d);
      const double lim = (om >= 0.0 || !pow2) ? __dmul_rn(ad, __dmul_rn(u, 0.5))
                                              : __dmul_rn(ad, __dmul_rn(u, 0.25));
      if (fabs(om) < lim) return q1;
    }
  }
  if (x == 0.0 && y != 0.0) return __dmul_rn(x, y);
  return __ddiv_rn(x, d);
}

// x / d without the remainder test, for divisors for which the one-correction
// quotient is exact on every input: the engine whitelists such divisors only
// when the exhaustive float self-test (gbs_check_division with check=0)
// proves it for that divisor, as it does for the artifact's 118 and 159.
__device__ __forceinline__ float div_by_fast(float x, float d, float y) {
  const float q0 = __fmul_rn(x, y);
  const float r = __fmaf_rn(-q0, d, x);
  const float q1 = __fmaf_rn(r, y, q0);
  const float a = fabsf(q1);
  if (a >= 0x1p-125f && a <= 0x1p+126f) return q1;
  if (x == 0.0f) return __fmul_rn(x, y);
  return __fdiv_rn(x, d);
}

// The same for V elements at once: one test of the whole vector instead of
// four branches (with x in the tested range, the quotient is too), and one copy
// of the rest, kept out of line so that the row loops stay in the instruction
// cache.
//
// The rest is no rarity: with the artifact's own coefficients j2d5pt, j2d9pt
// and j2d9pt-gol shrink a grid by 0.42 and 0.70 a step, and after 100 to 300
// steps every cell is denormal or nearly so. A small x is scaled by 2^64, where
// the quotient Q is exact as above, and Q 2^-64 rounded; it is rounded twice,
// which goes wrong only where Q lies half-way between two results, and there
// the remainder's sign says on which side of Q the quotient is. (IEEE division
// instead, called per element: j2d5pt f32 4096^2, 1000 steps in exact mode
// 135 ms, 46 now; before, with a test per element, 113.)
__device__ __forceinline__ float div_rest(float x, float d, float y) {
  const unsigned a = __float_as_uint(x) & 0x7fffffffu;
  if (a > 0x7e800000u) return __fdiv_rn(x, d);  // above 2^126, infinite or NaN
  const bool small = a < 0x05000000u;           // below 2^-117
  const float up = small ? 0x1p+64f : 1.0f, down = small ? 0x1p-64f : 1.0f;
  const float xs = __fmul_rn(x, up);
  const float q0 = __fmul_rn(xs, y);
  const float q = __fmaf_rn(__fmaf_rn(-q0, d, xs), y, q0);
  const float rem = __fmaf_rn(-q, d, xs);       // exact, of the sign of x/d - q
  const float q1 = __fmul_rn(q, down);
  const float err = __fsub_rn(q, __fmul_rn(q1, up));  // exact: 2^-86 is half a unit of a denormal result
  float fix = 0.0f;
  if (err == 0x1p-86f && rem > 0.0f) fix = 0x1p-149f;
  if (err == -0x1p-86f && rem < 0.0f) fix = -0x1p-149f;
  return x == 0.0f ? __fmul_rn(x, y) : fix != 0.0f ? __fadd_rn(q1, fix) : q1;  // (-0 + 0 is +0)
}
template <int V> __device__ __noinline__ Vec<float, V> div_rest_vec(Vec<float, V> x, float d, float y) {
#pragma unroll
  for (int e = 0; e < V; ++e) x.v[e] = div_rest(x.v[e], d, y);
  return x;
}
template <int V>
__device__ __forceinline__ void div_by_fast(float (&x)[V], float d, float y) {
  // |x| in [2^-117, 2^126] for every element: |x/d| in [2^-125, 2^126] for
  // 1 <= d <= 256 (the proven divisors are 118 and 159)
  unsigned lo = 0xffffffffu, hi = 0u;
  Vec<float, V> q;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const unsigned a = __float_as_uint(x[e]) & 0x7fffffffu;
    lo = min(lo, a);
    hi = max(hi, a);
    const float q0 = __fmul_rn(x[e], y);
    const float r = __fmaf_rn(-q0, d, x[e]);
    q.v[e] = __fmaf_rn(r, y, q0);
  }
  if (lo < 0x05000000u || hi > 0x7e800000u) {  // 2^-117, 2^126
#pragma unroll
    for (int e = 0; e < V; ++e) q.v[e] = x[e];
    q = div_rest_vec<V>(q, d, y);
  }
#pragma unroll
  for (int e = 0; e < V; ++e) x[e] = q.v[e];
}

// RN(1/d) for div_by, or 0 when d is outside the range div_by's test covers.
template <typename T> inline T div_reciprocal(double d) {
  const double lo = sizeof(T) == 4 ? 0x1p-16 : 0x1p-50, hi = sizeof(T) == 4 ? 0x1p+16 : 0x1p+50;
  const double ad = d < 0 ? -d : d;
  if (!(ad >= lo && ad <= hi)) return (T)0;
  volatile T one = (T)1;
  return one / (T)d;
}

}  // namespace gbs
