// Velocity sets, population storage and the per-node pieces of one LBM step
// (pull streaming with the reference's face rules, moments, forcing, BGK),
// shared by every kernel of the library.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/funlbm_b200.h"

namespace lbm {

// Bounds-checked build (-DLBM_BOUNDS_CHECK): kernels verify their index
// invariants before each access (node inside the lattice, population index
// inside the pitched buffer, pull source inside the lattice, field index
// inside the field); a violation is counted in this translation unit's
// g_lbm_oob and the access is skipped or clamped to a valid index
// (lbm_debug_bounds_faults reads the counts).  Without the flag lbm_in is
// always true and the checks compile away.
#ifdef LBM_BOUNDS_CHECK
static __device__ unsigned long long g_lbm_oob;
__device__ __forceinline__ bool lbm_in(bool ok) {
  if (!ok) atomicAdd(&g_lbm_oob, 1ull);
  return ok;
}
#else
__device__ __forceinline__ constexpr bool lbm_in(bool) { return true; }
#endif

// Chained launches (programmatic dependent launch).  The kernels of one
// lattice step -- interpolation, spreading, the rigid update and the fused
// step, observations, statistics and the reference call sequence -- are
// launched with programmatic stream serialization (launch_chained): the GPU
// may schedule such a kernel while the kernel before it in the stream is still
// running.  chain_wait() is therefore the first statement of each of them,
// executed by every thread before any memory access: it returns once the
// previous kernel has completed and its writes are visible, so every access
// happens in plain stream order.  A kernel that only reads what an earlier
// step wrote waits too: the kernel after it is ordered after this one alone.
// chain_release() right after it lets the next kernel be scheduled while
// this one runs (a kernel is only scheduled once every block of the one
// before it has started, so a waiting kernel never holds resources the
// running one still needs).  Launched without the attribute, both are no-ops.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_enter() {
  chain_wait();
  chain_release();
}

// Compile-time loop: calls fn(std::integral_constant<int, I>) for I < N, so
// every population index is a constant and f[Q] stays in registers.
template <typename F, int... I>
__host__ __device__ __forceinline__ void static_for_impl(F &&fn, std::integer_sequence<int, I...>) {
  (fn(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__host__ __device__ __forceinline__ void static_for(F &&fn) {
  static_for_impl(fn, std::make_integer_sequence<int, N>{});
}

// ---------------------------------------------------------------------------
// Velocity sets.  Direction order is the reference's (flow/d3/d3q13.py:7-21,
// d3q15.py:7-23, d3q19.py:8-28, d3q27.py:8-36): the opposite-direction table
// and the population layout depend on it.  Weights by speed class
// (d3q13.py:23-39, d3q15.py:25-43, d3q19.py:30-54, d3q27.py:38-71).
// Tables live inside constexpr functions so that fully unrolled loops fold
// every lookup to an immediate.
// ---------------------------------------------------------------------------
template <int Q>
struct VSet;

#define LBM_VSET_BODY(QN, EX, EY, EZ, W0, W1, W2, W3)                                   \
  static constexpr int kQ = QN;                                                           \
  __host__ __device__ static constexpr int ex(int i) {                                    \
    constexpr int t[QN] = EX;                                                             \
    return t[i];                                                                          \
  }                                                                                       \
  __host__ __device__ static constexpr int ey(int i) {                                    \
    constexpr int t[QN] = EY;                                                             \
    return t[i];                                                                          \
  }                                                                                       \
  __host__ __device__ static constexpr int ez(int i) {                                    \
    constexpr int t[QN] = EZ;                                                             \
    return t[i];                                                                          \
  }                                                                                       \
  __host__ __device__ static constexpr int speed2(int i) {                                \
    return ex(i) * ex(i) + ey(i) * ey(i) + ez(i) * ez(i);                                \
  }                                                                                       \
  __host__ __device__ static constexpr double wd(int i) {                                 \
    return speed2(i) == 0 ? (W0) : speed2(i) == 1 ? (W1) : speed2(i) == 2 ? (W2) : (W3); \
  }                                                                                       \
  __host__ __device__ static constexpr float w(int i) { return (float)wd(i); }           \
  template <typename R>                                                                   \
  __host__ __device__ static constexpr R wr(int i) { return (R)wd(i); }                   \
  __host__ __device__ static constexpr int rev(int i) {                                   \
    int r = 0;                                                                            \
    for (int j = 0; j < QN; ++j)                                                          \
      if (ex(j) == -ex(i) && ey(j) == -ey(i) && ez(j) == -ez(i)) r = j;                   \
    return r;                                                                             \
  }

#define LBM_ARR(...) {__VA_ARGS__}

template <>
struct VSet<13> {
  LBM_VSET_BODY(13,
                LBM_ARR(0, 1, 1, 1, 1, 0, 0, -1, -1, -1, -1, 0, 0),
                LBM_ARR(0, 1, -1, 0, 0, 1, 1, -1, 1, 0, 0, -1, -1),
                LBM_ARR(0, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1),
                1.0 / 2, 0.0, 1.0 / 24, 0.0)
};
template <>
struct VSet<15> {
  LBM_VSET_BODY(15,
                LBM_ARR(0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1),
                LBM_ARR(0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1),
                LBM_ARR(0, 0, 0, 0, 0, 1, -1, 1, 1, 1, 1, -1, -1, -1, -1),
                2.0 / 9, 1.0 / 9, 0.0, 1.0 / 72)
};
template <>
struct VSet<19> {
  LBM_VSET_BODY(19,
                LBM_ARR(0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1),
                LBM_ARR(0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 1, -1, 1, -1, 0, 0, 0, 0),
                LBM_ARR(0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1),
                1.0 / 3, 1.0 / 18, 1.0 / 36, 0.0)
};
template <>
struct VSet<27> {
  LBM_VSET_BODY(27,
                LBM_ARR(0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, 1, 1, 1,
                        -1, -1, -1, -1),
                LBM_ARR(0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1,
                        1, 1, -1, -1),
                LBM_ARR(0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1, 1, -1, 1, -1,
                        1, -1, 1, -1),
                8.0 / 27, 2.0 / 27, 1.0 / 54, 1.0 / 216)
};

#undef LBM_ARR
#undef LBM_VSET_BODY

// ---------------------------------------------------------------------------
// Population storage.  FP32 stores f; the shifted 16-bit forms store f - w_i
// (the deviation from the rest-state weight carries all the information and
// keeps the 16-bit mantissa busy), collided in float32.
// ---------------------------------------------------------------------------
template <int S>
struct Storage;

// The fused step works on the stored quantity itself (its "working value"):
// the deviation d = f - w_i for the shifted forms (kDev: FP32 and both 16-bit
// storages), whose moments and collision are restated for d (dev_moments /
// collide_dev), so no weight is added on load or subtracted on store; f
// itself for FP64.  work / put / work2 / put2 move working values; load /
// store always give f.
//
// FP32 stores the deviation too.  At the low Mach numbers of the reference's
// cases a population f ~ w_i ~ 0.05 carries its velocity part (w rho e.u /
// cs^2 ~ 1e-6) in its last ten bits, and a body or IBM force adds ~17 units
// in the last place per step: stored as f, those increments round with the
// same bias every step of a nearly steady flow, and the float32 run drifts
// from the float64 one (measured on B200: twice the reference's own float32
// drift on the 33 x 33 x 65 Poiseuille channel after 2000 steps, ten times
// in the sedimenting sphere's velocity after 5000).  Stored as d ~ 1e-6 the
// same 32 bits resolve the signal to ~1e-7 of itself, at the same bytes per
// node.
template <>
struct Storage<LBM_STORAGE_FP32> {
  using T = float;
  using R = float;   // arithmetic type of the kernels
  static constexpr int kBits = 32;
  static constexpr bool kDev = true;
  static constexpr int kShift = 0;   // working value = d * 2^kShift
  __device__ __forceinline__ static T raw(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static float cvt(T v) { return v; }
  __device__ __forceinline__ static float work(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static void put(T *p, float v) { *p = v; }
  __device__ __forceinline__ static float load(const T *p, float w) { return w + __ldg(p); }
  __device__ __forceinline__ static void store(T *p, float v, float w) { *p = v - w; }
};
// FP16 holds the deviation scaled by 2^12: float16's normal range starts at
// 6.1e-5, and at the velocities of the reference's particle cases (|u| ~
// 1e-6) a deviation w rho e.u / cs^2 ~ 1e-7 would fall among its subnormals
// (spacing 6e-8: a 90 % velocity error measured over 3000 steps of the
// 32-ellipsoid case).  Scaled, deviations from 1.5e-8 up to 16 keep the full
// 11-bit significand; populations stay in [0, 1], so |d| < 1.  The scale is
// a power of two: the scaling itself is exact.  The fused step keeps the
// scaled value as its working value (kShift): the moments unscale their sums
// and the collision and forcing carry the scale in their weight constants,
// so no element is multiplied on load or store.
constexpr float kFp16Scale = 4096.f;
constexpr float kFp16Unscale = 1.f / 4096.f;

template <>
struct Storage<LBM_STORAGE_FP16S> {
  using T = __half;
  using R = float;
  static constexpr int kBits = 16;
  static constexpr bool kDev = true;
  static constexpr int kShift = 12;
  __device__ __forceinline__ static T raw(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static float cvt(T v) { return __half2float(v); }
  __device__ __forceinline__ static float work(const T *p) { return __half2float(__ldg(p)); }
  __device__ __forceinline__ static void put(T *p, float v) { *p = __float2half_rn(v); }
  __device__ __forceinline__ static float load(const T *p, float w) {
    return w + __half2float(__ldg(p)) * kFp16Unscale;
  }
  __device__ __forceinline__ static void store(T *p, float v, float w) {
    *p = __float2half_rn((v - w) * kFp16Scale);
  }
};
template <>
struct Storage<LBM_STORAGE_BF16S> {
  using T = __nv_bfloat16;
  using R = float;
  static constexpr int kBits = 16;
  static constexpr bool kDev = true;
  static constexpr int kShift = 0;
  __device__ __forceinline__ static T raw(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static float cvt(T v) { return __bfloat162float(v); }
  __device__ __forceinline__ static float work(const T *p) { return __bfloat162float(__ldg(p)); }
  __device__ __forceinline__ static void put(T *p, float v) { *p = __float2bfloat16_rn(v); }
  __device__ __forceinline__ static float load(const T *p, float w) {
    return w + __bfloat162float(__ldg(p));
  }
  __device__ __forceinline__ static void store(T *p, float v, float w) {
    *p = __float2bfloat16_rn(v - w);
  }
};

// FP64: populations, moments, forcing and collision in double -- the
// comparison run against which the float32 and 16-bit storages are measured.
template <>
struct Storage<LBM_STORAGE_FP64> {
  using T = double;
  using R = double;
  static constexpr int kBits = 64;
  static constexpr bool kDev = false;
  static constexpr int kShift = 0;
  __device__ __forceinline__ static T raw(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static double cvt(T v) { return v; }
  __device__ __forceinline__ static double work(const T *p) { return __ldg(p); }
  __device__ __forceinline__ static void put(T *p, double v) { *p = v; }
  __device__ __forceinline__ static double load(const T *p, double) { return __ldg(p); }
  __device__ __forceinline__ static void store(T *p, double v, double) { *p = v; }
};

// Raw 16 bits of one stored element.
__device__ __forceinline__ unsigned short bits16(__half h) { return __half_as_ushort(h); }
__device__ __forceinline__ unsigned short bits16(__nv_bfloat16 h) { return __bfloat16_as_ushort(h); }

// Two consecutive stored elements <-> two working values (low element first).
template <int S>
__device__ __forceinline__ float2 work2(unsigned word);
template <>
__device__ __forceinline__ float2 work2<LBM_STORAGE_FP16S>(unsigned word) {
  __half2 h;
  memcpy(&h, &word, 4);
  return __half22float2(h);
}
template <>
__device__ __forceinline__ float2 work2<LBM_STORAGE_BF16S>(unsigned word) {
  return make_float2(__uint_as_float(word << 16), __uint_as_float(word & 0xffff0000u));
}
template <int S>
__device__ __forceinline__ unsigned put2(float a, float b);
template <>
__device__ __forceinline__ unsigned put2<LBM_STORAGE_FP16S>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  unsigned word;
  memcpy(&word, &h, 4);
  return word;
}
template <>
__device__ __forceinline__ unsigned put2<LBM_STORAGE_BF16S>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  unsigned word;
  memcpy(&word, &h, 4);
  return word;
}

// Aligned vector loads / stores of WORDS 32-bit words (4, 8 or 16 bytes).
template <int WORDS>
struct Words {
  unsigned w[WORDS];
};
template <int WORDS>
__device__ __forceinline__ Words<WORDS> ld_words(const void *p);
template <>
__device__ __forceinline__ Words<1> ld_words<1>(const void *p) {
  return Words<1>{{__ldg(static_cast<const unsigned *>(p))}};
}
template <>
__device__ __forceinline__ Words<2> ld_words<2>(const void *p) {
  const uint2 v = __ldg(static_cast<const uint2 *>(p));
  return Words<2>{{v.x, v.y}};
}
template <>
__device__ __forceinline__ Words<4> ld_words<4>(const void *p) {
  const uint4 v = __ldg(static_cast<const uint4 *>(p));
  return Words<4>{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ void st_words(void *p, const Words<1> &v) {
  *static_cast<unsigned *>(p) = v.w[0];
}
__device__ __forceinline__ void st_words(void *p, const Words<2> &v) {
  *static_cast<uint2 *>(p) = make_uint2(v.w[0], v.w[1]);
}
__device__ __forceinline__ void st_words(void *p, const Words<4> &v) {
  *static_cast<uint4 *>(p) = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
}

// ---------------------------------------------------------------------------
// Lattice constants passed by value to every kernel.
// ---------------------------------------------------------------------------
struct Geom {
  int nx, ny, nz;
  long long n;      // nodes
  long long nyz;    // ny * nz
  int pz;           // row pitch of the population buffers (>= nz)
  long long np;     // population plane: nx * ny * pz elements
  long long nyzp;   // ny * pz
  int face[LBM_NFACES];
  unsigned moving;  // bit fc: face fc is WALL_WITH_SPEED
  float uw[LBM_NFACES][3];
  long long plane_off[LBM_NFACES];  // offsets of the face-density planes
  float tau, inv_tau, cs2, inv_cs2, inv_cs4, force_c;  // force_c = 1 - 1/(2 tau)
  float re_mu;
  const double *neq_profile;
  // the same constants in double, for FP64 storage: tau as given, cs^2 =
  // double(sqrt(1/3))^2, wall velocities widened
  double inv_tau_d, inv_cs2_d, inv_cs4_d, force_c_d;
  double uw_d[LBM_NFACES][3];
};

// Two float32 values in one register pair (two neighbouring nodes of a row):
// sm_100's packed add / multiply / fused multiply-add round each half as the
// scalar instruction does, so a node has the same values in either form, at
// half the issue slots.  One exception: a product of -0 is +0 here (operator*).
struct F2 {
  float2 v;
  F2() = default;
  __device__ __forceinline__ explicit F2(float s) : v(make_float2(s, s)) {}
  __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
  __device__ __forceinline__ explicit F2(float2 p) : v(p) {}
};
__device__ __forceinline__ unsigned long long f2_bits(F2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.v.x), "f"(a.v.y));
  return r;
}
__device__ __forceinline__ F2 f2_of(unsigned long long r) {
  F2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.v.x), "=f"(a.v.y) : "l"(r));
  return a;
}
__device__ __forceinline__ F2 fma_rn(F2 a, F2 b, F2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
  return f2_of(r);
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
}
// a b as a b + 0: the assembler contracts a packed multiply followed by a
// packed add to one fused operation, also where both are written as rounded
// (add_force's ux fx + uy fy differed from the scalar code in one pair of 2000),
// but not this form.  The same value; only a product of -0 becomes +0.
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return fma_rn(a, b, F2(0.f)); }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-a.v.x, -a.v.y); }
// a - b as a + (-1) b: one rounding, as the subtraction
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return fma_rn(b, F2(-1.f), a); }
__device__ __forceinline__ F2 &operator+=(F2 &a, F2 b) { return a = a + b; }
__device__ __forceinline__ F2 &operator-=(F2 &a, F2 b) { return a = a - b; }
__device__ __forceinline__ float recip(float x) { return 1.f / x; }
__device__ __forceinline__ F2 recip(F2 x) { return F2(1.f / x.v.x, 1.f / x.v.y); }
// u, zero where the node lies on a boundary plane
__device__ __forceinline__ float off_face(bool face, float u) { return face ? 0.f : u; }
struct Face2 {
  bool a, b;
};
__device__ __forceinline__ F2 off_face(Face2 face, F2 u) {
  return F2(face.a ? 0.f : u.v.x, face.b ? 0.f : u.v.y);
}
// Lattice constants in the arithmetic type R of a kernel.
template <typename R>
struct Cst;
template <>
struct Cst<float> {
  __device__ __forceinline__ static float inv_tau(const Geom &g) { return g.inv_tau; }
  __device__ __forceinline__ static float inv_cs2(const Geom &g) { return g.inv_cs2; }
  __device__ __forceinline__ static float inv_cs4(const Geom &g) { return g.inv_cs4; }
  __device__ __forceinline__ static float force_c(const Geom &g) { return g.force_c; }
  __device__ __forceinline__ static float uw(const Geom &g, int fc, int k) { return g.uw[fc][k]; }
};
template <>
struct Cst<double> {
  __device__ __forceinline__ static double inv_tau(const Geom &g) { return g.inv_tau_d; }
  __device__ __forceinline__ static double inv_cs2(const Geom &g) { return g.inv_cs2_d; }
  __device__ __forceinline__ static double inv_cs4(const Geom &g) { return g.inv_cs4_d; }
  __device__ __forceinline__ static double force_c(const Geom &g) { return g.force_c_d; }
  __device__ __forceinline__ static double uw(const Geom &g, int fc, int k) { return g.uw_d[fc][k]; }
};

template <>
struct Cst<F2> {
  __device__ __forceinline__ static F2 inv_cs2(const Geom &g) { return F2(g.inv_cs2); }
  __device__ __forceinline__ static F2 inv_cs4(const Geom &g) { return F2(g.inv_cs4); }
  __device__ __forceinline__ static F2 force_c(const Geom &g) { return F2(g.force_c); }
};
// type of one node's values in the arithmetic type R
template <typename R>
struct OneOf {
  using type = R;
};
template <>
struct OneOf<F2> {
  using type = float;
};

// face-plane index of node (x, y, z) on face `fc`
__device__ __forceinline__ long long plane_index(const Geom &g, int fc, int x, int y, int z) {
  switch (fc >> 1) {
    case 0: return g.plane_off[fc] + (long long)y * g.nz + z;
    case 1: return g.plane_off[fc] + (long long)x * g.nz + z;
    default: return g.plane_off[fc] + (long long)x * g.ny + y;
  }
}

__device__ __forceinline__ bool on_any_face(const Geom &g, int x, int y, int z) {
  return x == 0 || x == g.nx - 1 || y == 0 || y == g.ny - 1 || z == 0 || z == g.nz - 1;
}

// ---------------------------------------------------------------------------
// Pull streaming with the reference's rules (flow/d3/base.py:161-323).
// For target node t and direction i the reference rolls every population
// periodically and then overrides, face by face in the order input, output,
// back, forward, bottom, top, the directions entering through that face; the
// last matching override wins.  Rolling wraps only where some face override
// applies, so the source is:
//   no face applies      -> (t - e_i, i)
//   PERIODICAL face      -> t with that axis moved to the opposite plane (no
//                           transverse shift), direction i
//   WALL face            -> (t, rev(i))                 half-way bounce-back
//   WALL_WITH_SPEED face -> (t, rev(i)) - 2 rho_t w_i (e_i . uw) / cs^2
// NON_EQUILIBRIUM x faces are handled by the caller (they need moments).
// ---------------------------------------------------------------------------
constexpr int kMaxQ = 27;

// Which of a row's faces its nodes lie on (a row: fixed x and y).
struct RowFaces {
  bool xl, xh, yl, yh;
  __device__ __forceinline__ RowFaces(const Geom &g, int x, int y)
      : xl(x == 0), xh(x == g.nx - 1), yl(y == 0), yh(y == g.ny - 1) {}
  // row class: 3 (x low, inside, high) x 3 (y)
  __device__ __forceinline__ int cls() const { return (xl ? 0 : xh ? 6 : 3) + (yl ? 0 : yh ? 2 : 1); }
  __device__ __forceinline__ bool any() const { return xl || xh || yl || yh; }
};
constexpr int kRowClasses = 9, kInnerRow = 4;

// Whether a direction with components EX, EY enters a row through one of its
// x / y faces.  Its source is then the opposite plane or the node itself, both
// without a z shift.
template <int EX, int EY>
__device__ __forceinline__ bool enters(const RowFaces &r) {
  bool e = false;
  if constexpr (EX > 0) e = e || r.xl;
  if constexpr (EX < 0) e = e || r.xh;
  if constexpr (EY > 0) e = e || r.yl;
  if constexpr (EY < 0) e = e || r.yh;
  return e;
}

// Per-direction plane pointers of one step, computed on the host
// (fill_step_planes), so that every population address in the kernels is
// one 32 x 32 -> 64-bit multiply-add of the node's population index
// (x ny + y) pz + z onto a parameter:
//   src[c][i] + idx  pull source of a row of class c at the node's z: inside,
//                  row (x - ex, y - ey) of plane i, to be read at z - ez;
//                  where direction i enters through an x / y face (the last
//                  of them in the order x, y), the opposite plane of i
//                  (PERIODICAL) or plane rev(i) of the row itself, read at z;
//   zlo[i] + idx   (ez > 0) source of a node at z = 0 under the bottom face
//                  rule, whatever its row: PERIODICAL -> (i, x, y, nz - 1),
//                  else (rev i, x, y, 0);
//   zhi[i] + idx   (ez < 0) source of a node at z = nz - 1 under the top face
//                  rule: PERIODICAL -> (i, x, y, 0), else (rev i, x, y, nz - 1);
//   dst[i] + idx   plane i of fb.
// A face row thus runs the same instructions as an inner one.  (One branch
// per direction and face instead: each load waited for the one before it, and
// 1.6 % of the rows of a periodic 256^3 lattice took 13 % of the 16-bit
// step's time.)
struct StepPlanes {
  const void *src[kRowClasses][kMaxQ];
  const void *zlo[kMaxQ];
  const void *zhi[kMaxQ];
  void *dst[kMaxQ];
  const void *lo, *hi;   // the population buffer (bounds-checked build)
};

// Densities of the previous step at a node of moving walls, one per axis.
template <typename R>
struct WallRho {
  R v[3];
  __device__ __forceinline__ explicit WallRho(R rho) : v{rho, rho, rho} {}
  __device__ __forceinline__ WallRho(const Geom &g, const R *__restrict__ face_rho,
                                     const RowFaces &r, int x, int y, int z) {
    auto at = [&](int fc, bool on) {
      return on && ((g.moving >> fc) & 1u) ? face_rho[plane_index(g, fc, x, y, z)] : R(0);
    };
    v[0] = at(r.xl ? 0 : 1, r.xl || r.xh);
    v[1] = at(r.yl ? 2 : 3, r.yl || r.yh);
    v[2] = at(z == 0 ? 4 : 5, z == 0 || z == g.nz - 1);
  }
};

// WALL_WITH_SPEED correction of direction I at a node of that face, applied
// after the bounce-back pull: the amount to subtract from f (WORK units: times
// 2^SH), 0 where the governing face (the last in the order x, y, z) is not a
// moving wall.
template <int Q, int I, int SH, typename R>
__device__ __forceinline__ R moving_wall(const Geom &g, const WallRho<R> &rho, const RowFaces &r,
                                         int z) {
  using V = VSet<Q>;
  constexpr int ex = V::ex(I), ey = V::ey(I), ez = V::ez(I);
  int fc = -1;
  if constexpr (ex > 0) fc = r.xl ? 0 : fc;
  if constexpr (ex < 0) fc = r.xh ? 1 : fc;
  if constexpr (ey > 0) fc = r.yl ? 2 : fc;
  if constexpr (ey < 0) fc = r.yh ? 3 : fc;
  if constexpr (ez > 0) fc = z == 0 ? 4 : fc;
  if constexpr (ez < 0) fc = z == g.nz - 1 ? 5 : fc;
  if (fc < 0 || !((g.moving >> fc) & 1u)) return R(0);
  const R rho_t = fc < 2 ? rho.v[0] : fc < 4 ? rho.v[1] : rho.v[2];
  const R eu = (R)ex * Cst<R>::uw(g, fc, 0) + (R)ey * Cst<R>::uw(g, fc, 1) +
               (R)ez * Cst<R>::uw(g, fc, 2);
  return R(2) * (rho_t * V::template wr<R>(I)) * eu * Cst<R>::inv_cs2(g) * R(1 << SH);
}

// Whether the node lies on a moving wall.
__device__ __forceinline__ bool on_moving_wall(const Geom &g, const RowFaces &r, int z) {
  return g.moving != 0 &&
         (((r.xl ? 1u : 0u) | (r.xh ? 2u : 0u) | (r.yl ? 4u : 0u) | (r.yh ? 8u : 0u) |
           (z == 0 ? 16u : 0u) | (z == g.nz - 1 ? 32u : 0u)) & g.moving) != 0;
}

// Pull of one node with the reference's face rules but for the moving walls'
// correction; no branch between the loads, so all Q of them issue together.
// WORK: working values (d for the shifted storages) as the fused step uses
// them; otherwise f.
template <int Q, int S, bool WORK>
__device__ __forceinline__ void pull_sources(const StepPlanes &p, const Geom &g, const RowFaces &r,
                                             unsigned idx, int z, typename Storage<S>::R f[Q]) {
  using St = Storage<S>;
  using T = typename St::T;
  using V = VSet<Q>;
  const bool bottom = z == 0, top = z == g.nz - 1;
  auto pull = [&](auto ic, const T *ps, bool shifted) {
    constexpr int i = decltype(ic)::value;
    constexpr int ez = V::ez(i);
    if constexpr (ez != 0) ps = shifted ? ps - ez : ps;
    if constexpr (ez > 0) ps = bottom ? static_cast<const T *>(p.zlo[i]) + idx : ps;
    if constexpr (ez < 0) ps = top ? static_cast<const T *>(p.zhi[i]) + idx : ps;
    if (!lbm_in(ps >= static_cast<const T *>(p.lo) && ps < static_cast<const T *>(p.hi)))
      ps = static_cast<const T *>(p.lo);
    if constexpr (WORK)
      f[i] = St::work(ps);
    else
      f[i] = St::load(ps, V::template wr<typename St::R>(i));   // (w_rev(i) = w_i)
  };
  // Two copies of the loads, so that the plane pointers of an inner row are
  // parameters at fixed places: with one copy indexed by the row's class,
  // lattices of odd rows ran 2 to 10 % slower (129^3 D3Q15: 52 -> 58 us).
  if (!r.any()) {
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      pull(ic, static_cast<const T *>(p.src[kInnerRow][i]) + idx, true);
    });
  } else {
    const void *const *src = p.src[r.cls()];
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      pull(ic, static_cast<const T *>(src[i]) + idx, !enters<V::ex(i), V::ey(i)>(r));
    });
  }
}

// Pull of one node with all of the reference's face rules.
template <int Q, int S, bool WORK>
__device__ __forceinline__ void pull_node(const StepPlanes &p, const Geom &g,
                                          const typename Storage<S>::R *__restrict__ face_rho,
                                          unsigned idx, int x, int y, int z,
                                          typename Storage<S>::R f[Q]) {
  const RowFaces r(g, x, y);
  pull_sources<Q, S, WORK>(p, g, r, idx, z, f);
  if (on_moving_wall(g, r, z)) {
    constexpr int kSh = WORK ? Storage<S>::kShift : 0;
    const WallRho<typename Storage<S>::R> rho(g, face_rho, r, x, y, z);
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      if constexpr (i != 0) f[i] -= moving_wall<Q, i, kSh>(g, rho, r, z);
    });
  }
}

// Rolled value (periodic wrap on every axis, no face rule): what the
// reference's f holds at a node before the face overrides run.  Used by the
// NON_EQUILIBRIUM faces, which read plane 1 / plane X-2 right after the roll.
template <int Q>
__device__ __forceinline__ float pull_rolled(const float *__restrict__ fa, const Geom &g, int i,
                                             int x, int y, int z) {
  using V = VSet<Q>;
  int sx = x - V::ex(i), sy = y - V::ey(i), sz = z - V::ez(i);
  sx = sx < 0 ? sx + g.nx : (sx >= g.nx ? sx - g.nx : sx);
  sy = sy < 0 ? sy + g.ny : (sy >= g.ny ? sy - g.ny : sy);
  sz = sz < 0 ? sz + g.nz : (sz >= g.nz ? sz - g.nz : sz);
  const long long src = ((long long)sx * g.ny + sy) * g.nz + sz;   // dense arrays only
  return fa[(long long)i * g.n + src];
}

// ---------------------------------------------------------------------------
// Per-node arithmetic.  Directions come in opposite pairs (i, rev(i)); the
// moments, the forcing term and the equilibrium share their work across the
// pair.  The library is built with -fmad=false and every fused multiply-add
// below is explicit (__fmaf_rn), so each kernel that calls these functions
// produces the same values whatever its launch shape (a zero's sign: see F2).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

#define LBM_FMA(a, b, c) ::lbm::fma_rn((a), (b), (c))

// Moments (flow/d3/base.py:116-133): rho = sum f, u = (sum f e + F/2) / rho,
// u := 0 on all six boundary planes whatever their condition.
template <int Q, typename R>
__device__ __forceinline__ void moments(const R f[Q], R fx, R fy, R fz, bool face, R &rho, R &ux,
                                        R &uy, R &uz) {
  using V = VSet<Q>;
  R r = f[0], jx = R(0), jy = R(0), jz = R(0);
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int j = V::rev(i);
    if constexpr (i != 0 && i < j) {
      const R s = f[i] + f[j];
      const R d = f[i] - f[j];
      r += s;
      if constexpr (V::ex(i) > 0) jx += d;
      if constexpr (V::ex(i) < 0) jx -= d;
      if constexpr (V::ey(i) > 0) jy += d;
      if constexpr (V::ey(i) < 0) jy -= d;
      if constexpr (V::ez(i) > 0) jz += d;
      if constexpr (V::ez(i) < 0) jz -= d;
    }
  });
  rho = r;
  const R inv = R(1) / r;
  ux = face ? R(0) : LBM_FMA(R(0.5), fx, jx) * inv;
  uy = face ? R(0) : LBM_FMA(R(0.5), fy, jy) * inv;
  uz = face ? R(0) : LBM_FMA(R(0.5), fz, jz) * inv;
}

// e_i . v with e_i in {-1, 0, 1}^3, folded at compile time: the components in
// the order x, y, z.  Where the first sign is negative the partial sum is
// kept negated until a positive component turns it (v_y - v_x for
// -v_x + v_y): the same bits without a negation.
template <int Q, int I, typename R>
__device__ __forceinline__ R edot(R vx, R vy, R vz) {
  using V = VSet<Q>;
  R r = R(0);
  bool first = true, neg = false;
  auto acc = [&](int e, R v) {
    if (e == 0) return;
    if (first) {
      r = v;
      neg = e < 0;
      first = false;
    } else if (neg) {
      r = e > 0 ? v - r : r + v;
      neg = e < 0;
    } else {
      r = e > 0 ? r + v : r - v;
    }
  };
  acc(V::ex(I), vx);
  acc(V::ey(I), vy);
  acc(V::ez(I), vz);
  return neg ? -r : r;
}

// Forcing term of FlowD3.cul_equ2 (flow/d3/base.py:103-114):
//   f_i += (1 - 1/(2 tau)) w_i [ (e_i - u)/cs^2 + (u o e_i) o e_i / cs^4 ] . F
// (component-wise u_k e_ik^2, the reference's form).  For the pair (i, j),
// e_j = -e_i: the e.F part flips sign, the rest is shared.
template <int Q, int SH = 0, typename R>
__device__ __forceinline__ void add_force(R f[Q], const Geom &g, R ux, R uy, R uz, R fx, R fy,
                                          R fz) {
  using V = VSet<Q>;
  using One = typename OneOf<R>::type;
  const R inv_cs2 = Cst<R>::inv_cs2(g), force_c = Cst<R>::force_c(g);
  const R uF = LBM_FMA(ux, fx, LBM_FMA(uy, fy, uz * fz));
  const R ax = ux * fx, ay = uy * fy, az = uz * fz;
  const R base = -uF * inv_cs2;
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int j = V::rev(i);
    constexpr One cw = V::template wr<One>(i) * One(1 << SH);     // working units
    if constexpr (i == 0) {
      f[0] = LBM_FMA(force_c * R(cw), base, f[0]);
    } else if constexpr (i < j) {
      R t2 = R(0);
      if constexpr (V::ex(i) != 0) t2 += ax;
      if constexpr (V::ey(i) != 0) t2 += ay;
      if constexpr (V::ez(i) != 0) t2 += az;
      const R shared = LBM_FMA(t2, Cst<R>::inv_cs4(g), base);
      const R eF = edot<Q, i>(fx, fy, fz) * inv_cs2;
      const R c = force_c * R(cw);
      f[i] = LBM_FMA(c, shared + eF, f[i]);
      f[j] = LBM_FMA(c, shared - eF, f[j]);
    }
  });
}

// BGK collision of FlowD3.cul_equ (flow/d3/base.py:150-159):
//   feq_i = (1 + t + t^2/2 - |u|^2/(2 cs^2)) rho w_i,  t = e_i.u / cs^2
//   f_i  <- f_i - (f_i - feq_i) / tau = f_i (1 - 1/tau) + feq_i / tau
// With a = rho w (1 - |u|^2/(2cs^2) + t^2/2) and b = rho w t, the pair gets
// feq_i = a + b, feq_rev(i) = a - b.
template <int Q>
__device__ __forceinline__ float feq_of(const Geom &g, int i, float rho, float ux, float uy,
                                        float uz, float u2) {
  using V = VSet<Q>;
  const float t = ((float)V::ex(i) * ux + (float)V::ey(i) * uy + (float)V::ez(i) * uz) * g.inv_cs2;
  return LBM_FMA(0.5f * t, t, (1.f - u2) + t) * (rho * V::w(i));
}

template <int Q, typename R>
__device__ __forceinline__ void collide(R f[Q], const Geom &g, R rho, R ux, R uy, R uz) {
  using V = VSet<Q>;
  const R inv_cs2 = Cst<R>::inv_cs2(g), inv_tau = Cst<R>::inv_tau(g);
  const R u2 = LBM_FMA(ux, ux, LBM_FMA(uy, uy, uz * uz)) * (R(0.5) * inv_cs2);
  const R om = inv_tau, keep = R(1) - inv_tau;
  const R orho = om * rho;
  const R one_u2 = R(1) - u2;
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int j = V::rev(i);
    constexpr R w = V::template wr<R>(i);
    if constexpr (i == 0) {
      f[0] = LBM_FMA(f[0], keep, (orho * w) * one_u2);
    } else if constexpr (i < j) {
      const R t = edot<Q, i>(ux, uy, uz) * inv_cs2;
      const R ow = orho * w;
      const R a = ow * LBM_FMA(R(0.5) * t, t, one_u2);
      const R b = ow * t;
      f[i] = LBM_FMA(f[i], keep, a + b);
      f[j] = LBM_FMA(f[j], keep, a - b);
    }
  });
}

// Deviation form, for the shifted storages.  With f_i = w_i + d_i,
// sum w_i = 1 and sum w_i e_i = 0:
//   rho = 1 + sum d_i,   rho u = sum d_i e_i + F/2,
// and the BGK update of FlowD3.cul_equ (flow/d3/base.py:150-159) becomes
//   d_i <- d_i (1 - 1/tau) + (feq_i - w_i) / tau,
//   feq_i - w_i = w_i [ (rho - 1) + rho (t + t^2/2 - |u|^2/(2 cs^2)) ],
// so the pair (i, rev(i)) gets A +- B with
//   A = w (drho - rho |u|^2/(2cs^2)) / tau + (w rho t / (2 tau)) t,  B = w rho t / tau.
// The forcing term (add_force) is additive and applies to d unchanged.
// R: float (one node) or F2 (two); FACE: bool or Face2.  FORCED = false: the
// force is zero and left out.
template <int Q, int SH, bool FORCED, typename R, typename FACE>
__device__ __forceinline__ void dev_moments(const R d[Q], R fx, R fy, R fz, FACE face, R &rho,
                                            R &drho, R &ux, R &uy, R &uz) {
  using V = VSet<Q>;
  R r = d[0], jx = R(0.f), jy = R(0.f), jz = R(0.f);
  bool jx0 = true, jy0 = true, jz0 = true;   // (folded: 0 + t is t)
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int j = V::rev(i);
    if constexpr (i != 0 && i < j) {
      const R s = d[i] + d[j];
      const R t = d[i] - d[j];
      r += s;
      if constexpr (V::ex(i) > 0) jx = jx0 ? t : jx + t;
      if constexpr (V::ex(i) < 0) jx -= t;
      if constexpr (V::ex(i) != 0) jx0 = false;
      if constexpr (V::ey(i) > 0) jy = jy0 ? t : jy + t;
      if constexpr (V::ey(i) < 0) jy -= t;
      if constexpr (V::ey(i) != 0) jy0 = false;
      if constexpr (V::ez(i) > 0) jz = jz0 ? t : jz + t;
      if constexpr (V::ez(i) < 0) jz -= t;
      if constexpr (V::ez(i) != 0) jz0 = false;
    }
  });
  constexpr float kUnscale = 1.f / (float)(1 << SH);      // d = working value / 2^SH
  if constexpr (SH != 0) {
    drho = r * R(kUnscale);
    jx = jx * R(kUnscale);
    jy = jy * R(kUnscale);
    jz = jz * R(kUnscale);
  } else {
    drho = r;
  }
  rho = R(1.f) + drho;
  const R inv = recip(rho);
  if constexpr (FORCED) {
    jx = LBM_FMA(R(0.5f), fx, jx);
    jy = LBM_FMA(R(0.5f), fy, jy);
    jz = LBM_FMA(R(0.5f), fz, jz);
  }
  ux = off_face(face, jx * inv);
  uy = off_face(face, jy * inv);
  uz = off_face(face, jz * inv);
}

template <int Q, int SH, typename R>
__device__ __forceinline__ void collide_dev(R d[Q], const Geom &g, R rho, R drho, R ux, R uy,
                                            R uz) {
  using V = VSet<Q>;
  const R nu2 = LBM_FMA(ux, ux, LBM_FMA(uy, uy, uz * uz)) * R(-0.5f * g.inv_cs2);   // -|u|^2/(2cs^2)
  const R ic = R(g.inv_cs2), om = R(g.inv_tau), keep = R(1.f - g.inv_tau);
  const R vx = ux * ic, vy = uy * ic, vz = uz * ic;
  const R orho = om * rho;
  const R c = om * LBM_FMA(rho, nu2, drho);
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int j = V::rev(i);
    constexpr float w = V::w(i) * (float)(1 << SH);         // working units
    if constexpr (i == 0) {
      d[0] = LBM_FMA(d[0], keep, R(w) * c);
    } else if constexpr (i < j) {
      const R t = edot<Q, i>(vx, vy, vz);
      const R a = LBM_FMA((orho * R(0.5f * w)) * t, t, R(w) * c);
      const R b = (orho * R(w)) * t;
      d[i] = LBM_FMA(d[i], keep, a + b);
      d[j] = LBM_FMA(d[j], keep, a - b);
    }
  });
}

template <typename R>
__device__ __forceinline__ void flag_bad(unsigned *status, R rho, R ux, R uy, R uz) {
  if (status == nullptr) return;
  if (!(rho > R(0)) || !(rho < R(3.0e38))) atomicOr(status, LBM_STATUS_RHO_BAD);
  if (!(fabs(ux) + fabs(uy) + fabs(uz) < R(3.0e38))) atomicOr(status, LBM_STATUS_U_BAD);
}

}  // namespace lbm
