// Fused-step kernels (scalar, vectorised, TMA row-staged) and their launch
// logic.  Included by lbm_flow.cu (declarations only) and by
// lbm_step_inst.cu, which the build compiles once per (velocity set,
// storage) with -DLBM_Q / -DLBM_S.
#pragma once
#include <algorithm>

#include "lbm_api.cuh"
#include "lbm_tma.cuh"

namespace lbm {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// Fused step
// ---------------------------------------------------------------------------
struct StepArgs {
  Geom g;
  NodeDecomp dec;    // dense node index -> (x, y, z)
  NodeDecomp pdec;   // population index (x ny + y) pz + z -> (x, y, z)
  const void *fa;
  void *fb;
  float go[3], gn[3];
  int uniform;       // go or gn is not zero
  // fields, face densities and observation buffers hold the storage's
  // arithmetic type (float64 for LBM_STORAGE_FP64, float32 otherwise)
  const void *fol_old, *fol_new;
  const uint8_t *ch_old, *ch_new;
  const void *face_rho_in;
  void *face_rho_out;
  void *obs_f, *obs_rho, *obs_u;
  int obs_pairs;     // observation buffers take aligned stores of two nodes
  unsigned *status;
  StepPlanes p;
};

template <int Q, typename R>
__device__ __forceinline__ void write_face_rho(const Geom &g, R *out, int x, int y, int z, R rho) {
  if (x == 0) out[plane_index(g, 0, x, y, z)] = rho;
  if (x == g.nx - 1) out[plane_index(g, 1, x, y, z)] = rho;
  if (y == 0) out[plane_index(g, 2, x, y, z)] = rho;
  if (y == g.ny - 1) out[plane_index(g, 3, x, y, z)] = rho;
  if (z == 0) out[plane_index(g, 4, x, y, z)] = rho;
  if (z == g.nz - 1) out[plane_index(g, 5, x, y, z)] = rho;
}

template <typename R>
__device__ __forceinline__ unsigned bad_bits(R rho, R ux, R uy, R uz) {
  unsigned b = 0;
  if (!(rho > R(0)) || !(rho < R(3.0e38))) b |= LBM_STATUS_RHO_BAD;
  if (!(fabs(ux) + fabs(uy) + fabs(uz) < R(3.0e38))) b |= LBM_STATUS_U_BAD;
  return b;
}

// Whether the previous / this step's force field applies in the 32-node
// chunk of node idx.
struct ChunkForce {
  bool old_here, new_here;
};

template <bool FORCE>
__device__ __forceinline__ ChunkForce chunk_force(const StepArgs &a, unsigned idx) {
  ChunkForce c{false, false};
  if constexpr (FORCE) {
    c.old_here = a.fol_old != nullptr && (a.ch_old == nullptr || a.ch_old[idx >> 5]);
    c.new_here = a.fol_new != nullptr && (a.ch_new == nullptr || a.ch_new[idx >> 5]);
  }
  return c;
}

// Force at the node: the uniform part plus the field where the node's chunk
// carries it.
template <typename R>
__device__ __forceinline__ void node_force(const float uniform[3], const void *field, bool here,
                                           unsigned idx, R F[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) F[k] = uniform[k];
  if (here) {
    const R *fol = static_cast<const R *>(field);
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k] += fol[3ull * idx + k];
  }
}

// Everything after the pull for one node: the first moments with the previous
// force, cul_equ2 with the new one, the second moments, status bits
// (accumulated in `bad`) and face densities.  DEV: f holds deviations d = f - w
// (shifted storage), handled by dev_moments / collide_dev.  finish_node_m hands
// the node's end-of-step moments to the caller; f is left at the end-of-step
// populations.
// Where neither step has a force (no uniform part, neither field in the
// node's chunk) cul_equ2 adds nothing and the second moment pass repeats the
// first, so both are skipped -- the same rule in every kernel, and a node of a
// flagged chunk without force of its own gets the same values either way while
// its velocity is finite (else the status bits stop the run).  The
// new force is read only there: kept from the start of the node together with
// the old one it cost 20 to 28 registers per thread of the pair kernels.
template <int Q, bool FORCE, bool DEV, int SH, typename R>
__device__ __forceinline__ void finish_node_m(const StepArgs &a, R f[Q], unsigned idx, int x,
                                              int y, int z, bool face, ChunkForce cf,
                                              unsigned &bad, R &rho, R &drho, R &ux, R &uy, R &uz) {
  R F[3] = {R(0), R(0), R(0)};
  if constexpr (FORCE) node_force<R>(a.go, a.fol_old, cf.old_here, idx, F);
  if constexpr (DEV) {
    dev_moments<Q, SH, FORCE>(f, F[0], F[1], F[2], face, rho, drho, ux, uy, uz);
  } else {
    drho = R(0);
    moments<Q>(f, F[0], F[1], F[2], face, rho, ux, uy, uz);
  }
  if (FORCE && (a.uniform || cf.old_here || cf.new_here)) {
    node_force<R>(a.gn, a.fol_new, cf.new_here, idx, F);
    add_force<Q, SH>(f, a.g, ux, uy, uz, F[0], F[1], F[2]);
    if constexpr (DEV)
      dev_moments<Q, SH, true>(f, F[0], F[1], F[2], face, rho, drho, ux, uy, uz);
    else
      moments<Q>(f, F[0], F[1], F[2], face, rho, ux, uy, uz);
  }
  bad |= bad_bits(rho, ux, uy, uz);
  if (face && a.face_rho_out != nullptr)
    write_face_rho<Q>(a.g, static_cast<R *>(a.face_rho_out), x, y, z, rho);
}

// A node's end-of-step state to the observation buffers.
template <int Q, bool DEV, int SH, typename R>
__device__ __forceinline__ void observe_node(const StepArgs &a, const R f[Q], unsigned idx, R rho,
                                             R ux, R uy, R uz) {
  using V = VSet<Q>;
  if (a.obs_f != nullptr) {
    R *of = static_cast<R *>(a.obs_f);
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      of[(long long)i * a.g.n + idx] =
          DEV ? f[i] * (R(1) / R(1 << SH)) + V::template wr<R>(i) : f[i];
    });
  }
  if (a.obs_rho != nullptr) static_cast<R *>(a.obs_rho)[idx] = rho;
  if (a.obs_u != nullptr) {
    R *ou = static_cast<R *>(a.obs_u);
    ou[3ull * idx] = ux;
    ou[3ull * idx + 1] = uy;
    ou[3ull * idx + 2] = uz;
  }
}

// A thread's one or (two) two values into an array that the threads of a warp
// fill one after the other, in aligned stores of two: where the thread's place
// is odd, its last value leaves with its right neighbour's first.  lanes: the
// warp's threads that take part.
__device__ __forceinline__ void store_run(float *dst, float a, float b, bool two, unsigned lanes) {
  const unsigned lane = threadIdx.x & 31u;
  const bool prev = lane > 0u && ((lanes >> (lane - 1u)) & 1u);
  const bool next = lane < 31u && ((lanes >> (lane + 1u)) & 1u);
  const float na = __shfl_down_sync(lanes, a, 1);
  const bool odd = ((uintptr_t)dst & 4u) != 0;
  if (odd && !prev) dst[0] = a;
  if (odd && !two) return;
  const bool own = !odd && two;
  const float v0 = odd ? b : a, v1 = own ? b : na;
  dst += odd ? 1 : 0;
  if (own || next)
    *reinterpret_cast<float2 *>(dst) = make_float2(v0, v1);
  else
    dst[0] = v0;
}
// The same for three values a node.
__device__ __forceinline__ void store_run3(float *dst, F2 vx, F2 vy, F2 vz, bool two,
                                           unsigned lanes) {
  const unsigned lane = threadIdx.x & 31u;
  const bool prev = lane > 0u && ((lanes >> (lane - 1u)) & 1u);
  const bool next = lane < 31u && ((lanes >> (lane + 1u)) & 1u);
  const float nx = __shfl_down_sync(lanes, vx.v.x, 1);
  const bool odd = ((uintptr_t)dst & 4u) != 0;
  if (odd && !prev) dst[0] = vx.v.x;
  float2 *d = reinterpret_cast<float2 *>(dst + (odd ? 1 : 0));
  d[0] = odd ? make_float2(vy.v.x, vz.v.x) : make_float2(vx.v.x, vy.v.x);
  if (two) d[1] = odd ? make_float2(vx.v.y, vy.v.y) : make_float2(vz.v.x, vx.v.y);
  if (odd && !two) return;
  const float v0 = two ? (odd ? vz.v.y : vy.v.y) : vz.v.x;
  const float v1 = two && !odd ? vz.v.y : nx;
  if (two) ++d;
  if ((two && !odd) || next)
    d[1] = make_float2(v0, v1);
  else
    *reinterpret_cast<float *>(d + 1) = v0;
}

// The same for nodes idx and (two) idx + 1.  Rows of odd length put half of the
// pairs at odd places.  Stored element by element, each store instruction then
// touched all sectors for half of their bytes: a step of 257^3 D3Q19 fp32 with f,
// rho and u took 1201 us, with store_run 723 (dense rows, one node per thread: 850).
template <int Q, int SH>
__device__ __forceinline__ void observe_pair(const StepArgs &a, const F2 f[Q], unsigned idx,
                                             bool two, unsigned lanes, F2 rho, F2 ux, F2 uy,
                                             F2 uz) {
  float *of = static_cast<float *>(a.obs_f), *orho = static_cast<float *>(a.obs_rho),
        *ou = static_cast<float *>(a.obs_u);
  auto value = [&](int i) {
    return f[i] * F2(1.f / (float)(1 << SH)) + F2(VSet<Q>::w(i));
  };
  if (a.obs_pairs) {   // (every pair whole and at an even place)
    if (of != nullptr)
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        *reinterpret_cast<float2 *>(of + (long long)i * a.g.n + idx) = value(i).v;
      });
    if (orho != nullptr) *reinterpret_cast<float2 *>(orho + idx) = rho.v;
    if (ou != nullptr) {
      float2 *d = reinterpret_cast<float2 *>(ou + 3ull * idx);
      d[0] = make_float2(ux.v.x, uy.v.x);
      d[1] = make_float2(uz.v.x, ux.v.y);
      d[2] = make_float2(uy.v.y, uz.v.y);
    }
    return;
  }
  if (of != nullptr)
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      const F2 v = value(i);
      store_run(of + (long long)i * a.g.n + idx, v.v.x, v.v.y, two, lanes);
    });
  if (orho != nullptr) store_run(orho + idx, rho.v.x, rho.v.y, two, lanes);
  if (ou != nullptr) store_run3(ou + 3ull * idx, ux, uy, uz, two, lanes);
}

// What a launch does with its nodes: advance them (collide and store), write
// their end-of-step state, or both in one read of the populations (kernels of
// their own, so the step carries none of that code).
enum class Op { kStep, kObserve, kBoth };
__host__ __device__ constexpr bool advances(Op op) { return op != Op::kObserve; }
__host__ __device__ constexpr bool observes(Op op) { return op != Op::kStep; }

template <int Q, bool FORCE, bool DEV, int SH, Op OP, typename R>
__device__ __forceinline__ void finish_node(const StepArgs &a, R f[Q], unsigned idx, int x,
                                            int y, int z, bool face, ChunkForce cf,
                                            unsigned &bad) {
  R rho, drho, ux, uy, uz;
  finish_node_m<Q, FORCE, DEV, SH>(a, f, idx, x, y, z, face, cf, bad, rho, drho, ux, uy, uz);
  if constexpr (observes(OP)) observe_node<Q, DEV, SH>(a, f, idx, rho, ux, uy, uz);
  if constexpr (advances(OP)) {
    if constexpr (DEV)
      collide_dev<Q, SH>(f, a.g, rho, drho, ux, uy, uz);
    else
      collide<Q>(f, a.g, rho, ux, uy, uz);
  }
}

// finish_node for two neighbouring nodes (z, z + 1) of a row at once, in
// packed arithmetic: the same operations in the same order, so the same values
// (a zero may differ in sign, see F2).
// two: the second node exists (the last of a pitched row's odd length has no
// partner: its lane holds padding and reports nothing).
template <int Q, bool FORCE, int SH, Op OP>
__device__ __forceinline__ void finish_pair(const StepArgs &a, F2 f[Q], unsigned idx, int x, int y,
                                            int z, bool row_face, bool two, unsigned lanes,
                                            ChunkForce c0, ChunkForce c1, unsigned &bad) {
  Face2 face;
  face.a = row_face || z == 0 || z == a.g.nz - 1;
  face.b = row_face || z + 1 == a.g.nz - 1;
  F2 rho, drho, ux, uy, uz;
  F2 F[3] = {F2(0.f), F2(0.f), F2(0.f)};
  auto force = [&](const float uniform[3], const void *field, bool here0, bool here1) {
    float p[3], q[3];
    node_force<float>(uniform, field, here0, idx, p);
    node_force<float>(uniform, field, here1 && two, idx + 1, q);
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k] = F2(p[k], q[k]);
  };
  if constexpr (FORCE) force(a.go, a.fol_old, c0.old_here, c1.old_here);
  dev_moments<Q, SH, FORCE>(f, F[0], F[1], F[2], face, rho, drho, ux, uy, uz);
  if constexpr (FORCE) {
    if (a.uniform || c0.old_here || c0.new_here || c1.old_here || c1.new_here) {
      force(a.gn, a.fol_new, c0.new_here, c1.new_here);
      add_force<Q, SH>(f, a.g, ux, uy, uz, F[0], F[1], F[2]);
      dev_moments<Q, SH, true>(f, F[0], F[1], F[2], face, rho, drho, ux, uy, uz);
    }
  }
  bad |= bad_bits(rho.v.x, ux.v.x, uy.v.x, uz.v.x);
  if (two) bad |= bad_bits(rho.v.y, ux.v.y, uy.v.y, uz.v.y);
  if (a.face_rho_out != nullptr) {
    float *fr = static_cast<float *>(a.face_rho_out);
    if (face.a) write_face_rho<Q>(a.g, fr, x, y, z, rho.v.x);
    if (face.b && two) write_face_rho<Q>(a.g, fr, x, y, z + 1, rho.v.y);
  }
  if constexpr (observes(OP)) observe_pair<Q, SH>(a, f, idx, two, lanes, rho, ux, uy, uz);
  if constexpr (advances(OP)) collide_dev<Q, SH>(f, a.g, rho, drho, ux, uy, uz);
}

__device__ __forceinline__ void report_bad(unsigned *status, unsigned bad) {
  if (bad != 0 && status != nullptr) atomicOr(status, bad);
}

// Row padding of a pitched lattice (population index p, p + 1, ... up to the
// row's pitch) is written by the kernel that writes the row's last node,
// with any value: it is never a pull source and never observed, but a
// 32-byte sector that a step writes only in part makes L2 fetch the rest
// from DRAM before it can write the sector back (measured on B200 at 257^3
// in FP32: +2 % DRAM reads and 16 % longer steps while the padding was left
// unwritten).
template <int Q, int S>
__device__ __forceinline__ void put_row_padding(const StepArgs &a, unsigned p, int count,
                                                const typename Storage<S>::R f[Q]) {
  using St = Storage<S>;
  using T = typename St::T;
#pragma unroll 1
  for (int j = 0; j < count; ++j) {
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      St::put(static_cast<T *>(a.p.dst[i]) + p + j, f[i]);
    });
  }
}

// A vector of padding only (a pitched row's last vector, past its nodes):
// zero words, stored for the same reason.
template <int Q, int S, int NZ>
__device__ __forceinline__ void put_padding_vector(const StepArgs &a, unsigned pidx0) {
  using St = Storage<S>;
  using T = typename St::T;
  constexpr int kWords = NZ * St::kBits / 32;
  Words<kWords> zero;
#pragma unroll
  for (int k = 0; k < kWords; ++k) zero.w[k] = 0u;
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    st_words(static_cast<T *>(a.p.dst[i]) + pidx0, zero);
  });
}

// One node per thread, nodes in memory order so that each warp owns one
// 32-node chunk.  FORCE adds cul_equ2
// and the second moment pass; without it both are exact no-ops (the
// reference adds zeros and recomputes identical moments), so they are
// skipped.
template <int Q, int S, bool FORCE, Op OP = Op::kStep>
__device__ __forceinline__ void step_scalar_body(const StepArgs &a, const unsigned idx) {
  using St = Storage<S>;
  using T = typename St::T;
  if (idx >= (unsigned)a.g.n) return;
  int x, y, z;
  a.dec(idx, x, y, z);
  const unsigned pidx = (unsigned)(x * a.g.ny + y) * (unsigned)a.g.pz + (unsigned)z;
  if (!lbm_in(x < a.g.nx && y < a.g.ny && z < a.g.nz && pidx < (unsigned)a.g.np)) return;
  using R = typename St::R;
  const R *face_rho = static_cast<const R *>(a.face_rho_in);
  R f[Q];
  pull_node<Q, S, true>(a.p, a.g, face_rho, pidx, x, y, z, f);
  const ChunkForce cf = chunk_force<FORCE>(a, idx);   // (after the loads, see step_pairs_at)
  unsigned bad = 0;
  finish_node<Q, FORCE, St::kDev, St::kShift, OP>(a, f, idx, x, y, z, on_any_face(a.g, x, y, z), cf,
                                                  bad);
  report_bad(a.status, bad);
  if constexpr (advances(OP)) {
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      St::put(static_cast<T *>(a.p.dst[i]) + pidx, f[i]);
    });
    if (z == a.g.nz - 1 && a.g.pz > a.g.nz)
      put_row_padding<Q, S>(a, pidx + 1, a.g.pz - a.g.nz, f);
  }
}

// Register cap of the one-node kernel (resident blocks per SM asked of the
// compiler, 0 = none).  The one-node kernel runs dense rows of odd length and
// rows of two nodes, and observes odd rows (go_observe); it is latency-bound:
// more resident warps pay until the compiler spills.  Measured on B200 on
// dense rows, us per step without / with the cap: D3Q19 161 x 65 x 65 fp32 19.0 / 18.5, fp16s 15.1 / 13.3; 177 x 113
// x 97 fp16s 41.3 / 36.3; D3Q15 129^3 fp32 52.1 / 50.1, fp16s 48.3 / 44.8;
// D3Q27 257 x 129 x 129 fp32 162 with 4 blocks, 180 with 5; fp16s 120, 124
// with 5, and 110 uncapped in blocks of 128 threads.
template <int Q, int S>
constexpr int scalar_min_blocks() {
  constexpr int bits = Storage<S>::kBits;
  if (bits == 64) return 0;
  if (bits == 16) return Q == 27 ? 0 : 5;
  return Q == 27 ? 4 : 5;
}
// Threads per block of the one-node kernel.
template <int Q, int S>
__host__ __device__ constexpr int scalar_threads() {
  return Q == 27 && Storage<S>::kBits == 16 ? 128 : kThreads;
}

template <int Q, int S, bool FORCE>
__global__ void __launch_bounds__((scalar_threads<Q, S>()), (scalar_min_blocks<Q, S>()))
    k_step(const __grid_constant__ StepArgs a) {
  chain_enter();
  step_scalar_body<Q, S, FORCE>(a, blockIdx.x * scalar_threads<Q, S>() + threadIdx.x);
}

// The end-of-step state of every node to the observation buffers, and with
// Op::kBoth the step itself: one node per thread (rows that take no pairs, FP64).
template <int Q, int S, bool FORCE, Op OP>
__global__ void __launch_bounds__((scalar_threads<Q, S>()), (scalar_min_blocks<Q, S>()))
    k_observe(const __grid_constant__ StepArgs a) {
  chain_enter();
  step_scalar_body<Q, S, FORCE, OP>(a, blockIdx.x * scalar_threads<Q, S>() + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Step statistics: min / sum / max of f, u and rho at the end of the step the
// populations `fa` stream into (FlowD3.to_json, flow/base.py:183-206, as
// LBMBase._log_step_info logs it, lbm/base.py:105-144), in one read of the
// populations and nothing written but 9 numbers.  Grid-stride, one node per
// thread per iteration; per-block reduction, then one atomic per quantity
// and block into `out`: min / max as order-preserving 64-bit keys of the
// doubles, sums as doubles (k_stats_finish turns them into min, mean, max).
// ---------------------------------------------------------------------------
constexpr int kStatsThreads = 256;

__device__ __forceinline__ unsigned long long ordered_bits(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double from_ordered_bits(unsigned long long o) {
  const unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
  return __longlong_as_double((long long)b);
}

// Per-thread accumulators: extremes in the arithmetic type (exact), sums in
// double.
template <typename R>
struct StatAcc {
  R mn[3], mx[3];
  double sm[3];
};

// sum of v[0..N), added to `acc`.  The conversion of every value to double was
// what bounded the kernel (a quarter of the float64 rate): here the even and
// the odd values are summed in packed float32 with the error of each addition
// (Knuth's two-sum, exact whichever term is the larger), and four values are
// converted per node.
template <int N>
__device__ __forceinline__ void add_all(const float v[N], double &acc) {
  F2 s(v[0], v[1]), e(0.f);
#pragma unroll
  for (int i = 2; i < N; i += 2) {
    const F2 x(v[i], i + 1 < N ? v[i + 1 < N ? i + 1 : i] : 0.f);
    const F2 t = s + x;
    const F2 w = t - s;                // the part of x that t holds
    e += (s - (t - w)) + (x - w);
    s = t;
  }
  if (fabsf(s.v.x) + fabsf(s.v.y) < 3.0e38f) {
    acc += (double)s.v.x;
    acc += (double)s.v.y;
    acc += (double)(e.v.x + e.v.y);
  } else {                             // (sums without an error term)
#pragma unroll
    for (int i = 0; i < N; ++i) acc += (double)v[i];
  }
}
template <int N>
__device__ __forceinline__ void add_all(const double v[N], double &acc) {
#pragma unroll
  for (int i = 0; i < N; ++i) acc += v[i];
}

// Resident blocks per SM of k_stats, also its grid (5 blocks of D3Q19 spilled
// and took 3 % longer than 4).
template <int Q, int S>
constexpr int stats_blocks() {
  return Storage<S>::kBits == 64 ? 2 : Q == 27 ? 3 : 4;
}

// Bound by the read of the populations (D3Q19 fp32 193 x 161 x 129: 305 MB, 47
// us at the copy peak); float32 extremes and the sums above took the registers
// from 80 to 64 (4 resident blocks instead of 3) and the three launches of
// lbm_flow_stats from 99 to 70 us (65 with sums that are exact only while the rest
// population is the largest).
template <int Q, int S, bool FORCE>
__global__ void __launch_bounds__(kStatsThreads, (stats_blocks<Q, S>()))
    k_stats(const __grid_constant__ StepArgs a, unsigned long long *out) {
  chain_enter();
  using St = Storage<S>;
  using R = typename St::R;
  using V = VSet<Q>;
  __shared__ StatAcc<R> sh[kStatsThreads / 32];
  StatAcc<R> acc;
  for (int k = 0; k < 3; ++k) {
    acc.mn[k] = R(INFINITY);
    acc.mx[k] = -R(INFINITY);
    acc.sm[k] = 0.0;
  }
  const R *face_rho = static_cast<const R *>(a.face_rho_in);
  unsigned bad = 0;
  for (unsigned idx = blockIdx.x * kStatsThreads + threadIdx.x; idx < (unsigned)a.g.n;
       idx += gridDim.x * kStatsThreads) {
    int x, y, z;
    const ChunkForce cf = chunk_force<FORCE>(a, idx);
    a.dec(idx, x, y, z);
    const unsigned pidx = (unsigned)(x * a.g.ny + y) * (unsigned)a.g.pz + (unsigned)z;
    if (!lbm_in(x < a.g.nx && y < a.g.ny && z < a.g.nz && pidx < (unsigned)a.g.np)) continue;
    R f[Q];
    pull_node<Q, S, true>(a.p, a.g, face_rho, pidx, x, y, z, f);
    R rho, drho, ux, uy, uz;
    finish_node_m<Q, FORCE, St::kDev, St::kShift>(a, f, idx, x, y, z, on_any_face(a.g, x, y, z), cf,
                                                  bad, rho, drho, ux, uy, uz);
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      f[i] = St::kDev ? f[i] * (R(1) / R(1 << St::kShift)) + V::template wr<R>(i) : f[i];
      acc.mn[0] = fmin(acc.mn[0], f[i]);
      acc.mx[0] = fmax(acc.mx[0], f[i]);
    });
    add_all<Q>(f, acc.sm[0]);
    acc.mn[1] = fmin(acc.mn[1], fmin(ux, fmin(uy, uz)));
    acc.mx[1] = fmax(acc.mx[1], fmax(ux, fmax(uy, uz)));
    acc.sm[1] += (double)ux;
    acc.sm[1] += (double)uy;
    acc.sm[1] += (double)uz;
    acc.mn[2] = fmin(acc.mn[2], rho);
    acc.mx[2] = fmax(acc.mx[2], rho);
    acc.sm[2] += (double)rho;
  }
  report_bad(a.status, bad);
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      acc.mn[k] = fmin(acc.mn[k], __shfl_xor_sync(0xffffffffu, acc.mn[k], o));
      acc.mx[k] = fmax(acc.mx[k], __shfl_xor_sync(0xffffffffu, acc.mx[k], o));
      acc.sm[k] += __shfl_xor_sync(0xffffffffu, acc.sm[k], o);
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = acc;
  __syncthreads();
  if (threadIdx.x < 3) {   // thread k: quantity k
    const int k = threadIdx.x;
    R mn = sh[0].mn[k], mx = sh[0].mx[k];
    double sm = sh[0].sm[k];
    for (int w = 1; w < kStatsThreads / 32; ++w) {
      mn = fmin(mn, sh[w].mn[k]);
      mx = fmax(mx, sh[w].mx[k]);
      sm += sh[w].sm[k];
    }
    atomicMin(out + 3 * k, ordered_bits((double)mn));
    atomicAdd(reinterpret_cast<double *>(out + 3 * k + 1), sm);
    atomicMax(out + 3 * k + 2, ordered_bits((double)mx));
  }
}

// slots of the 9 statistics: min / max keys of +inf / -inf, sums 0 (a
// template, instantiated beside each k_stats, so that every translation unit
// that includes this header may carry it)
template <int Q>
__global__ void k_stats_init(unsigned long long *out) {
  chain_enter();
  const int k = threadIdx.x;
  if (k >= 9) return;
  const int c = k % 3;
  out[k] = c == 0 ? ordered_bits(INFINITY)
                  : c == 2 ? ordered_bits(-INFINITY) : (unsigned long long)__double_as_longlong(0.0);
}

// in place: keys -> min / max, sums -> means over n*q, 3n and n values
template <int Q>
__global__ void k_stats_finish(unsigned long long *out, double n) {
  chain_enter();
  const int k = threadIdx.x;
  if (k >= 9) return;
  const int c = k % 3;
  double v;
  if (c == 1) {
    const double count = k == 1 ? n * Q : k == 4 ? 3.0 * n : n;
    v = __longlong_as_double((long long)out[k]) / count;
  } else {
    v = from_ordered_bits(out[k]);
  }
  reinterpret_cast<double *>(out)[k] = v;
}

// ---------------------------------------------------------------------------
// Vectorised fused step: thread = NZ consecutive nodes of one z-row (pz a
// multiple of NZ), populations moved as NZ-element vectors (16 / 8 / 4 byte
// loads and stores), float32 arithmetic packed two nodes to an instruction.
// What bounds it: HBM for FP32; for 16-bit storage, where a node moves half
// the bytes, the instructions and the registers per node.  Packing the
// arithmetic, two branches in place of 2 x 10 address selects and face rows
// that run the inner rows' code took the 16-bit D3Q19 step from ~610 to ~440
// instructions per node pair.  Measured at 256^3 (one B200, us per step before
// -> now, 128 threads): D3Q13 bf16s 199 -> 144, D3Q15 bf16s 220 -> 176, D3Q19
// bf16s 266 -> 205, fp16s 236 -> 226, D3Q27 fp16s 372 -> 334, bf16s 460 -> 338.
// Staging rows in shared memory instead (persistent blocks, TMA or cp.async
// rings, up to three stages) measured slower for every set: 266-350 us for
// D3Q19 fp16s.
// ---------------------------------------------------------------------------
// One direction's stored elements of a thread's NZ nodes, still packed: the
// vector at the thread's own z and the element beyond it that the shifted
// directions pull.
template <int S, int NZ>
struct Pulled {
  Words<(NZ * Storage<S>::kBits + 31) / 32> w;
  typename Storage<S>::T extra;
};

// Element k of a pulled vector as a working value.
template <int S, int NZ>
__device__ __forceinline__ float elem(const Pulled<S, NZ> &p, int k) {
  if constexpr (Storage<S>::kBits == 32) {
    return __uint_as_float(p.w.w[k]);
  } else {
    const float2 v = work2<S>(p.w.w[k >> 1]);
    return (k & 1) ? v.y : v.x;
  }
}

// NZ consecutive nodes of one z-row per thread (NZ even), worked through as
// NZ / 2 pairs in packed arithmetic; idx of node 0 is pidx0 in the population
// buffers.  The vectors stay packed in registers and a pair is unpacked right
// before it is finished; each direction leaves in one vector store.
//   One aligned vector load per direction gives NZ - |ez| of the NZ values,
// one scalar load the remaining one: from the neighbouring vector, or at
// z = 0 / z = nz - 1 from the bottom / top face rule.  For 16-bit elements two
// branches per thread, each over all its directions, instead of an address
// select per direction: 59 instead of 97 instructions per pair (D3Q19), and
// the loads of both sides still issue together.  A direction that enters
// through an x / y face takes its vector unshifted.
//   ALIGNED = false (16-bit, NZ = 2): the pair starts at any index (dense rows
// of odd length) and moves element by element.
//   PITCH: rows may carry padding (pz > nz); the last vector of a row may be
// partial or hold padding only.  Padding is stored with the vector (see
// put_row_padding); its lanes report and observe nothing.
template <int Q, int S, bool FORCE, int NZ, bool PITCH, Op OP = Op::kStep, bool ALIGNED = true>
__device__ __forceinline__ void step_pairs_at(const StepArgs &a, const unsigned pidx0) {
  using St = Storage<S>;
  using T = typename St::T;
  using V = VSet<Q>;
  static_assert(St::kBits <= 32 && NZ % 2 == 0, "pairs of float32 arithmetic");
  static_assert(ALIGNED || (NZ == 2 && St::kBits == 16), "unaligned pairs are single 16-bit pairs");
  constexpr int kWords = NZ * St::kBits / 32;
  int x = 0, y = 0, z0 = 0;
  unsigned lanes = 0;   // observing: the warp's threads that hold nodes (store_run)
  if constexpr (observes(OP)) {
    static_assert(NZ == 2, "a thread observes one pair");
    const bool inside = pidx0 < (unsigned)a.g.np;
    if (inside) a.pdec(pidx0, x, y, z0);
    lanes = __ballot_sync(0xffffffffu, inside && z0 < a.g.nz);
    if (!inside) return;
  } else {
    if (pidx0 >= (unsigned)a.g.np) return;
    a.pdec(pidx0, x, y, z0);
  }
  if constexpr (PITCH) {
    if (z0 >= a.g.nz) {                      // row padding only
      if constexpr (advances(OP)) put_padding_vector<Q, S, NZ>(a, pidx0);
      return;
    }
  }
  const unsigned idx0 = (unsigned)(x * a.g.ny + y) * (unsigned)a.g.nz + (unsigned)z0;
  const int nv = PITCH && a.g.nz - z0 < NZ ? a.g.nz - z0 : NZ;    // nodes inside the row
  const bool in_bounds = lbm_in(x < a.g.nx && y < a.g.ny && pidx0 + NZ <= (unsigned)a.g.np &&
                                idx0 + nv <= (unsigned)a.g.n);
  if constexpr (observes(OP)) lanes = __ballot_sync(lanes, in_bounds);
  if (!in_bounds) return;
  const bool bottom = z0 == 0, top = z0 + NZ >= a.g.nz;
  const RowFaces rf(a.g, x, y);
  const void *const *src = a.p.src[rf.cls()];
  unsigned bad = 0;
  Pulled<S, NZ> in[Q];
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    const T *ps = static_cast<const T *>(src[i]) + pidx0;
    if constexpr (ALIGNED)
      in[i].w = ld_words<kWords>(ps);
    else
      in[i].w.w[0] = (unsigned)bits16(St::raw(ps)) | ((unsigned)bits16(St::raw(ps + 1)) << 16);
  });
  if constexpr (St::kBits == 32) {
    // (select: 0.5 % faster than the branches at 512^3, D3Q19)
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      const T *ps = static_cast<const T *>(src[i]) + pidx0;
      if constexpr (V::ez(i) > 0)
        in[i].extra = St::raw(bottom ? static_cast<const T *>(a.p.zlo[i]) + pidx0 : ps - 1);
      if constexpr (V::ez(i) < 0)
        in[i].extra =
            St::raw(top ? static_cast<const T *>(a.p.zhi[i]) + (pidx0 + (nv - 1)) : ps + NZ);
    });
  } else {
    if (bottom) {
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (V::ez(i) > 0)
          in[i].extra = St::raw(static_cast<const T *>(a.p.zlo[i]) + pidx0);
      });
    } else {
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (V::ez(i) > 0)
          in[i].extra = St::raw(static_cast<const T *>(src[i]) + pidx0 - 1);
      });
    }
    if (top) {
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (V::ez(i) < 0)
          in[i].extra = St::raw(static_cast<const T *>(a.p.zhi[i]) + (pidx0 + (nv - 1)));
      });
    } else {
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (V::ez(i) < 0)
          in[i].extra = St::raw(static_cast<const T *>(src[i]) + pidx0 + NZ);
      });
    }
  }
  // A thread's nodes may lie in two force chunks (dense rows of any length).
  // The flags are read after the population loads are issued: the branches
  // here wait for them, and ahead of the loads that wait was a memory round
  // trip of its own (forced D3Q27 257 x 129 x 129: 212 -> 161 us).
  const ChunkForce cf0 = chunk_force<FORCE>(a, idx0);
  ChunkForce cf1 = cf0;
  if constexpr (FORCE) {
    if (((idx0 + nv - 1) >> 5) != (idx0 >> 5)) cf1 = chunk_force<FORCE>(a, idx0 + nv - 1);
  }
  Words<kWords> out[advances(OP) ? Q : 1];
#pragma unroll
  for (int pr = 0; pr < NZ / 2; ++pr) {
    const int k0 = 2 * pr, k1 = 2 * pr + 1;
    F2 f[Q];
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      constexpr int ez = V::ez(i);
      const float c0 = elem<S, NZ>(in[i], k0), c1 = elem<S, NZ>(in[i], k1);
      if constexpr (ez == 0) {
        f[i] = F2(c0, c1);
      } else {
        const float e = St::cvt(in[i].extra);
        float s0, s1;
        if constexpr (ez > 0) {
          s0 = pr == 0 ? e : elem<S, NZ>(in[i], pr == 0 ? 0 : k0 - 1);
          s1 = c0;
        } else {
          s0 = c1;
          s1 = k1 == NZ - 1 ? e : elem<S, NZ>(in[i], k1 == NZ - 1 ? k1 : k1 + 1);
        }
        if constexpr (V::ex(i) != 0 || V::ey(i) != 0) {
          const bool in_row = enters<V::ex(i), V::ey(i)>(rf);
          // (at the bottom / top plane the z face's rule governs)
          s0 = in_row && !(ez > 0 && pr == 0 && bottom) ? c0 : s0;
          s1 = in_row && !(ez < 0 && k1 == NZ - 1 && top) ? c1 : s1;
        }
        if constexpr (PITCH && ez < 0) {
          // (partial vector: the row's last node is lane nv - 1; the padding
          // lanes after it keep any value)
          s0 = top && k0 == nv - 1 ? e : s0;
          s1 = top && k1 == nv - 1 ? e : s1;
        }
        f[i] = F2(s0, s1);
      }
    });
    if (k0 < nv && (on_moving_wall(a.g, rf, z0 + k0) ||
                    (k1 < nv && on_moving_wall(a.g, rf, z0 + k1)))) {
      const float *face_rho = static_cast<const float *>(a.face_rho_in);
      const int za = z0 + k0, zb = k1 < nv ? z0 + k1 : za;   // (a padding lane repeats its neighbour's)
      const WallRho<float> rho0(a.g, face_rho, rf, x, y, za), rho1(a.g, face_rho, rf, x, y, zb);
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (i != 0) {
          f[i].v.x -= moving_wall<Q, i, St::kShift>(a.g, rho0, rf, za);
          f[i].v.y -= moving_wall<Q, i, St::kShift>(a.g, rho1, rf, zb);
        }
      });
    }
    if (!PITCH || k0 < nv) {
      const bool s0 = ((idx0 + k0) >> 5) == (idx0 >> 5), s1 = ((idx0 + k1) >> 5) == (idx0 >> 5);
      finish_pair<Q, FORCE, St::kShift, OP>(a, f, idx0 + k0, x, y, z0 + k0, rf.any(),
                                            !PITCH || k1 < nv, lanes, s0 ? cf0 : cf1,
                                            s1 ? cf0 : cf1, bad);
    }
    if constexpr (advances(OP)) {
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if constexpr (St::kBits == 32) {
          out[i].w[k0] = __float_as_uint(f[i].v.x);
          out[i].w[k1] = __float_as_uint(f[i].v.y);
        } else {
          out[i].w[pr] = put2<S>(f[i].v.x, f[i].v.y);
        }
      });
    }
  }
  report_bad(a.status, bad);
  if constexpr (advances(OP)) {
    static_for<Q>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      T *dst = static_cast<T *>(a.p.dst[i]) + pidx0;
      if constexpr (ALIGNED) {
        st_words(dst, out[i]);
      } else {
        reinterpret_cast<unsigned short *>(dst)[0] = (unsigned short)(out[i].w[0] & 0xffffu);
        reinterpret_cast<unsigned short *>(dst)[1] = (unsigned short)(out[i].w[0] >> 16);
      }
    });
  }
}

// Vectorised step of FP64 rows (pz = nz or padded): thread = NZ consecutive
// nodes, pulled and finished node by node in double arithmetic, stored as
// vectors.
template <int Q, int S, bool FORCE, int NZ, bool PITCH>
__device__ __forceinline__ void step_vec64_body(const StepArgs &a, const unsigned t) {
  using St = Storage<S>;
  using T = typename St::T;
  using V = VSet<Q>;
  using R = typename St::R;
  static_assert(St::kBits == 64, "float64 rows");
  constexpr int kWords = 2 * NZ;
  const unsigned pidx0 = t * NZ;
  if (pidx0 >= (unsigned)a.g.np) return;
  int x, y, z0;
  a.pdec(pidx0, x, y, z0);
  if constexpr (PITCH) {
    if (z0 >= a.g.nz) {                      // row padding only
      put_padding_vector<Q, S, NZ>(a, pidx0);
      return;
    }
  }
  const unsigned idx0 = (unsigned)(x * a.g.ny + y) * (unsigned)a.g.nz + (unsigned)z0;
  const int nv = PITCH && a.g.nz - z0 < NZ ? a.g.nz - z0 : NZ;
  if (!lbm_in(x < a.g.nx && y < a.g.ny && pidx0 + NZ <= (unsigned)a.g.np &&
              idx0 + nv <= (unsigned)a.g.n))
    return;
  const R *face_rho = static_cast<const R *>(a.face_rho_in);
  R f[NZ][Q];
#pragma unroll
  for (int k = 0; k < NZ; ++k) {
    const int kk = k < nv ? k : nv - 1;   // (padding lanes repeat the row's last node)
    pull_node<Q, S, true>(a.p, a.g, face_rho, pidx0 + kk, x, y, z0 + kk, f[k]);
  }
  unsigned bad = 0;
#pragma unroll
  for (int k = 0; k < NZ; ++k) {
    const int z = z0 + k;
    if (k < nv)
      finish_node<Q, FORCE, St::kDev, St::kShift, Op::kStep>(
          a, f[k], idx0 + k, x, y, z, on_any_face(a.g, x, y, z),
          chunk_force<FORCE>(a, idx0 + k), bad);
  }
  report_bad(a.status, bad);
  static_for<Q>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    Words<kWords> raw;
#pragma unroll
    for (int k = 0; k < NZ; ++k) {
      raw.w[2 * k] = (unsigned)__double2loint(f[k][i]);
      raw.w[2 * k + 1] = (unsigned)__double2hiint(f[k][i]);
    }
    st_words(static_cast<T *>(a.p.dst[i]) + pidx0, raw);
  });
}

// PITCH: rows may carry padding (pz > nz); lattices without padding run the
// variant that has none of that code.
template <int Q, int S, bool FORCE, int NZ, bool PITCH>
__device__ __forceinline__ void step_vec_body(const StepArgs &a, const unsigned t) {
  if constexpr (Storage<S>::kBits == 64)
    step_vec64_body<Q, S, FORCE, NZ, PITCH>(a, t);
  else
    step_pairs_at<Q, S, FORCE, NZ, PITCH>(a, t * NZ);
}

// Register cap of the vectorised step for 16-bit storage, as resident blocks
// per SM asked of the compiler (0 = no cap).  A 16-bit population costs a
// whole float register once unpacked, so the 16-bit kernels hold too few
// bytes in flight per SM to cover HBM latency unless enough warps are
// resident (measured on B200 at 256^3, unforced, 128 threads, fraction of the
// copy peak without / with the cap: D3Q13 4 nodes 0.915 / 0.927, D3Q15 bf16s
// 4 nodes - / 0.873, D3Q19 4 nodes 0.687 / 0.859, D3Q27 2 nodes 0.821 /
// 0.828).  FP32 runs uncapped but for the forced D3Q19 pairs, us with 94 / 80
// registers: 161 x 65 x 65 18.6 / 17.5, 97 x 97 x 96 22.3 / 21.1, 129^3 55.1 /
// 54.6, 193 x 161 x 129 98.6 / 97.8, 256^3 376 / 377, 257^3 399 / 399; D3Q27 is
// faster uncapped, 161 against 165 us on 257 x 129 x 129.
template <int Q, int S, int NZ, bool FORCE>
constexpr int vec_reg_cap() {
  if (Storage<S>::kBits == 32) return FORCE && NZ == 2 && Q == 19 ? 80 : 0;
  if (Storage<S>::kBits != 16) return 0;
  if (NZ == 2 && FORCE) return Q == 19 ? 72 : Q == 27 ? 96 : 0;
  if (NZ == 2) return Q == 27 ? 96 : 0;
  if (NZ == 4) return Q == 13 ? 96 : Q == 15 || Q == 19 ? 128 : 0;
  return 0;
}
template <int Q, int S, int NZ, int TB, bool FORCE>
constexpr int vec_min_blocks() {
  return vec_reg_cap<Q, S, NZ, FORCE>() == 0 ? 0 : 65536 / (vec_reg_cap<Q, S, NZ, FORCE>() * TB);
}

template <int Q, int S, bool FORCE, int NZ, int TB, bool PITCH>
__global__ void __launch_bounds__(TB, (vec_min_blocks<Q, S, NZ, TB, FORCE>()))
    k_step_vec(const __grid_constant__ StepArgs a) {
  chain_enter();
  step_vec_body<Q, S, FORCE, NZ, PITCH>(a, blockIdx.x * TB + threadIdx.x);
}

// The same, two nodes per thread.
template <int Q, int S, bool FORCE, bool PITCH, Op OP>
__global__ void __launch_bounds__(128) k_observe_vec(const __grid_constant__ StepArgs a) {
  chain_enter();
  step_pairs_at<Q, S, FORCE, 2, PITCH, OP>(a, 2u * (blockIdx.x * 128u + threadIdx.x));
}

// Rows of odd length in 16-bit storage: thread k of a row takes the node pair
// (2k, 2k + 1) through the pair code with element-wise loads, and the last
// thread of the row the single node nz - 1 through the one-node code.  Same
// per-node arithmetic as every other shape.  For callers that keep odd rows
// dense (Lattice(pitch=False), lbm_lattice.pz = 0): padded rows run aligned
// pairs instead.  Measured on B200 it beats one node per thread only for
// unforced D3Q19 (+7 % at 257^3) and loses for D3Q27, so it is a tuner
// candidate, not a default.
template <int Q, int S, bool FORCE, int TB>
__global__ void __launch_bounds__(TB, (vec_min_blocks<Q, S, 2, TB, FORCE>()))
    k_step_odd(const __grid_constant__ StepArgs a, const FastDiv per_row, unsigned rows) {
  chain_enter();
  const unsigned t = blockIdx.x * TB + threadIdx.x;
  const unsigned row = fdiv(t, per_row);
  if (row >= rows) return;
  const unsigned z = 2u * (t - row * per_row.d);
  const unsigned idx = row * (unsigned)a.g.nz + z;
  if (z + 1u < (unsigned)a.g.nz)
    step_pairs_at<Q, S, FORCE, 2, false, Op::kStep, false>(a, idx);
  else
    step_scalar_body<Q, S, FORCE>(a, idx);
}

// ---------------------------------------------------------------------------
// Multi-lattice step: one launch advances `count` independent lattices of one
// velocity set and storage by one step.  Lattice e owns blocks
// [block_begin[e], block_begin[e+1]); each block finds its lattice by binary
// search, copies that lattice's StepArgs into shared memory and runs the
// same per-node code as the single-lattice kernels (NZ = 1: k_step's body,
// NZ > 1: k_step_vec's) on kBatchTiles consecutive tiles, so a lattice's
// result does not depend on which other lattices share the launch.
// ---------------------------------------------------------------------------
constexpr int kBatchTiles = 4;   // tiles of TB threads per block (amortises the lookup)

template <int Q, int S, bool FORCE, int NZ, int TB>
__global__ void __launch_bounds__(TB, (vec_min_blocks<Q, S, NZ, TB, FORCE>()))
    k_step_batch(const StepArgs *__restrict__ entries, const unsigned *__restrict__ block_begin,
                 int count) {
  __shared__ __align__(16) StepArgs sa;
  __shared__ unsigned s_entry;
  if (threadIdx.x == 0) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (block_begin[mid] <= blockIdx.x)
        lo = mid;
      else
        hi = mid - 1;
    }
    s_entry = (unsigned)lo;
  }
  __syncthreads();
  const unsigned e = s_entry;
  constexpr int kWordsArgs = (int)(sizeof(StepArgs) / 4);
  static_assert(sizeof(StepArgs) % 4 == 0, "StepArgs is copied as 32-bit words");
  const unsigned *src = reinterpret_cast<const unsigned *>(entries + e);
  unsigned *dst = reinterpret_cast<unsigned *>(&sa);
  for (int w = threadIdx.x; w < kWordsArgs; w += TB) dst[w] = src[w];
  __syncthreads();
  const unsigned t0 = (blockIdx.x - block_begin[e]) * (TB * kBatchTiles) + threadIdx.x;
#pragma unroll 1
  for (int it = 0; it < kBatchTiles; ++it) {
    if constexpr (NZ == 1)
      step_scalar_body<Q, S, FORCE>(sa, t0 + it * TB);
    else
      step_vec_body<Q, S, FORCE, NZ, true>(sa, t0 + it * TB);
  }
}


// ---------------------------------------------------------------------------
// TMA-staged persistent step.  Each CTA walks groups of R whole z-rows
// (row = (x, y)); for a row with interior (x, y) the source of direction i is
// row (x - ex, y - ey) of plane i, so one elected thread brings the group in
// with Q * R bulk copies (cp.async.bulk, completion counted on an mbarrier)
// into a ring of `stages` shared-memory stages, several groups ahead of the
// compute.  Threads then read their two consecutive nodes per direction from
// shared memory (z-1 / z+1 neighbours included; z = 0 / nz - 1 take the
// bottom / top face rule from global memory), finish the nodes and store
// them as 8-byte (fp32) / 4-byte (16-bit) pairs.  Rows on an x / y face are
// pulled from global memory with the full face rules.  Bytes in flight are
// bounded by shared memory, not registers -- what the 16-bit storage needs
// to reach HBM bandwidth.  Every barrier wait is bounded; a timeout sets
// LBM_STATUS_WAIT_TIMEOUT and the CTA drains its copies (bounded by the
// default limit) and stops; a drain that also times out sets
// LBM_STATUS_DRAIN_FAILED.
// ---------------------------------------------------------------------------
constexpr int kTmaThreads = 256;
constexpr unsigned kTmaWaitPolls = kTmaWaitPollsDefault;

struct TmaPlan {
  int rows_per_stage;
  int stages;
  unsigned row_bytes;
  long long groups;
  unsigned wait_polls;   // limit of the consumer waits (the drain keeps kTmaWaitPolls)
};


// working value(s) of one / two staged elements
template <int S>
__device__ __forceinline__ float sm_elem(const typename Storage<S>::T *p) {
  if constexpr (Storage<S>::kBits == 32)
    return *p;
  else if constexpr (S == LBM_STORAGE_FP16S)
    return __half2float(*p);
  else
    return __bfloat162float(*p);
}

template <int S>
__device__ __forceinline__ float2 sm_pair(const typename Storage<S>::T *p) {
  if constexpr (Storage<S>::kBits == 32)
    return *reinterpret_cast<const float2 *>(p);
  else
    return work2<S>(*reinterpret_cast<const unsigned *>(p));
}

template <int Q, int S, bool FORCE>
__global__ void __launch_bounds__(kTmaThreads) k_step_tma(const __grid_constant__ StepArgs a, const TmaPlan p) {
  using St = Storage<S>;
  using T = typename St::T;
  using V = VSet<Q>;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  T *buf = reinterpret_cast<T *>(smem + 128);
  const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
  const int R = p.rows_per_stage;
  const T *__restrict__ fa = static_cast<const T *>(a.fa);
  const float *face_rho = static_cast<const float *>(a.face_rho_in);
  const int tid = threadIdx.x;
  const long long G = gridDim.x;
  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) mbar_init(&bars[s], 1);
    mbar_init_fence();
  }
  __syncthreads();

  auto row_xy = [&](long long r, int &x, int &y) {
    x = (int)(r / ny);
    y = (int)(r - (long long)x * ny);
  };
  auto interior = [&](int x, int y) { return x > 0 && x < nx - 1 && y > 0 && y < ny - 1; };
  auto issue = [&](int s, long long g) {
    const long long r0 = g * R;
    unsigned bytes = 0;
    for (int j = 0; j < R; ++j) {
      int x, y;
      row_xy(r0 + j, x, y);
      if (interior(x, y)) bytes += Q * p.row_bytes;
    }
    if (bytes == 0) {
      mbar_arrive(&bars[s]);
      return;
    }
    mbar_arrive_expect_tx(&bars[s], bytes);
    for (int j = 0; j < R; ++j) {
      int x, y;
      row_xy(r0 + j, x, y);
      if (!interior(x, y)) continue;
      T *dst = buf + (long long)(s * R + j) * Q * nz;
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        const T *src = fa + (long long)i * a.g.n +
                       ((long long)(x - V::ex(i)) * ny + (y - V::ey(i))) * nz;
        bulk_copy_g2s(dst + (long long)i * nz, src, p.row_bytes, &bars[s]);
      });
    }
  };
  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      const long long g = blockIdx.x + s * G;
      if (g < p.groups) issue(s, g);
    }
  }

  const int half = nz / 2;
  long long k = 0;
  bool timed_out = false;
  for (;; ++k) {
    const long long g = blockIdx.x + k * G;
    if (g >= p.groups) break;
    const int s = (int)(k % p.stages);
    const unsigned par = (unsigned)((k / p.stages) & 1);
    const bool ok = mbar_wait_bounded(&bars[s], par, p.wait_polls);
    if (__syncthreads_or(!ok)) {
      timed_out = true;
      break;
    }
    for (int pi = tid; pi < R * half; pi += kTmaThreads) {
      const int j = pi / half, zp = pi - j * half;
      const long long r = g * R + j;
      int x, y;
      row_xy(r, x, y);
      const int z = 2 * zp;
      const unsigned idx = (unsigned)(r * nz + z);
      const ChunkForce cf = chunk_force<FORCE>(a, idx);
      float f0[Q], f1[Q];
      const bool row_in = interior(x, y);
      if (row_in) {
        const T *srow = buf + (long long)(s * R + j) * Q * nz;
        static_for<Q>([&](auto ic) {
          constexpr int i = decltype(ic)::value;
          constexpr int ez = V::ez(i);
          const T *rp = srow + (long long)i * nz;
          if constexpr (ez == 0) {
            const float2 v = sm_pair<S>(rp + z);
            f0[i] = v.x;
            f1[i] = v.y;
          } else if constexpr (ez > 0) {
            f1[i] = sm_elem<S>(rp + z);
            f0[i] = z == 0 ? St::work(static_cast<const T *>(a.p.zlo[i]) + idx)
                           : sm_elem<S>(rp + z - 1);
          } else {
            f0[i] = sm_elem<S>(rp + z + 1);
            f1[i] = z + 2 == nz ? St::work(static_cast<const T *>(a.p.zhi[i]) + (idx + 1))
                                : sm_elem<S>(rp + z + 2);
          }
        });
        if (a.g.moving != 0 && (z == 0 || z + 2 == nz)) {
          const RowFaces rf(a.g, x, y);
          const WallRho<float> rho0(a.g, face_rho, rf, x, y, z), rho1(a.g, face_rho, rf, x, y, z + 1);
          static_for<Q>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            if constexpr (i != 0) {
              f0[i] -= moving_wall<Q, i, St::kShift>(a.g, rho0, rf, z);
              f1[i] -= moving_wall<Q, i, St::kShift>(a.g, rho1, rf, z + 1);
            }
          });
        }
      } else {
        pull_node<Q, S, true>(a.p, a.g, face_rho, idx, x, y, z, f0);
        pull_node<Q, S, true>(a.p, a.g, face_rho, idx + 1, x, y, z + 1, f1);
      }
      unsigned bad = 0;
      finish_node<Q, FORCE, St::kDev, St::kShift, Op::kStep>(a, f0, idx, x, y, z, !row_in || z == 0, cf, bad);
      finish_node<Q, FORCE, St::kDev, St::kShift, Op::kStep>(a, f1, idx + 1, x, y, z + 1,
                                                             !row_in || z + 1 == nz - 1, cf, bad);
      report_bad(a.status, bad);
      static_for<Q>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        T *dst = static_cast<T *>(a.p.dst[i]) + idx;
        if constexpr (St::kBits == 32)
          *reinterpret_cast<float2 *>(dst) = make_float2(f0[i], f1[i]);
        else
          *reinterpret_cast<unsigned *>(dst) = put2<S>(f0[i], f1[i]);
      });
    }
    __syncthreads();
    if (tid == 0) {
      const long long g2 = g + (long long)p.stages * G;
      if (g2 < p.groups) {
        fence_proxy_async_smem();
        issue(s, g2);
      }
    }
  }
  if (timed_out && tid == 0) {
    unsigned bits = LBM_STATUS_WAIT_TIMEOUT;
    // drain the copies still in flight into this CTA's shared memory
    for (long long kk = k; kk < k + p.stages; ++kk) {
      if (blockIdx.x + kk * G >= p.groups) break;
      if (!mbar_wait_bounded(&bars[kk % p.stages], (unsigned)((kk / p.stages) & 1), kTmaWaitPolls))
        bits |= LBM_STATUS_DRAIN_FAILED;
    }
    if (a.status != nullptr) atomicOr(a.status, bits);
  }
}

// Launch shape of the fused step: nodes per thread (1 = scalar kernel, or
// NZ consecutive z-nodes moved as 4 / 8 / 16-byte vectors, the row pitch pz a
// multiple of NZ; a row's last vector may hold padding) and threads per block.
// Shapes lbm_flow_step accepts: the above, plus 2 nodes per thread for 16-bit
// rows of odd pitch (k_step_odd where they are dense, else one node).
inline bool step_shape_ok(int nodes, int pz, int bits);
inline bool step_shape_legal(int nodes, int pz, int bits) {
  return step_shape_ok(nodes, pz, bits) || (nodes == 2 && bits == 16 && pz % 2 == 1 && pz >= 3);
}

inline bool step_shape_ok(int nodes, int pz, int bits) {
  if (nodes == 1) return true;
  if (nodes != 2 && nodes != 4 && nodes != 8) return false;
  if (nodes * bits / 32 < 1 || nodes * bits / 32 > 4) return false;
  return pz % nodes == 0 && pz >= 2 * nodes;
}

// Shared-memory plan of the TMA-staged step for this device, or false when
// the lattice does not qualify (rows must be a multiple of 16 bytes, the
// population buffer 16-byte aligned, and two stages must fit).
struct DeviceInfo {
  int sms = 0, smem_sm = 0, smem_optin = 0;
};

inline bool device_info(DeviceInfo &d) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&d.smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) !=
      cudaSuccess)
    return false;
  if (cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
      cudaSuccess)
    return false;
  return true;
}

inline bool tma_plan(const Geom &g, int q, int bits, const void *fa, TmaPlan &p, int &ctas,
                     size_t &smem, unsigned &grid) {
  const int elem = bits / 8;
  const long long row_bytes = (long long)g.nz * elem;
  if (g.pz != g.nz) return false;   // whole rows are copied: no padding between them
  if (row_bytes % 16 != 0 || g.nz < 16 || ((uintptr_t)fa & 15u) != 0) return false;
  DeviceInfo d;
  if (!device_info(d)) return false;
  const long long rows = (long long)g.nx * g.ny;
  int R = 2 * kTmaThreads / g.nz;
  if (R < 1 || rows % R != 0) R = 1;
  const long long stage = (long long)R * q * row_bytes;
  const long long reserve = 1024 + 128;
  int stages = (int)std::min<long long>(8, (d.smem_sm / 2 - reserve) / stage);
  ctas = 2;
  if (stages < 3) {
    ctas = 1;
    stages = (int)std::min<long long>(8, (std::min(d.smem_optin, d.smem_sm) - reserve) / stage);
  }
  if (stages < 2) return false;
  p.rows_per_stage = R;
  p.stages = stages;
  p.row_bytes = (unsigned)row_bytes;
  p.groups = rows / R;
  p.wait_polls = tma_wait_polls();
  smem = 128 + (size_t)stages * stage;
  const long long want = (long long)ctas * d.sms;
  grid = (unsigned)std::min<long long>(p.groups, want);
  return true;
}

template <int Q, int S>
struct StepLauncher {
  template <bool FORCE>
  static int go_tma_f(const StepArgs &a, cudaStream_t s) {
    TmaPlan p;
    int ctas;
    size_t smem;
    unsigned grid;
    if (!tma_plan(a.g, Q, Storage<S>::kBits, a.fa, p, ctas, smem, grid)) {
      set_error("lbm_flow_step: this lattice does not qualify for row staging (rows must be a "
                "multiple of 16 bytes and at least 16 nodes, buffers 16-byte aligned)");
      return LBM_ERR_INVALID;
    }
    cudaError_t e = cudaFuncSetAttribute(k_step_tma<Q, S, FORCE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail_cuda(e, "lbm_flow_step");
    k_step_tma<Q, S, FORCE><<<grid, kTmaThreads, smem, s>>>(a, p);
    return LBM_OK;
  }
  static int go_tma(const StepArgs &a, bool force, cudaStream_t s) {
    if constexpr (Storage<S>::kBits == 64) {
      set_error("lbm_flow_step: row staging is not built for FP64 storage");
      return LBM_ERR_UNSUPPORTED;
    } else {
      return force ? go_tma_f<true>(a, s) : go_tma_f<false>(a, s);
    }
  }

  template <int NZ, int TB>
  static void go_vec(const StepArgs &a, bool force, cudaStream_t s) {
    const unsigned nb = blocks_for(a.g.np / NZ, TB);
    if (a.g.pz != a.g.nz) {
      if (force)
        launch_chained(k_step_vec<Q, S, true, NZ, TB, true>, nb, TB, 0, s, a);
      else
        launch_chained(k_step_vec<Q, S, false, NZ, TB, true>, nb, TB, 0, s, a);
    } else {
      if (force)
        launch_chained(k_step_vec<Q, S, true, NZ, TB, false>, nb, TB, 0, s, a);
      else
        launch_chained(k_step_vec<Q, S, false, NZ, TB, false>, nb, TB, 0, s, a);
    }
  }
  template <int NZ>
  static void go_nz(const StepArgs &a, bool force, int threads, cudaStream_t s) {
    if (threads == 128)
      go_vec<NZ, 128>(a, force, s);
    else
      go_vec<NZ, 256>(a, force, s);
  }
  template <bool FORCE, int TB>
  static void go_odd_f(const StepArgs &a, cudaStream_t s) {
    if constexpr (Storage<S>::kBits == 16) {
      const unsigned per_row = (unsigned)(a.g.nz + 1) / 2;
      const unsigned rows = (unsigned)(a.g.nx * a.g.ny);
      const unsigned nb = blocks_for((long long)rows * per_row, TB);
      launch_chained(k_step_odd<Q, S, FORCE, TB>, nb, TB, 0, s, a, make_fastdiv(per_row), rows);
    }
  }
  static void go_odd(const StepArgs &a, bool force, int threads, cudaStream_t s) {
    if (threads == 256)
      force ? go_odd_f<true, 256>(a, s) : go_odd_f<false, 256>(a, s);
    else
      force ? go_odd_f<true, 128>(a, s) : go_odd_f<false, 128>(a, s);
  }
  // Observation launch (Op::kBoth: with the step): its shape does not depend on
  // the step's own, but that one node per thread stays one.
  template <Op OP, bool FORCE>
  static void go_observe_f(const StepArgs &a, bool pairs, cudaStream_t s) {
    if constexpr (Storage<S>::kBits != 64) {
      if (pairs) {
        const unsigned nb = blocks_for(a.g.np / 2, 128);
        if (a.g.pz != a.g.nz)
          launch_chained(k_observe_vec<Q, S, FORCE, true, OP>, nb, 128, 0, s, a);
        else
          launch_chained(k_observe_vec<Q, S, FORCE, false, OP>, nb, 128, 0, s, a);
        return;
      }
    }
    constexpr int tb = scalar_threads<Q, S>();
    launch_chained(k_observe<Q, S, FORCE, OP>, blocks_for(a.g.n, tb), tb, 0, s, a);
  }
  template <Op OP>
  static int go_observe(StepArgs a, bool force, int nodes, cudaStream_t s) {
    constexpr int bits = Storage<S>::kBits;
    if (nodes == LBM_STEP_ROWS) {   // (a lattice that cannot be row-staged is refused here too)
      TmaPlan p;
      int ctas;
      size_t smem;
      unsigned grid;
      if (bits == 64 || !tma_plan(a.g, Q, bits, a.fa, p, ctas, smem, grid)) return go_tma(a, force, s);
    }
    const uintptr_t at = (uintptr_t)a.obs_f | (uintptr_t)a.obs_rho | (uintptr_t)a.obs_u;
    a.obs_pairs = a.g.n % 2 == 0 && a.g.nz % 2 == 0 && at % 8 == 0;
    // Odd rows (or buffers at odd places) without the step: one node per thread
    // but for the narrower 16-bit sets.  Measured on B200, us with pairs / one
    // node per thread, rho and u, then f: D3Q19 fp32 257^3 236 / 223, 419 /
    // 415, 256 x 256 x 255 230 / 220, 417 / 385; D3Q15 fp32 129^3 37 / 27, 58 /
    // 46; D3Q27 257 x 129 x 129 fp32 103 / 94, 174 / 161, fp16s 96 / 89, 175 /
    // 162; fp16s D3Q19 257^3 176 / 220, 361 / 416, D3Q15 129^3 23 / 29, 46 / 47,
    // D3Q13 bf16s 257^3 142 / 193, 253 / 281.  With the step, pairs win
    // throughout (D3Q19 fp32 257^3, all fields: 723 / 895).
    const bool pairs = nodes != 1 && step_shape_ok(2, a.g.pz, bits) &&
                       (a.obs_pairs || OP == Op::kBoth || (bits == 16 && Q != 27));
    if (force)
      go_observe_f<OP, true>(a, pairs, s);
    else
      go_observe_f<OP, false>(a, pairs, s);
    return LBM_OK;
  }
  static int go(const StepArgs &a, bool force, int nodes, int threads, cudaStream_t s) {
    constexpr int bits = Storage<S>::kBits;
    if (a.fb == nullptr) return go_observe<Op::kObserve>(a, force, nodes, s);
    if (a.obs_f != nullptr || a.obs_rho != nullptr || a.obs_u != nullptr)
      return go_observe<Op::kBoth>(a, force, nodes, s);
    if (nodes == LBM_STEP_ROWS) return go_tma(a, force, s);
    const bool odd_pairs = bits == 16 && a.g.pz % 2 == 1 && a.g.pz == a.g.nz && a.g.nz >= 3;
    // (k_step_odd's rows are dense: an odd pitch beyond nz takes one node per thread)
    if (nodes == 2 && a.g.pz % 2 == 1 && !odd_pairs) nodes = 1;
    if (nodes == 0) {
      // Measured on B200, blocks of 128 threads, fraction of the copy peak for
      // 2 / 4 nodes per thread (256^3 unless said): FP32 D3Q19 1.02 / 1.00
      // (512^3 3007 us a step; one node per thread is 1 % slower); 16-bit
      // D3Q13 0.83 / 0.93; D3Q15 fp16s 0.83 / 0.77, bf16s 0.82 / 0.87; D3Q19
      // fp16s 0.87 / 0.86 (512^3 0.88 / 0.89), bf16s 0.87 / 0.95; D3Q27 fp16s
      // 0.83 / 0.82.  Padded rows keep pairs but for D3Q13 (D3Q19 fp16s 257^3
      // 240 us with pairs, 267 with 4 nodes; D3Q13 170, 162), and so do forced
      // kernels (4 nodes spill).  Rows of odd length without padding take one
      // node per thread; the odd-row pair kernel is a tuner candidate only.
      constexpr bool four = bits == 16 && (Q == 13 || Q == 19 || (Q == 15 && S == LBM_STORAGE_BF16S));
      const int want = four && !force && (Q == 13 || a.g.pz == a.g.nz) ? 4 : 2;
      nodes = step_shape_ok(want, a.g.pz, bits) ? want : step_shape_ok(2, a.g.pz, bits) ? 2 : 1;
      threads = threads ? threads : 128;
    }
    if (nodes == 2 && odd_pairs) {
      go_odd(a, force, threads, s);
      return LBM_OK;
    }
    if (nodes == 2) {
      go_nz<2>(a, force, threads, s);
      return LBM_OK;
    }
    if constexpr (bits != 64) {
      if (nodes == 4) {
        go_nz<4>(a, force, threads, s);
        return LBM_OK;
      }
    }
    if constexpr (bits == 16) {
      if (nodes == 8) {
        go_nz<8>(a, force, threads, s);
        return LBM_OK;
      }
    }
    constexpr int tb = scalar_threads<Q, S>();
    const unsigned nb = blocks_for(a.g.n, tb);
    if (force)
      launch_chained(k_step<Q, S, true>, nb, tb, 0, s, a);
    else
      launch_chained(k_step<Q, S, false>, nb, tb, 0, s, a);
    return LBM_OK;
  }
};

// Step statistics of velocity set Q and storage S: init, k_stats (stats_blocks
// blocks per SM at most; the kernel streams the populations once), finish.
template <int Q, int S>
int run_stats_qs(const StepArgs &a, bool force, unsigned long long *out, cudaStream_t s) {
  DeviceInfo d;
  int sms = 148;
  if (device_info(d)) sms = d.sms;
  const unsigned blocks = (unsigned)std::min<long long>(blocks_for(a.g.n, kStatsThreads),
                                                        (long long)sms * stats_blocks<Q, S>());
  launch_chained(k_stats_init<Q>, 1, 32, 0, s, out);
  if (force)
    launch_chained(k_stats<Q, S, true>, blocks, kStatsThreads, 0, s, a, out);
  else
    launch_chained(k_stats<Q, S, false>, blocks, kStatsThreads, 0, s, a, out);
  launch_chained(k_stats_finish<Q>, 1, 32, 0, s, out, (double)a.g.n);
  LBM_LAUNCH_CHECK("lbm_flow_stats");
  return LBM_OK;
}

// Multi-lattice launch for velocity set Q and storage S: nodes per thread 1
// (256 threads), 2 or 4 (128 threads).
template <int Q, int S>
int run_step_batch_qs(const StepArgs *entries, const unsigned *block_begin, int count,
                      unsigned total_blocks, bool force, int nodes, cudaStream_t s) {
  if (nodes == 2) {
    if (force)
      k_step_batch<Q, S, true, 2, 128><<<total_blocks, 128, 0, s>>>(entries, block_begin, count);
    else
      k_step_batch<Q, S, false, 2, 128><<<total_blocks, 128, 0, s>>>(entries, block_begin, count);
  } else if (nodes == 4 && Storage<S>::kBits != 64) {
    if constexpr (Storage<S>::kBits != 64) {
      if (force)
        k_step_batch<Q, S, true, 4, 128><<<total_blocks, 128, 0, s>>>(entries, block_begin, count);
      else
        k_step_batch<Q, S, false, 4, 128><<<total_blocks, 128, 0, s>>>(entries, block_begin, count);
    }
  } else {
    if (force)
      k_step_batch<Q, S, true, 1, 256><<<total_blocks, 256, 0, s>>>(entries, block_begin, count);
    else
      k_step_batch<Q, S, false, 1, 256><<<total_blocks, 256, 0, s>>>(entries, block_begin, count);
  }
  LBM_LAUNCH_CHECK("lbm_flow_step_batch");
  return LBM_OK;
}

// One fused step for velocity set Q and storage S (explicitly instantiated
// once per (Q, S) in lbm_step_inst.cu, so the launch-shape variants compile
// in parallel translation units).
template <int Q, int S>
int run_step_qs(const StepArgs &a, bool force, int nodes, int threads, cudaStream_t s) {
  const int rc = StepLauncher<Q, S>::go(a, force, nodes, threads, s);
  if (rc) return rc;
  LBM_LAUNCH_CHECK("lbm_flow_step");
  return LBM_OK;
}

#define LBM_FOR_EACH_QS(X)                                                                  \
  X(13, 0) X(13, 1) X(13, 2) X(13, 3) X(15, 0) X(15, 1) X(15, 2) X(15, 3) X(19, 0) X(19, 1) \
  X(19, 2) X(19, 3) X(27, 0) X(27, 1) X(27, 2) X(27, 3)

}  // namespace lbm
