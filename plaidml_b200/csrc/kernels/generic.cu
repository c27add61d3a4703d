// General Tile contraction and element-wise kernels: complete but unspecialised.
//
// contraction  one thread per output element.  When every output coordinate is a single
//              index variable (the usual case) those variables are read off the element's
//              position and the thread loops over the remaining (reduction) variables;
//              otherwise, per output dim that mixes variables (`s*x + i`), one variable is
//              solved for from the element's coordinate and the others are looped over, and
//              only with a rational output coordinate does the thread walk the whole index
//              box and keep the points that land on its element.  A point contributes only
//              if every tensor access is in range, every constraint holds and every rational
//              index is integral.
// eltwise      one thread per output element, operands read through broadcast strides.
//
// Arithmetic happens in the contraction's element type: integers wrap (computed in 64
// bits and truncated on store), f16 / bf16 round after every operation, max / min are a
// compare-and-select with an ordered compare.
#include "dependent_launch.h"
#include "generic.h"
#include "typed_access.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>
#include <cstdlib>

namespace pmlb {

namespace {

template <class T>
__device__ __forceinline__ T agg_identity(int agg, int dtype) {
  constexpr bool is_float = static_cast<T>(0.5) != T(0);
  if (agg == PMLB_AGG_PROD) return T(1);
  if (agg == PMLB_AGG_MAX) {
    if constexpr (is_float) return static_cast<T>(-INFINITY);
    switch (dtype) {
      case PMLB_I8: return static_cast<T>(-128);
      case PMLB_I16: return static_cast<T>(-32768);
      case PMLB_I32: return static_cast<T>(-2147483647 - 1);
      case PMLB_I64: return static_cast<T>(-9223372036854775807LL - 1);
      default: return T(0);
    }
  }
  if (agg == PMLB_AGG_MIN) {
    if constexpr (is_float) return static_cast<T>(INFINITY);
    switch (dtype) {
      case PMLB_BOOL: return T(1);
      case PMLB_I8: return static_cast<T>(127);
      case PMLB_U8: return static_cast<T>(255);
      case PMLB_I16: return static_cast<T>(32767);
      case PMLB_U16: return static_cast<T>(65535);
      case PMLB_I32: return static_cast<T>(2147483647);
      case PMLB_U32: return static_cast<T>(4294967295LL);
      case PMLB_I64: return static_cast<T>(9223372036854775807LL);
      default: return static_cast<T>(~0ULL);
    }
  }
  return T(0);
}

__device__ __forceinline__ long long floor_div_exact(long long num, int den, bool* integral) {
  if (den == 1) return num;
  const long long q = num / den;
  if (q * den != num) *integral = false;
  return q;
}

// ------------------------------------------------------------------ contraction

template <class T>
__global__ void __launch_bounds__(256) contract_kernel(const __grid_constant__ GenericParams p) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= p.out_elems) return;

  long long oc[PMLB_MAX_RANK];
  long long rem = e;
  long long out_off = 0, init_off = 0;
  for (int d = p.out.rank - 1; d >= 0; --d) {
    oc[d] = rem % p.out.sizes[d];
    rem /= p.out.sizes[d];
    out_off += oc[d] * p.out.strides[d];
    init_off += oc[d] * p.init.strides[d];
  }

  long long x[PMLB_MAX_IDX];
  for (int i = 0; i < PMLB_MAX_IDX; ++i) x[i] = 0;
  bool alive = true;
  if (p.direct) {
    for (int d = 0; d < p.out.rank; ++d) {
      const int v = p.out_var[d];
      const long long xv = oc[d] - p.out.off[d];
      if (xv < 0 || xv >= p.range[v]) alive = false;
      x[v] = xv;
    }
  }
  for (int j = 0; j < p.n_loop; ++j) {
    if (p.range[p.loop_var[j]] <= 0) alive = false;
  }
  for (int s = 0; s < p.n_solve; ++s) {
    if (p.range[p.solve_var[s]] <= 0) alive = false;
  }

  T acc = p.has_init ? narrow<T>(load_as<T>(p.initp, p.init.dtype, init_off), p.out.dtype)
                     : agg_identity<T>(p.agg, p.out.dtype);

  while (alive) {
    bool ok = true;
    for (int s = 0; s < p.n_solve && ok; ++s) {
      const int d = p.solve_dim[s];
      const int v = p.solve_var[s];
      x[v] = 0;
      long long num = oc[d] - p.out.off[d];
      for (int i = 0; i < p.n_idx; ++i) num -= static_cast<long long>(p.out.coef[d][i]) * x[i];
      const long long xv = floor_div_exact(num, p.out.coef[d][v], &ok);
      if (xv < 0 || xv >= p.range[v]) ok = false;
      x[v] = xv;
    }
    if (!p.direct) {
      for (int d = 0; d < p.out.rank && ok; ++d) {
        long long num = p.out.off[d];
        for (int i = 0; i < p.n_idx; ++i) num += static_cast<long long>(p.out.coef[d][i]) * x[i];
        const long long c = floor_div_exact(num, p.out.den[d], &ok);
        if (c != oc[d]) ok = false;
      }
    }
    for (int c = 0; c < p.n_cons && ok; ++c) {
      long long v = p.cons_off[c];
      for (int i = 0; i < p.n_idx; ++i) v += static_cast<long long>(p.cons_coef[c][i]) * x[i];
      if (v < 0 || v >= p.cons_range[c]) ok = false;
    }
    long long soff[3] = {0, 0, 0};
    for (int s = 0; s < p.n_src && ok; ++s) {
      const GAccess& a = p.src[s];
      for (int d = 0; d < a.rank; ++d) {
        long long num = a.off[d];
        for (int i = 0; i < p.n_idx; ++i) num += static_cast<long long>(a.coef[d][i]) * x[i];
        const long long c = floor_div_exact(num, a.den[d], &ok);
        if (c < 0 || c >= a.sizes[d]) ok = false;
        soff[s] += c * a.strides[d];
      }
    }
    if (ok) {
      T v;
      const int odt = p.out.dtype;
      switch (p.combo) {
        case PMLB_COMBO_MUL:
          v = narrow<T>(load_as<T>(p.srcp[0], p.src[0].dtype, soff[0]) *
                            load_as<T>(p.srcp[1], p.src[1].dtype, soff[1]),
                        odt);
          break;
        case PMLB_COMBO_ADD:
          v = narrow<T>(load_as<T>(p.srcp[0], p.src[0].dtype, soff[0]) +
                            load_as<T>(p.srcp[1], p.src[1].dtype, soff[1]),
                        odt);
          break;
        case PMLB_COMBO_EQ: {
          bool eq;
          if (dtype_is_float(p.src[0].dtype) || dtype_is_float(p.src[1].dtype)) {
            eq = load_as<double>(p.srcp[0], p.src[0].dtype, soff[0]) ==
                 load_as<double>(p.srcp[1], p.src[1].dtype, soff[1]);
          } else {
            eq = load_as<long long>(p.srcp[0], p.src[0].dtype, soff[0]) ==
                 load_as<long long>(p.srcp[1], p.src[1].dtype, soff[1]);
          }
          v = eq ? T(1) : T(0);
          break;
        }
        case PMLB_COMBO_COND: {
          bool eq;
          if (dtype_is_float(p.src[0].dtype) || dtype_is_float(p.src[1].dtype)) {
            eq = load_as<double>(p.srcp[0], p.src[0].dtype, soff[0]) ==
                 load_as<double>(p.srcp[1], p.src[1].dtype, soff[1]);
          } else {
            eq = load_as<long long>(p.srcp[0], p.src[0].dtype, soff[0]) ==
                 load_as<long long>(p.srcp[1], p.src[1].dtype, soff[1]);
          }
          v = eq ? narrow<T>(load_as<T>(p.srcp[2], p.src[2].dtype, soff[2]), odt) : T(0);
          break;
        }
        default:
          v = narrow<T>(load_as<T>(p.srcp[0], p.src[0].dtype, soff[0]), odt);
          break;
      }
      switch (p.agg) {
        case PMLB_AGG_SUM: acc = narrow<T>(acc + v, odt); break;
        case PMLB_AGG_PROD: acc = narrow<T>(acc * v, odt); break;
        case PMLB_AGG_MAX: acc = (acc > v) ? acc : v; break;
        case PMLB_AGG_MIN: acc = (acc < v) ? acc : v; break;
        default: acc = v; break;
      }
    }
    int j = p.n_loop - 1;
    while (j >= 0) {
      const int v = p.loop_var[j];
      if (++x[v] < p.range[v]) break;
      x[v] = 0;
      --j;
    }
    if (j < 0) break;
  }
  store_as<T>(p.outp, p.out.dtype, out_off, acc);
}

// ------------------------------------------------------------------ contraction, strided form

template <class T> __device__ __forceinline__ T rounded_mul(T a, T b) { return a * b; }
template <class T> __device__ __forceinline__ T rounded_add(T a, T b) { return a + b; }
template <> __device__ __forceinline__ float rounded_mul<float>(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float rounded_add<float>(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ double rounded_mul<double>(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double rounded_add<double>(double a, double b) { return __dadd_rn(a, b); }

// The terms of [lo, hi) of the innermost loop, in order, every operation rounded on its own as in the kernel above.
__device__ __forceinline__ float lean_term(int combo, float a, float b) {
  return combo == PMLB_COMBO_MUL ? __fmul_rn(a, b) : (combo == PMLB_COMBO_ADD ? __fadd_rn(a, b) : a);
}
__device__ __forceinline__ float lean_fold(int agg, float acc, float v) {
  switch (agg) {
    case PMLB_AGG_SUM: return __fadd_rn(acc, v);
    case PMLB_AGG_PROD: return __fmul_rn(acc, v);
    case PMLB_AGG_MAX: return (acc > v) ? acc : v;
    case PMLB_AGG_MIN: return (acc < v) ? acc : v;
    default: return v;
  }
}

template <int V>
struct LeanVec {
  float v[V];
};
// V consecutive elements, or (step 0) one for all of them.
template <int V>
__device__ __forceinline__ LeanVec<V> lean_load(const float* p, bool one) {
  LeanVec<V> r;
  if constexpr (V == 4) {
    if (one) {
      const float x = __ldg(p);
#pragma unroll
      for (int i = 0; i < V; ++i) r.v[i] = x;
    } else {
      const float4 u = __ldg(reinterpret_cast<const float4*>(p));
      r.v[0] = u.x, r.v[1] = u.y, r.v[2] = u.z, r.v[3] = u.w;
    }
  } else {
    r.v[0] = __ldg(p);
  }
  return r;
}

// What every thread of the strided form has: its element's coordinates turned into offsets and bounds values.
struct LeanPlace {
  long long out, init;
  int src[2];
  int check[4];
};
__device__ __forceinline__ LeanPlace lean_place(const LeanParams& p, int e) {
  LeanPlace w;
  w.out = w.init = 0;
  w.src[0] = p.src[0].base, w.src[1] = p.src[1].base;
#pragma unroll
  for (int k = 0; k < 4; ++k) w.check[k] = p.check[k].base;
  for (int d = p.rank - 1; d >= 0; --d) {
    const int q = fast_div(e, p.fd_size[d]);
    const int c = e - q * p.size[d];
    e = q;
    w.out += c * p.out_stride[d];
    w.init += c * p.init_stride[d];
    w.src[0] += c * p.src[0].out[d];
    w.src[1] += c * p.src[1].out[d];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k < p.n_check) w.check[k] += c * p.check[k].out[d];
    }
  }
  return w;
}

// Narrows [lo, hi) to the values x of the innermost loop with 0 <= c + step * x < size.
__device__ __forceinline__ void lean_clip(int c, int step, int size, int* lo, int* hi) {
  if (step == 0) {
    if (static_cast<unsigned>(c) >= static_cast<unsigned>(size)) *hi = 0;
  } else if (step == 1) {
    *lo = max(*lo, -c);
    *hi = min(*hi, size - c);
  } else {
    // first and last x of the run (exact in 64 bits: c and size are anywhere in 32)
    const long long s = step, first = s > 0 ? -static_cast<long long>(c) : static_cast<long long>(size) - 1 - c;
    const long long last = s > 0 ? static_cast<long long>(size) - 1 - c : -static_cast<long long>(c);
    const long long a = s > 0 ? s : -s;
    const long long f = s > 0 ? first : -first, l = s > 0 ? last : -last;   // f <= a * x <= l
    const long long from = f > 0 ? (f + a - 1) / a : 0, to = l >= 0 ? l / a : -1;
    if (from > *lo) *lo = static_cast<int>(from < 0x7fffffff ? from : 0x7fffffff);
    if (to + 1 < *hi) *hi = static_cast<int>(to + 1);
  }
}

// f32 throughout.  A thread computes V consecutive elements of the last output dim (V = 4: both sources have step 1 or 0
// there, rows 16-byte aligned, no bounds test looks at it).  Per term one load per source and the two operations: the
// innermost loop's run is cut to its valid part beforehand instead of testing every term, and offsets advance by steps
// instead of being recomputed from all ten variables in 64 bits.  Bound by the loads it repeats from L1 / L2 (3x3
// depthwise: nine of each per result).  32 x 56 x 56 x 128 depthwise 3x3: general kernel 3898 us, this one
// 86 us, and 6 us on one image (142 us before).
template <int V>
__global__ void __launch_bounds__(256) contract_lean_f32_kernel(const __grid_constant__ LeanParams p) {
  const long long t = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (t * V >= p.elems) return;
  const LeanPlace w = lean_place(p, static_cast<int>(t * V));
  const float* s0 = static_cast<const float*>(p.srcp[0]);
  const float* s1 = static_cast<const float*>(p.n_src > 1 ? p.srcp[1] : p.srcp[0]);
  const int last = p.rank - 1;
  const bool one0 = V > 1 && p.src[0].out[last] == 0, one1 = V > 1 && p.src[1].out[last] == 0;
  const bool two = p.n_src > 1;
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    acc[i] = p.has_init ? __ldg(static_cast<const float*>(p.initp) + w.init + (V > 1 ? i * p.init_stride[last] : 0))
                        : agg_identity<float>(p.agg, PMLB_F32);
  }
  const int st0 = p.src[0].loop[3], st1 = p.src[1].loop[3];
  for (int a = 0; a < p.loop[0]; ++a) {
    for (int b = 0; b < p.loop[1]; ++b) {
      for (int c = 0; c < p.loop[2]; ++c) {
        int lo = 0, hi = p.loop[3];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < p.n_check) {
            const LeanParams::Check& ck = p.check[k];
            lean_clip(w.check[k] + a * ck.loop[0] + b * ck.loop[1] + c * ck.loop[2], ck.loop[3], ck.size, &lo, &hi);
          }
        }
        const float* q0 = s0 + (w.src[0] + a * p.src[0].loop[0] + b * p.src[0].loop[1] + c * p.src[0].loop[2] + lo * st0);
        const float* q1 = s1 + (two ? w.src[1] + a * p.src[1].loop[0] + b * p.src[1].loop[1] + c * p.src[1].loop[2] + lo * st1 : 0);
        if (p.agg == PMLB_AGG_SUM && p.combo == PMLB_COMBO_MUL) {
#pragma unroll 4
          for (int x = lo; x < hi; ++x) {
            const LeanVec<V> u = lean_load<V>(q0, one0), v = lean_load<V>(q1, one1);
            q0 += st0;
            q1 += st1;
#pragma unroll
            for (int i = 0; i < V; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(u.v[i], v.v[i]));
          }
        } else {
          for (int x = lo; x < hi; ++x) {
            const LeanVec<V> u = lean_load<V>(q0, one0);
            LeanVec<V> v = u;
            if (two) v = lean_load<V>(q1, one1);
            q0 += st0;
            q1 += st1;
#pragma unroll
            for (int i = 0; i < V; ++i) acc[i] = lean_fold(p.agg, acc[i], lean_term(p.combo, u.v[i], v.v[i]));
          }
        }
      }
    }
  }
  float* out = static_cast<float*>(p.outp) + w.out;
  if constexpr (V == 4) {
    *reinterpret_cast<float4*>(out) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else {
    *out = acc[0];
  }
}

// Sums of f32 products, kRun neighbours of the last-but-one output dim (columns of an image, rows of a matrix) times W
// elements of the last dim per thread: the operand that does not move along the run (the filter) is read once per term
// for all of them, and set-up, clipping and loop control are shared.  Terms are added in the same order, with one
// rounding per term instead of two.  kRun = 4: the filter's share of the loads drops to a fifth, 64 registers leave 32
// warps per SM.  Takes problems with at least kRunThreads threads at that width (four blocks per SM): smaller ones need
// the parallelism more, and keep the separate roundings that small exact expectations were written for.  Bound by
// instruction issue and the latency of the loads.  3x3 depthwise, 32 x 56 x 56 x 128: 86 -> 38 us (103 MB of
// compulsory traffic: 2.7 TB/s); 16 x 57 x 57 x 145
// (W = 1): 156 -> 58 us.
constexpr int kRun = 4;
constexpr int kRunBlock = 128;
constexpr long long kRunThreads = 75776;

struct LeanRun {
  int moving;                 // the source that moves along the run
  int groups, runs;           // groups of W of the last dim, runs of the last-but-one
  FastDiv fd_groups, fd_runs;
  int n_clip, n_test;         // bounds tests that the run does not change / changes
  LeanParams::Check clip[4], test[4];
  int reach_low[4], reach_high[4];   // how far a run and the innermost loop move a test's value
  long long threads;
};

template <int W>
struct alignas(W * 4) RunVec {
  float v[W];
};

// a + u * f (the packed form of sm_100 does two lanes per instruction).
__device__ __forceinline__ void add_products(RunVec<4>& a, const RunVec<4>& u, const RunVec<4>& f) {
  asm("{\n\t"
      ".reg .b64 x, y, p;\n\t"
      "mov.b64 x, {%4, %5};\n\t"
      "mov.b64 y, {%8, %9};\n\t"
      "mov.b64 p, {%0, %1};\n\t"
      "fma.rn.f32x2 p, x, y, p;\n\t"
      "mov.b64 {%0, %1}, p;\n\t"
      "mov.b64 x, {%6, %7};\n\t"
      "mov.b64 y, {%10, %11};\n\t"
      "mov.b64 p, {%2, %3};\n\t"
      "fma.rn.f32x2 p, x, y, p;\n\t"
      "mov.b64 {%2, %3}, p;\n\t"
      "}"
      : "+f"(a.v[0]), "+f"(a.v[1]), "+f"(a.v[2]), "+f"(a.v[3])
      : "f"(u.v[0]), "f"(u.v[1]), "f"(u.v[2]), "f"(u.v[3]), "f"(f.v[0]), "f"(f.v[1]), "f"(f.v[2]), "f"(f.v[3]));
}
__device__ __forceinline__ void add_products(RunVec<1>& a, const RunVec<1>& u, const RunVec<1>& f) {
  a.v[0] = __fmaf_rn(u.v[0], f.v[0], a.v[0]);
}

// W consecutive elements, or (ONE) one for all of them.
template <int W, bool ONE>
__device__ __forceinline__ RunVec<W> run_load(const float* p) {
  RunVec<W> r;
  if constexpr (W == 4 && !ONE) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p));
    r.v[0] = u.x, r.v[1] = u.y, r.v[2] = u.z, r.v[3] = u.w;
  } else {
    const float x = __ldg(p);
#pragma unroll
    for (int i = 0; i < W; ++i) r.v[i] = x;
  }
  return r;
}

// ONE_M / ONE_F: that source is one value for a whole group.  NT: at most this many clips and tests.
template <int W, bool ONE_M, bool ONE_F, int NT>
__global__ void __launch_bounds__(kRunBlock, 1024 / kRunBlock)
contract_lean_run_kernel(const __grid_constant__ LeanParams p, const __grid_constant__ LeanRun r) {
  const long long t = static_cast<long long>(blockIdx.x) * kRunBlock + threadIdx.x;
  if (t >= r.threads) return;
  const int last = p.rank - 1, along = p.rank - 2;
  int e = static_cast<int>(t);
  const int group = e - fast_div(e, r.fd_groups) * r.groups;
  e = fast_div(e, r.fd_groups);
  const int run = e - fast_div(e, r.fd_runs) * r.runs;
  e = fast_div(e, r.fd_runs);
  const int x0 = run * kRun;
  const LeanParams::Source& sm = p.src[r.moving];
  const LeanParams::Source& sf = p.src[1 - r.moving];
  long long out = x0 * p.out_stride[along] + group * W * p.out_stride[last];
  int om = sm.base + x0 * sm.out[along] + group * W * sm.out[last], of = sf.base + group * W * sf.out[last];
  int clip[NT], test[NT];
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    clip[k] = r.clip[k].base + group * W * r.clip[k].out[last];
    test[k] = r.test[k].base + x0 * r.test[k].out[along] + group * W * r.test[k].out[last];
  }
  for (int d = along - 1; d >= 0; --d) {
    const int q = fast_div(e, p.fd_size[d]);
    const int c = e - q * p.size[d];
    e = q;
    out += c * p.out_stride[d];
    om += c * sm.out[d];
    of += c * sf.out[d];
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      clip[k] += c * r.clip[k].out[d];
      test[k] += c * r.test[k].out[d];
    }
  }
  const float* ms = static_cast<const float*>(p.srcp[r.moving]) + om;
  const float* fs = static_cast<const float*>(p.srcp[1 - r.moving]) + of;
  const long long step_x = sm.out[along];
  const int st_m = sm.loop[3], st_f = sf.loop[3];
  const int n = min(kRun, p.size[along] - x0);
  RunVec<W> acc[kRun];
#pragma unroll
  for (int x = 0; x < kRun; ++x) {
#pragma unroll
    for (int i = 0; i < W; ++i) acc[x].v[i] = 0.f;
  }
  for (int a = 0; a < p.loop[0]; ++a) {
    for (int b = 0; b < p.loop[1]; ++b) {
      for (int c = 0; c < p.loop[2]; ++c) {
        // tests that the run does not change cut the innermost loop; the others hold for all of the run and the loop
        // (the inside of the image), or are made per term
        int lo = 0, hi = p.loop[3];
        bool inside = n == kRun;
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (k < r.n_clip) {
            const LeanParams::Check& ck = r.clip[k];
            lean_clip(clip[k] + a * ck.loop[0] + b * ck.loop[1] + c * ck.loop[2], ck.loop[3], ck.size, &lo, &hi);
          }
          if (k < r.n_test) {
            const LeanParams::Check& ck = r.test[k];
            const int now = test[k] + a * ck.loop[0] + b * ck.loop[1] + c * ck.loop[2];
            inside = inside && now + r.reach_low[k] >= 0 && now + r.reach_high[k] < ck.size;
          }
        }
        if (lo >= hi) continue;
        const float* qm = ms + (a * sm.loop[0] + b * sm.loop[1] + c * sm.loop[2] + lo * st_m);
        const float* qf = fs + (a * sf.loop[0] + b * sf.loop[1] + c * sf.loop[2] + lo * st_f);
        if (inside && st_m == sm.out[along]) {
          // the next term's elements are this one's moved on by one neighbour: one new element per term
          RunVec<W> u[kRun];
#pragma unroll
          for (int x = 1; x < kRun; ++x) u[x] = run_load<W, ONE_M>(qm + (x - 1) * step_x);
          qm += (kRun - 1) * step_x;
#pragma unroll 3
          for (int j = lo; j < hi; ++j) {
            const RunVec<W> f = run_load<W, ONE_F>(qf);
#pragma unroll
            for (int x = 1; x < kRun; ++x) u[x - 1] = u[x];
            u[kRun - 1] = run_load<W, ONE_M>(qm);
            qm += st_m;
            qf += st_f;
#pragma unroll
            for (int x = 0; x < kRun; ++x) add_products(acc[x], u[x], f);
          }
        } else if (inside) {
#pragma unroll(W == 1 ? 3 : 2)
          for (int j = lo; j < hi; ++j) {
            const RunVec<W> f = run_load<W, ONE_F>(qf);
            RunVec<W> u[kRun];
#pragma unroll
            for (int x = 0; x < kRun; ++x) u[x] = run_load<W, ONE_M>(qm + x * step_x);
            qm += st_m;
            qf += st_f;
#pragma unroll
            for (int x = 0; x < kRun; ++x) add_products(acc[x], u[x], f);
          }
        } else {
#pragma unroll 1
          for (int j = lo; j < hi; ++j) {
            const RunVec<W> f = run_load<W, ONE_F>(qf);
#pragma unroll
            for (int x = 0; x < kRun; ++x) {
              bool ok = x < n;
#pragma unroll
              for (int k = 0; k < NT; ++k) {
                if (k < r.n_test) {
                  const LeanParams::Check& ck = r.test[k];
                  const int at = test[k] + a * ck.loop[0] + b * ck.loop[1] + c * ck.loop[2] + x * ck.out[along] + j * ck.loop[3];
                  ok = ok && static_cast<unsigned>(at) < static_cast<unsigned>(ck.size);
                }
              }
              if (ok) add_products(acc[x], run_load<W, ONE_M>(qm + x * step_x), f);
            }
            qm += st_m;
            qf += st_f;
          }
        }
      }
    }
  }
  float* o = static_cast<float*>(p.outp) + out;
#pragma unroll
  for (int x = 0; x < kRun; ++x) {
    if (x < n) *reinterpret_cast<RunVec<W>*>(o + x * p.out_stride[along]) = acc[x];
  }
}

// The same for any element types, one element per thread, values in the class of the output type.
template <class T>
__global__ void __launch_bounds__(256) contract_lean_kernel(const __grid_constant__ LeanParams p) {
  const long long t = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (t >= p.elems) return;
  const LeanPlace w = lean_place(p, static_cast<int>(t));
  const int odt = p.out_dtype;
  T acc = p.has_init ? narrow<T>(load_as<T>(p.initp, p.init_dtype, w.init), odt) : agg_identity<T>(p.agg, odt);
  for (int a = 0; a < p.loop[0]; ++a) {
    for (int b = 0; b < p.loop[1]; ++b) {
      for (int c = 0; c < p.loop[2]; ++c) {
        int lo = 0, hi = p.loop[3];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < p.n_check) {
            const LeanParams::Check& ck = p.check[k];
            lean_clip(w.check[k] + a * ck.loop[0] + b * ck.loop[1] + c * ck.loop[2], ck.loop[3], ck.size, &lo, &hi);
          }
        }
        int o0 = w.src[0] + a * p.src[0].loop[0] + b * p.src[0].loop[1] + c * p.src[0].loop[2] + lo * p.src[0].loop[3];
        int o1 = w.src[1] + a * p.src[1].loop[0] + b * p.src[1].loop[1] + c * p.src[1].loop[2] + lo * p.src[1].loop[3];
        for (int x = lo; x < hi; ++x) {
          T v = load_as<T>(p.srcp[0], p.src[0].dtype, o0);
          if (p.n_src > 1) {
            const T u = load_as<T>(p.srcp[1], p.src[1].dtype, o1);
            v = p.combo == PMLB_COMBO_MUL ? rounded_mul(v, u) : rounded_add(v, u);
          }
          v = narrow<T>(v, odt);
          o0 += p.src[0].loop[3];
          o1 += p.src[1].loop[3];
          switch (p.agg) {
            case PMLB_AGG_SUM: acc = narrow<T>(rounded_add(acc, v), odt); break;
            case PMLB_AGG_PROD: acc = narrow<T>(rounded_mul(acc, v), odt); break;
            case PMLB_AGG_MAX: acc = (acc > v) ? acc : v; break;
            case PMLB_AGG_MIN: acc = (acc < v) ? acc : v; break;
            default: acc = v; break;
          }
        }
      }
    }
  }
  store_as<T>(p.outp, odt, w.out, acc);
}

// ------------------------------------------------------------------ eltwise

template <class T>
__device__ __forceinline__ T ew_apply(int op, T a, T b, T c, bool a_nz) {
  constexpr bool is_float = static_cast<T>(0.5) != T(0);
  switch (op) {
    case kEwIdent: return a;
    case kEwAdd: return a + b;
    case kEwSub: return a - b;
    case kEwMul: return a * b;
    case kEwDiv:
      if constexpr (is_float) return a / b;
      else return b == T(0) ? T(0) : a / b;
    case kEwMod:
      if constexpr (is_float) return static_cast<T>(fmod(static_cast<double>(a), static_cast<double>(b)));
      else return b == T(0) ? T(0) : a % b;
    case kEwMax: return (a > b) ? a : b;
    case kEwMin: return (a < b) ? a : b;
    case kEwNeg: return T(0) - a;
    case kEwAbs: return a < T(0) ? T(0) - a : a;
    case kEwRelu: return a < T(0) ? T(0) : a;
    case kEwSign: return a > T(0) ? T(1) : (a < T(0) ? T(0) - T(1) : T(0));
    case kEwSelect: return a_nz ? b : c;
    case kEwCmpEq: return a == b ? T(1) : T(0);
    case kEwCmpNe: return a != b ? T(1) : T(0);
    case kEwCmpLt: return a < b ? T(1) : T(0);
    case kEwCmpLe: return a <= b ? T(1) : T(0);
    case kEwCmpGt: return a > b ? T(1) : T(0);
    case kEwCmpGe: return a >= b ? T(1) : T(0);
    case kEwLogicalAnd: return (a != T(0) && b != T(0)) ? T(1) : T(0);
    case kEwLogicalOr: return (a != T(0) || b != T(0)) ? T(1) : T(0);
    case kEwLogicalXor: return ((a != T(0)) != (b != T(0))) ? T(1) : T(0);
    case kEwLogicalNot: return a == T(0) ? T(1) : T(0);
    default: break;
  }
  if constexpr (is_float) {
    const double x = static_cast<double>(a);
    const double y = static_cast<double>(b);
    switch (op) {
      case kEwExp: return static_cast<T>(exp(x));
      case kEwLog: return static_cast<T>(log(x));
      case kEwSqrt: return static_cast<T>(sqrt(x));
      case kEwRsqrt: return static_cast<T>(1.0 / sqrt(x));
      case kEwTanh: return static_cast<T>(tanh(x));
      case kEwSigmoid: return static_cast<T>(1.0 / (1.0 + exp(-x)));
      case kEwSin: return static_cast<T>(sin(x));
      case kEwCos: return static_cast<T>(cos(x));
      case kEwTan: return static_cast<T>(tan(x));
      case kEwSinh: return static_cast<T>(sinh(x));
      case kEwCosh: return static_cast<T>(cosh(x));
      case kEwAsin: return static_cast<T>(asin(x));
      case kEwAcos: return static_cast<T>(acos(x));
      case kEwAtan: return static_cast<T>(atan(x));
      case kEwAsinh: return static_cast<T>(asinh(x));
      case kEwAcosh: return static_cast<T>(acosh(x));
      case kEwAtanh: return static_cast<T>(atanh(x));
      case kEwErf: return static_cast<T>(erf(x));
      case kEwPow: return static_cast<T>(pow(x, y));
      case kEwFloor: return static_cast<T>(floor(x));
      case kEwCeil: return static_cast<T>(ceil(x));
      case kEwRound: return static_cast<T>(round(x));
      default: return a;
    }
  } else {
    switch (op) {
      case kEwBitAnd: return a & b;
      case kEwBitOr: return a | b;
      case kEwBitXor: return a ^ b;
      case kEwBitNot: return ~a;
      case kEwBitShl: return (b < T(0) || b >= T(64)) ? T(0) : static_cast<T>(a << b);
      case kEwBitShr: return (b < T(0) || b >= T(64)) ? T(0) : static_cast<T>(a >> b);
      case kEwPow: {
        T r = 1;
        for (T i = 0; i < b; ++i) r *= a;
        return r;
      }
      case kEwFloor:
      case kEwCeil:
      case kEwRound: return a;
      default: return a;
    }
  }
}

// `T` is the class the operation is evaluated in (chosen from the operand types for
// comparisons, from the result type otherwise); `arith_dtype` is the element type results
// are rounded / wrapped to before the final conversion to the output type.
template <class T>
__device__ __forceinline__ void eltwise_one(const EltwiseParams& p, long long e, const long long (&off)[3]) {
  T a = T(0), b = T(0), c = T(0);
  bool a_nz = false;
  if (p.op == kEwSelect) {
    // the condition keeps its own type; the branches are read in the result class
    a_nz = load_as<double>(p.in[0], p.in_dtype[0], off[0]) != 0.0;
    b = narrow<T>(load_as<T>(p.in[1], p.in_dtype[1], off[1]), p.arith_dtype);
    c = narrow<T>(load_as<T>(p.in[2], p.in_dtype[2], off[2]), p.arith_dtype);
  } else {
    a = load_as<T>(p.in[0], p.in_dtype[0], off[0]);
    if (p.n_in > 1) b = load_as<T>(p.in[1], p.in_dtype[1], off[1]);
    if (p.n_in > 2) c = load_as<T>(p.in[2], p.in_dtype[2], off[2]);
    if (p.narrow_inputs) {
      a = narrow<T>(a, p.arith_dtype);
      b = narrow<T>(b, p.arith_dtype);
      c = narrow<T>(c, p.arith_dtype);
    }
  }
  T r = ew_apply<T>(p.op, a, b, c, a_nz);
  if (p.narrow_result) r = narrow<T>(r, p.arith_dtype);
  store_as<T>(p.out, p.out_dtype, e, r);
}

template <class T>
__global__ void __launch_bounds__(256) eltwise_kernel(const __grid_constant__ EltwiseParams p) {
  dependent_entry();
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= p.elems) return;
  long long rem = e;
  long long off[3] = {0, 0, 0};
  for (int d = p.rank - 1; d >= 0; --d) {
    const long long c = rem % p.sizes[d];
    rem /= p.sizes[d];
    off[0] += c * p.in_strides[0][d];
    off[1] += c * p.in_strides[1][d];
    off[2] += c * p.in_strides[2][d];
  }
  eltwise_one<T>(p, e, off);
}

// Every operand as dense as the result or one value for all of it, any element types: no index arithmetic, four
// elements per thread a grid apart (`one_value` has bit k set if operand k is a single value).
template <class T>
__global__ void __launch_bounds__(256) eltwise_dense_kernel(const __grid_constant__ EltwiseParams p, int one_value,
                                                            long long threads) {
  dependent_entry();
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= threads) return;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const long long e = t + u * threads;
    if (e >= p.elems) return;
    const long long off[3] = {(one_value & 1) ? 0 : e, (one_value & 2) ? 0 : e, (one_value & 4) ? 0 : e};
    eltwise_one<T>(p, e, off);
  }
}

// The common case of the kernel above -- f32 in and out, every operand either as dense as the result or one value
// for all of it -- without the per-element index arithmetic: eight elements per thread as two 16-byte pieces a grid
// apart, all loads before the arithmetic.  The arithmetic is the same function, so the results are the same bits.
struct DenseF32 {
  const float* in[3];
  int scalar[3];   // operand k: 0 dense, 1 one value, 2 repeats every `period` quads (a bias along the trailing dims),
                   // 3 one value per `period` quads (a column along the leading dims)
  long long period[3];
  float* out;
  long long quads;  // elements / 4
  int op, n_in;
};

__global__ void __launch_bounds__(256) eltwise_f32_dense_kernel(const DenseF32 p, long long threads) {
  dependent_entry();
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= threads) return;
  float4 v[2][3];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    long long q = t + u * threads;
    if (q >= p.quads) q = p.quads - 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (k >= p.n_in) {
        v[u][k] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else if (p.scalar[k] == 1) {
        const float s = p.in[k][0];
        v[u][k] = make_float4(s, s, s, s);
      } else if (p.scalar[k] == 2) {
        v[u][k] = reinterpret_cast<const float4*>(p.in[k])[q % p.period[k]];
      } else if (p.scalar[k] == 3) {
        const float s = p.in[k][q / p.period[k]];
        v[u][k] = make_float4(s, s, s, s);
      } else {
        v[u][k] = reinterpret_cast<const float4*>(p.in[k])[q];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const long long q = t + u * threads;
    if (q >= p.quads) continue;
    float4 r;
    r.x = ew_apply<float>(p.op, v[u][0].x, v[u][1].x, v[u][2].x, false);
    r.y = ew_apply<float>(p.op, v[u][0].y, v[u][1].y, v[u][2].y, false);
    r.z = ew_apply<float>(p.op, v[u][0].z, v[u][1].z, v[u][2].z, false);
    r.w = ew_apply<float>(p.op, v[u][0].w, v[u][1].w, v[u][2].w, false);
    reinterpret_cast<float4*>(p.out)[q] = r;
  }
}

// The dense form for f16 / bf16 in and out: eight elements per 16-byte piece, the operation evaluated in f32 and
// rounded to the 16-bit type as the general kernel does (operands of that type need no rounding).
template <class S>
struct Dense16 {
  const S* in[3];
  int scalar[3];
  S* out;
  long long octets;
  int op, n_in, dtype;
};

__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
template <class S> __device__ __forceinline__ S shorten(float v);
template <> __device__ __forceinline__ __half shorten<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 shorten<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <class S>
__global__ void __launch_bounds__(256) eltwise_16bit_dense_kernel(const Dense16<S> p) {
  dependent_entry();
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= p.octets) return;
  struct alignas(16) Vec { S v[8]; };
  Vec a[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k >= p.n_in) {
#pragma unroll
      for (int i = 0; i < 8; ++i) a[k].v[i] = shorten<S>(0.f);
    } else if (p.scalar[k]) {
      const S s = p.in[k][0];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[k].v[i] = s;
    } else {
      a[k] = reinterpret_cast<const Vec*>(p.in[k])[t];
    }
  }
  Vec r;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = ew_apply<float>(p.op, widen(a[0].v[i]), widen(a[1].v[i]), widen(a[2].v[i]), false);
    r.v[i] = shorten<S>(narrow<float>(x, p.dtype));
  }
  reinterpret_cast<Vec*>(p.out)[t] = r;
}

// Dense casts between f32 and the two 16-bit float types (round to nearest even, as the general kernel's store does):
// eight elements per thread, 16- and 32-byte accesses.
template <class In, class Out>
__device__ __forceinline__ Out convert_one(In v);
template <> __device__ __forceinline__ float convert_one<__half, float>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float convert_one<__nv_bfloat16, float>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ __half convert_one<float, __half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 convert_one<float, __nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <class In, class Out>
__global__ void __launch_bounds__(256) convert_dense_kernel(const In* __restrict__ in, Out* __restrict__ out, long long octets) {
  dependent_entry();
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= octets) return;
  struct alignas(sizeof(In) * 8) InVec { In v[8]; };
  struct alignas(sizeof(Out) * 8) OutVec { Out v[8]; };
  const InVec a = reinterpret_cast<const InVec*>(in)[t];
  OutVec r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = convert_one<In, Out>(a.v[i]);
  reinterpret_cast<OutVec*>(out)[t] = r;
}

template <class T>
__global__ void __launch_bounds__(256) fill_kernel(void* out, int dtype, long long n, T value) {
  dependent_entry();
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e < n) store_as<T>(out, dtype, e, value);
}

unsigned grid_for(long long elems) { return static_cast<unsigned>((elems + 255) / 256); }

}  // namespace

int dtype_class(int dtype) {
  switch (dtype) {
    case PMLB_F16:
    case PMLB_BF16:
    case PMLB_F32: return kClassF32;
    case PMLB_F64: return kClassF64;
    case PMLB_BOOL:
    case PMLB_U8:
    case PMLB_U16:
    case PMLB_U32:
    case PMLB_U64: return kClassU64;
    case PMLB_I8:
    case PMLB_I16:
    case PMLB_I32:
    case PMLB_I64: return kClassI64;
    default: return -1;
  }
}

cudaError_t launch_contract(const GenericParams& p, cudaStream_t stream) {
  if (p.out_elems <= 0) return cudaSuccess;
  const unsigned grid = grid_for(p.out_elems);
  switch (dtype_class(p.out.dtype)) {
    case kClassF32: contract_kernel<float><<<grid, 256, 0, stream>>>(p); break;
    case kClassF64: contract_kernel<double><<<grid, 256, 0, stream>>>(p); break;
    case kClassI64: contract_kernel<long long><<<grid, 256, 0, stream>>>(p); break;
    case kClassU64: contract_kernel<unsigned long long><<<grid, 256, 0, stream>>>(p); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

namespace {
// Whether a problem goes kRun neighbours per thread, `width` elements of the last dim each.
bool lean_run_form(const LeanParams& p, int width, LeanRun* r) {
  if (p.one_order || p.rank < 2 || p.n_src != 2 || p.has_init || p.agg != PMLB_AGG_SUM || p.combo != PMLB_COMBO_MUL) return false;
  const int along = p.rank - 2;
  const bool move0 = p.src[0].out[along] != 0, move1 = p.src[1].out[along] != 0;
  if (move0 == move1) return false;
  r->moving = move0 ? 0 : 1;
  r->groups = p.size[p.rank - 1] / width;
  r->runs = (p.size[along] + kRun - 1) / kRun;
  r->threads = p.elems / width / p.size[along] * r->runs;
  if (r->threads < kRunThreads) return false;
  for (int k = 0; k < p.n_check; ++k) {
    const LeanParams::Check& c = p.check[k];
    // the kernel adds a run's and a loop's reach to a bounds value in 32 bits
    const long long far_x = (kRun - 1ll) * c.out[along], far_j = (p.loop[3] - 1ll) * c.loop[3];
    if (std::abs(far_x) + std::abs(far_j) > (1 << 29)) return false;
    if (c.out[along] == 0) {
      r->clip[r->n_clip++] = c;
    } else {
      r->reach_low[r->n_test] = static_cast<int>(std::min(far_x, 0ll) + std::min(far_j, 0ll));
      r->reach_high[r->n_test] = static_cast<int>(std::max(far_x, 0ll) + std::max(far_j, 0ll));
      r->test[r->n_test++] = c;
    }
  }
  r->fd_groups = make_fastdiv(static_cast<uint32_t>(r->groups));
  r->fd_runs = make_fastdiv(static_cast<uint32_t>(r->runs));
  return true;
}

template <int W, bool ONE_M, bool ONE_F>
void launch_run(const LeanParams& p, const LeanRun& r, cudaStream_t stream) {
  const unsigned grid = static_cast<unsigned>((r.threads + kRunBlock - 1) / kRunBlock);
  if (r.n_clip <= 1 && r.n_test <= 1) {
    contract_lean_run_kernel<W, ONE_M, ONE_F, 1><<<grid, kRunBlock, 0, stream>>>(p, r);
  } else {
    contract_lean_run_kernel<W, ONE_M, ONE_F, 4><<<grid, kRunBlock, 0, stream>>>(p, r);
  }
}
}  // namespace

cudaError_t launch_contract_lean(const LeanParams& p, cudaStream_t stream) {
  bool f32 = p.out_dtype == PMLB_F32 && (!p.has_init || p.init_dtype == PMLB_F32);
  for (int s = 0; s < p.n_src; ++s) f32 = f32 && p.src[s].dtype == PMLB_F32;
  if (f32) {
    // four elements per thread?
    const int last = p.rank - 1;
    bool quads = p.rank > 0 && p.size[last] % 4 == 0 && p.out_stride[last] == 1 && reinterpret_cast<uintptr_t>(p.outp) % 16 == 0;
    for (int d = 0; d < last && quads; ++d) quads = p.out_stride[d] % 4 == 0;
    for (int s = 0; s < p.n_src && quads; ++s) {
      const LeanParams::Source& a = p.src[s];
      if (a.out[last] == 0) continue;
      quads = a.out[last] == 1 && a.base % 4 == 0 && reinterpret_cast<uintptr_t>(p.srcp[s]) % 16 == 0;
      for (int d = 0; d < last; ++d) quads = quads && a.out[d] % 4 == 0;
      for (int j = 0; j < 4; ++j) quads = quads && (p.loop[j] == 1 || a.loop[j] % 4 == 0);
    }
    for (int k = 0; k < p.n_check && quads; ++k) quads = p.check[k].out[last] == 0;
    LeanRun run{};
    if (lean_run_form(p, quads ? 4 : 1, &run)) {
      const bool one_m = quads && p.src[run.moving].out[last] == 0, one_f = quads && p.src[1 - run.moving].out[last] == 0;
      if (!quads) launch_run<1, false, false>(p, run, stream);
      else if (one_m && one_f) launch_run<4, true, true>(p, run, stream);
      else if (one_m) launch_run<4, true, false>(p, run, stream);
      else if (one_f) launch_run<4, false, true>(p, run, stream);
      else launch_run<4, false, false>(p, run, stream);
    } else if (quads) {
      contract_lean_f32_kernel<4><<<grid_for(p.elems / 4), 256, 0, stream>>>(p);
    } else {
      contract_lean_f32_kernel<1><<<grid_for(p.elems), 256, 0, stream>>>(p);
    }
    return cudaGetLastError();
  }
  const unsigned grid = grid_for(p.elems);
  switch (dtype_class(p.out_dtype)) {
    case kClassF32: contract_lean_kernel<float><<<grid, 256, 0, stream>>>(p); break;
    case kClassF64: contract_lean_kernel<double><<<grid, 256, 0, stream>>>(p); break;
    case kClassI64: contract_lean_kernel<long long><<<grid, 256, 0, stream>>>(p); break;
    case kClassU64: contract_lean_kernel<unsigned long long><<<grid, 256, 0, stream>>>(p); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

namespace {
// Fills `d` if the operation takes the dense f32 form: f32 throughout, not a select (its condition has a type of its
// own), a multiple of four elements, 16-byte aligned buffers, and operands that are dense like the result or a single
// value.
bool dense_f32_form(const EltwiseParams& p, DenseF32* d) {
  if (p.compute_class != kClassF32 || p.out_dtype != PMLB_F32 || p.arith_dtype != PMLB_F32 || p.op == kEwSelect) return false;
  if (p.elems % 4 != 0 || reinterpret_cast<uintptr_t>(p.out) % 16 != 0) return false;
  long long dense[PMLB_MAX_RANK];
  long long stride = 1;
  for (int dd = p.rank - 1; dd >= 0; --dd) {
    dense[dd] = stride;
    stride *= p.sizes[dd];
  }
  for (int k = 0; k < p.n_in; ++k) {
    if (p.in_dtype[k] != PMLB_F32) return false;
    bool as_result = true, one_value = true;
    for (int dd = 0; dd < p.rank; ++dd) {
      if (p.sizes[dd] == 1) continue;
      if (p.in_strides[k][dd] != dense[dd]) as_result = false;
      if (p.in_strides[k][dd] != 0) one_value = false;
    }
    int mode = as_result ? 0 : (one_value ? 1 : -1);
    long long period = 0;
    if (mode < 0) {
      // dense over the trailing dims and repeated over the leading ones (a bias), or one value per run of the
      // trailing dims (a column)?
      int split = -1;   // first dim of the trailing part
      bool bias = true, column = true;
      for (int dd = 0; dd < p.rank; ++dd) {
        if (p.sizes[dd] == 1) continue;
        if (p.in_strides[k][dd] != 0 && split < 0) split = dd;
      }
      // bias: stride 0 before `split`, dense strides from `split` on
      for (int dd = 0; dd < p.rank && split >= 0; ++dd) {
        if (p.sizes[dd] == 1) continue;
        if (dd < split ? p.in_strides[k][dd] != 0 : p.in_strides[k][dd] != dense[dd]) bias = false;
      }
      if (split >= 0 && bias) {
        period = dense[split] * p.sizes[split];          // elements of the trailing part
        if (period % 4 == 0) mode = 2;
      }
      if (mode < 0) {
        // column: non-zero strides on a leading part only, dense within that part; zero on the trailing part
        int last = -1;
        for (int dd = 0; dd < p.rank; ++dd) {
          if (p.sizes[dd] != 1 && p.in_strides[k][dd] != 0) last = dd;
        }
        long long run = last >= 0 ? dense[last] : 0;     // elements of the trailing part behind `last`
        for (int dd = 0; dd < p.rank && last >= 0; ++dd) {
          if (p.sizes[dd] == 1) continue;
          if (dd <= last ? p.in_strides[k][dd] * run != dense[dd] : p.in_strides[k][dd] != 0) column = false;
        }
        if (last >= 0 && column && run % 4 == 0) {
          period = run;
          mode = 3;
        }
      }
      if (mode < 0) return false;
      period /= 4;
    }
    if ((mode == 0 || mode == 2) && reinterpret_cast<uintptr_t>(p.in[k]) % 16 != 0) return false;
    d->in[k] = static_cast<const float*>(p.in[k]);
    d->scalar[k] = mode;
    d->period[k] = period;
  }
  d->out = static_cast<float*>(p.out);
  d->quads = p.elems / 4;
  d->op = p.op;
  d->n_in = p.n_in;
  return true;
}
}  // namespace

namespace {
// A cast between f32 and f16 / bf16 of a dense operand, eight elements at a time; false if the operation is not one.
bool launch_dense_convert(const EltwiseParams& p, cudaStream_t stream) {
  if (p.op != kEwIdent || p.n_in != 1 || p.elems % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(p.in[0]) | reinterpret_cast<uintptr_t>(p.out)) % 32 != 0) return false;
  long long stride = 1;
  for (int dd = p.rank - 1; dd >= 0; --dd) {
    if (p.sizes[dd] != 1 && p.in_strides[0][dd] != stride) return false;
    stride *= p.sizes[dd];
  }
  const long long octets = p.elems / 8;
  const unsigned grid = grid_for(octets);
  const int from = p.in_dtype[0], to = p.out_dtype;
  if (from == PMLB_F32 && to == PMLB_F16) {
    launch_dependent(convert_dense_kernel<float, __half>, grid, 256, stream, static_cast<const float*>(p.in[0]), static_cast<__half*>(p.out), octets);
  } else if (from == PMLB_F32 && to == PMLB_BF16) {
    launch_dependent(convert_dense_kernel<float, __nv_bfloat16>, grid, 256, stream, static_cast<const float*>(p.in[0]),
                                                                         static_cast<__nv_bfloat16*>(p.out), octets);
  } else if (from == PMLB_F16 && to == PMLB_F32) {
    launch_dependent(convert_dense_kernel<__half, float>, grid, 256, stream, static_cast<const __half*>(p.in[0]), static_cast<float*>(p.out), octets);
  } else if (from == PMLB_BF16 && to == PMLB_F32) {
    launch_dependent(convert_dense_kernel<__nv_bfloat16, float>, grid, 256, stream, static_cast<const __nv_bfloat16*>(p.in[0]),
                                                                         static_cast<float*>(p.out), octets);
  } else {
    return false;
  }
  return true;
}
}  // namespace

namespace {
template <class S>
bool launch_dense_16bit(const EltwiseParams& p, int dtype, cudaStream_t stream) {
  if (p.compute_class != kClassF32 || p.out_dtype != dtype || p.arith_dtype != dtype || p.op == kEwSelect) return false;
  if (p.elems % 8 != 0 || reinterpret_cast<uintptr_t>(p.out) % 16 != 0) return false;
  long long dense[PMLB_MAX_RANK];
  long long stride = 1;
  for (int dd = p.rank - 1; dd >= 0; --dd) {
    dense[dd] = stride;
    stride *= p.sizes[dd];
  }
  Dense16<S> d{};
  for (int k = 0; k < p.n_in; ++k) {
    if (p.in_dtype[k] != dtype) return false;
    bool as_result = true, one_value = true;
    for (int dd = 0; dd < p.rank; ++dd) {
      if (p.sizes[dd] == 1) continue;
      if (p.in_strides[k][dd] != dense[dd]) as_result = false;
      if (p.in_strides[k][dd] != 0) one_value = false;
    }
    if (!as_result && !one_value) return false;
    if (as_result && reinterpret_cast<uintptr_t>(p.in[k]) % 16 != 0) return false;
    d.in[k] = static_cast<const S*>(p.in[k]);
    d.scalar[k] = as_result ? 0 : 1;
  }
  d.out = static_cast<S*>(p.out);
  d.octets = p.elems / 8;
  d.op = p.op;
  d.n_in = p.n_in;
  d.dtype = dtype;
  launch_dependent(eltwise_16bit_dense_kernel<S>, grid_for(d.octets), 256, stream, d);
  return true;
}
}  // namespace

cudaError_t launch_eltwise(const EltwiseParams& p, cudaStream_t stream) {
  if (p.elems <= 0) return cudaSuccess;
  if (launch_dense_convert(p, stream)) return cudaGetLastError();
  if (launch_dense_16bit<__half>(p, PMLB_F16, stream) || launch_dense_16bit<__nv_bfloat16>(p, PMLB_BF16, stream)) {
    return cudaGetLastError();
  }
  DenseF32 dense{};
  if (dense_f32_form(p, &dense)) {
    const long long threads = (dense.quads + 1) / 2;
    launch_dependent(eltwise_f32_dense_kernel, grid_for(threads), 256, stream, dense, threads);
    return cudaGetLastError();
  }
  // every operand dense like the result or a single value?
  {
    long long dense_stride[PMLB_MAX_RANK];
    long long stride = 1;
    for (int dd = p.rank - 1; dd >= 0; --dd) {
      dense_stride[dd] = stride;
      stride *= p.sizes[dd];
    }
    int one_value = 0;
    bool all = true;
    for (int k = 0; k < p.n_in && all; ++k) {
      bool as_result = true, single = true;
      for (int dd = 0; dd < p.rank; ++dd) {
        if (p.sizes[dd] == 1) continue;
        if (p.in_strides[k][dd] != dense_stride[dd]) as_result = false;
        if (p.in_strides[k][dd] != 0) single = false;
      }
      if (!as_result && !single) all = false;
      if (!as_result && single) one_value |= 1 << k;
    }
    if (all) {
      const long long threads = (p.elems + 3) / 4;
      const unsigned g4 = grid_for(threads);
      switch (p.compute_class) {
        case kClassF32: launch_dependent(eltwise_dense_kernel<float>, g4, 256, stream, p, one_value, threads); break;
        case kClassF64: launch_dependent(eltwise_dense_kernel<double>, g4, 256, stream, p, one_value, threads); break;
        case kClassI64: launch_dependent(eltwise_dense_kernel<long long>, g4, 256, stream, p, one_value, threads); break;
        case kClassU64: launch_dependent(eltwise_dense_kernel<unsigned long long>, g4, 256, stream, p, one_value, threads); break;
        default: return cudaErrorInvalidValue;
      }
      return cudaGetLastError();
    }
  }
  const unsigned grid = grid_for(p.elems);
  switch (p.compute_class) {
    case kClassF32: launch_dependent(eltwise_kernel<float>, grid, 256, stream, p); break;
    case kClassF64: launch_dependent(eltwise_kernel<double>, grid, 256, stream, p); break;
    case kClassI64: launch_dependent(eltwise_kernel<long long>, grid, 256, stream, p); break;
    case kClassU64: launch_dependent(eltwise_kernel<unsigned long long>, grid, 256, stream, p); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_fill_f32(float* out, long long n, float value, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  launch_dependent(fill_kernel<float>, grid_for(n), 256, stream, out, PMLB_F32, n, value);
  return cudaGetLastError();
}

}  // namespace pmlb
