// Shared machinery of the all-pairs Gaussian kernel sums (sm_100a).
//
// Every hot operator of the point-set path is a map-reduce over (target k, source l) pairs:
//     out_k = epilogue_k( sum_l pair(target_k, source_l) ).
// The pair loop is FP32-pipe / MUFU bound (arithmetic intensity >> 100 flop/byte), so the design is an N-body
// tiling: a CTA owns TPB*RT targets held in registers (RT per thread) and streams tiles of TPB sources through
// shared memory (all threads of a warp read the same source record: broadcast LDS.128). The (target block, source
// tile) units are split evenly over exactly one resident wave of CTAs (stream-K style, see SKPlan), so every
// problem size keeps all 148 SMs equally busy.
//
// FP32 path: the pair arithmetic runs on Blackwell's packed FP32 instructions (fma/add/sub/mul .f32x2), halving the
// issue slots of the FP32 work. In the ordered sums of this file an instruction evaluates the same source against TWO
// targets of the thread; source fields are stored duplicated ((f, f) pairs) in shared memory so that a 16-byte LDS
// yields two ready-to-use packed operands. (The symmetric sums of pairs_sym.cuh evaluate two sources against the same
// target.) Coordinates are relative to an origin, the caller's or the target block's own (segment_origin), and
// pre-scaled by s = sqrt(log2(e)/2)/sigma so that exp(-|y-x|^2/(2 sigma^2)) = 2^-(|y'-x'|^2), one `ex2.approx.ftz`
// (MUFU) per pair. Each tile is summed in plain FP32; tile sums are merged into a (hi, lo) pair by a two-sum
// (compensated accumulation across tiles). Chunk partials are reduced in FP64, in fixed order, by the epilogue
// kernel, which applies the per-target constants and writes float64 outputs (and, for shooting steps, the
// float64 Euler update of the state).
// Ops whose sum needs no coordinate differences (K a, the surface energies) run pairs_kernel_x instead: the
// squared distance expanded about the centre of each target block, three packed FMAs per pair (see there).
// FP64 path (the faithful baseline): the same pair functors instantiated with double, exp2_neg() and FP64 sums.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#ifndef LDDMM_MIN_CTAS
#define LDDMM_MIN_CTAS 1  // minimum resident CTAs per SM requested from ptxas (caps registers when > 1)
#endif
// per-op minimum resident CTAs (1: no register cap beyond the op's needs)
#ifndef LDDMM_SOFWD_MIN_CTAS
#define LDDMM_SOFWD_MIN_CTAS 4
#endif
#ifndef LDDMM_SOBWD_MIN_CTAS
#define LDDMM_SOBWD_MIN_CTAS 1  // at 4 targets per thread (LDDMM_RT_ADJOINT) no cap: 254 registers, 2 CTAs per SM
#endif
#ifndef LDDMM_SOBWD_SYM_MIN_CTAS
#define LDDMM_SOBWD_SYM_MIN_CTAS 2  // the symmetric adjoint step (pairs_kernel_sym)
#endif
#ifndef LDDMM_SOFWD_SYM_MIN_CTAS
#define LDDMM_SOFWD_SYM_MIN_CTAS 3  // the symmetric forward step (pairs_kernel_sym) up to 4 targets per thread
#endif
#ifndef LDDMM_KSYM_MIN_CTAS
#define LDDMM_KSYM_MIN_CTAS 2  // the symmetric K(x, x) a (pairs_kernel_symx)
#endif
#ifndef LDDMM_FOBWD_SYM_MIN_CTAS
#define LDDMM_FOBWD_SYM_MIN_CTAS 2  // the symmetric first-order adjoint step (pairs_kernel_sym)
#endif
#ifndef LDDMM_FOBWD_MIN_CTAS
#define LDDMM_FOBWD_MIN_CTAS 1
#endif
#ifndef LDDMM_SURFGRAD_MIN_CTAS
#define LDDMM_SURFGRAD_MIN_CTAS 1
#endif
#ifndef LDDMM_COMP_SMEM
#define LDDMM_COMP_SMEM 1  // 0: keep every op's compensated (hi, lo) sums in registers
#endif
#ifndef LDDMM_CULL
#define LDDMM_CULL 1  // 0: no exact culling of far tile pairs (no box pre-pass)
#endif
#ifndef LDDMM_EXPAND
#define LDDMM_EXPAND 1  // 0: the Gaussian sums of ops with an expanded-distance form use the difference form
#endif
#ifndef LDDMM_SOFWD_EXPAND
#define LDDMM_SOFWD_EXPAND 1  // 0: the second-order forward step keeps the difference form
#endif
#ifndef LDDMM_SURFGRAD_EXPAND
#define LDDMM_SURFGRAD_EXPAND 1  // 0: the varifold and measure gradients keep the difference form
#endif
#ifndef LDDMM_SOURCE_UNROLL
#define LDDMM_SOURCE_UNROLL 4  // unroll depth of the per-source loop over a shared-memory tile
#endif

namespace lddmm {

enum Status : int {
  kOk = 0,
  kInvalidArgument = 1,
  kLaunchFailure = 2,
  kNonFinite = 3,
  kWorkspaceTooSmall = 4,
  kCudaError = 5,
  kUnsupported = 6,
};

enum Precision : int { kFP32Compensated = 0, kFP64 = 1 };

constexpr int kSourceUnroll = LDDMM_SOURCE_UNROLL;

// ---------------------------------------------------------------------------------------------------------
// Programmatic dependent launch. Every kernel of a sum starts with chain_wait(), which returns when the previous kernel
// of the stream has completed and its writes are visible; nothing global is read or written before it, so the order is
// that of an ordinary stream. What overlaps is the next kernel's launch with the previous one's drain: 4 us per step
// of two kernels at every size (second-order forward step at 300 / 2,562 / 10,242 points: 18.9 -> 13.5, 19.7 -> 15.5,
// 85.1 -> 80.5 us). A CTA of a split kernel releases its epilogue (chain_go()) when its last tile is done, so that the
// epilogue's blocks are resident when the last partial is written: 0.3-0.4 us per step (2,562 points, forward / adjoint
// / first-order adjoint step: 13.2 -> 12.8, 18.2 -> 17.8, 14.0 -> 13.6 us). The unsplit kernels, whose calls are long
// against that, do not (forward step at 40,962 points 777 -> 810 us with it: the register allocation of the loop).
// No kernel releases its dependents earlier, and an epilogue not at all: the blocks of the next pair kernel would take
// slots while others are still held, and a grid of one or two blocks per SM then lands on half of the SMs (adjoint step
// at 2,562 points: 24.4 us without the attribute, 33.5 with a release at the start of every kernel; forward step 14.8
// -> 16.3 with one in the epilogue).
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... KArgs, class... Args>
inline void launch_chained(void (*kernel)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t stream,
                           Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);  // an error stays for the caller's cudaPeekAtLastError
}

// ---------------------------------------------------------------------------------------------------------
// Packed FP32 pair (two lanes in one 64-bit register pair) and its arithmetic (PTX .f32x2, sm_100a).
// ---------------------------------------------------------------------------------------------------------
struct F2 {
  unsigned long long v;
};

__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void split(F2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2& operator+=(F2& a, F2 b) { return a = a + b; }
// Lane by lane: a sign in front of an operand, not a packed operation.
__device__ __forceinline__ F2 operator-(F2 a) {
  float x, y;
  split(a, x, y);
  return f2(-x, -y);
}

__device__ __forceinline__ float ex2neg(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(-x));
  return y;
}

// 2^-t in FP64 for t >= 0, by Tang's table-driven scheme (P. T. P. Tang, ACM TOMS 15(2), 1989, for exp): t is rounded
// to a multiple of 1/16, t = k/16 - f with |f| <= 1/32, and 2^-t = 2^-m T[j] (1 + f q(f)) with k = 16 m - j, T[j] =
// 2^(j/16) and q the degree-5 Chebyshev interpolant of (2^f - 1)/f on |f| <= 1/32 (1.4e-17 relative). 10 FP64
// instructions (exp() of the CUDA library: as long as ~25 of them, 53 against 22 clocks per warp and scheduler), the
// exponent arithmetic on the integer pipe, one 8-byte shared-memory load: the 16 entries cover the 32 banks once, so
// lanes on different entries never conflict. Results below 2^-1022 are zero; NaN stays NaN.
static __constant__ double kExp2Frac[16] = {
    1.0, 1.0442737824274138, 1.0905077326652577, 1.1387886347566916, 1.189207115002721, 1.241857812073484,
    1.2968395546510096, 1.3542555469368927, 1.4142135623730951, 1.4768261459394993, 1.5422108254079407,
    1.6104903319492543, 1.681792830507429, 1.7562521603732995, 1.8340080864093424, 1.9152065613971474};
__device__ __forceinline__ double* exp2_table() {
  __shared__ double t[16];
  return t;
}
// Fills the kernel's table; a barrier must follow before the first exp2_neg.
__device__ __forceinline__ void exp2_table_fill() {
  if (threadIdx.x < 16) exp2_table()[threadIdx.x] = kExp2Frac[threadIdx.x];
}
__device__ __forceinline__ double exp2_neg(double t) {
  constexpr double kRound = 422212465065984.0;  // 1.5 * 2^48: the low word of t + kRound is t rounded to 1/16
  const double s = t + kRound;
  const int k = __double2loint(s);
  const double f = (s - kRound) - t;
  double q = 0.00015403723980749256;
  q = ::fma(q, f, 0.0013333781576784268);
  q = ::fma(q, f, 0.009618129106919537);
  q = ::fma(q, f, 0.0555041086566393);
  q = ::fma(q, f, 0.24022650695910075);
  q = ::fma(q, f, 0.6931471805599457);
  const double tj = exp2_table()[-k & 15];
  const double ts = __hiloint2double(__double2hiint(tj) - (((k + 15) >> 4) << 20), __double2loint(tj));
  const double e = ::fma(ts, q * f, ts);
  // t in [1022, inf]: zero (high words 0x408ff000 .. 0x7ff00000; a NaN's is above)
  const bool zero = (unsigned)__double2hiint(t) - 0x408ff000u <= 0x7ff00000u - 0x408ff000u;
  return zero ? 0.0 : e;
}

// sqrt(log2(e) / 2): exp(-r^2/(2 sigma^2)) == 2^-(s r)^2 with s = kScale / sigma.
constexpr double kScale = 0.84932180028801904272;

// Value-type traits: V = F2 (two FP32 targets per lane group) or double (one FP64 target).
template <typename V> struct VT;
template <> struct VT<F2> {
  using Scalar = float;
  static constexpr int kLanes = 2;
  using Partial = float2;  // (hi, lo) of the compensated chunk sum
  static __device__ __forceinline__ void setup() {}
  static __device__ __forceinline__ Partial to_partial(double w) {
    const float h = (float)w;
    return make_float2(h, (float)(w - (double)h));
  }
  static __device__ __forceinline__ F2 zero() { return f2(0.f, 0.f); }
  static __device__ __forceinline__ F2 dup(double a) { return f2((float)a, (float)a); }
  static __device__ __forceinline__ F2 pack(double a, double b) { return f2((float)a, (float)b); }
  static __device__ __forceinline__ F2 expneg(F2 r2) {
    float a, b;
    split(r2, a, b);
    return f2(ex2neg(a), ex2neg(b));
  }
  // the sum of a value's lanes
  static __device__ __forceinline__ float hsum(F2 v) {
    float a, b;
    split(v, a, b);
    return a + b;
  }
  static __device__ __forceinline__ double lane(F2 v, int k) {
    float a, b;
    split(v, a, b);
    return k ? (double)b : (double)a;
  }
};
template <> struct VT<double> {
  using Scalar = double;
  static constexpr int kLanes = 1;
  using Partial = double;
  static __device__ __forceinline__ void setup() { exp2_table_fill(); }  // a barrier must follow before expneg
  static __device__ __forceinline__ Partial to_partial(double w) { return w; }
  static __device__ __forceinline__ double zero() { return 0.0; }
  static __device__ __forceinline__ double dup(double a) { return a; }
  static __device__ __forceinline__ double pack(double a, double) { return a; }
  static __device__ __forceinline__ double expneg(double r2) { return exp2_neg(r2); }
  // the sum of a value's lanes
  static __device__ __forceinline__ double hsum(double v) { return v; }
  static __device__ __forceinline__ double lane(double v, int) { return v; }
};

// Compensated accumulator: a tile sum `t` is folded into (hi, lo) by Knuth's two-sum (FP32); plain sum (FP64).
template <typename V> struct Comp;
template <> struct Comp<F2> {
  static constexpr int kWords = 2;  // (hi, lo)
  F2 hi, lo;
  __device__ __forceinline__ void zero() { hi = lo = f2(0.f, 0.f); }
  template <int TPB>
  __device__ __forceinline__ void load(const F2 (*cs)[TPB], int i, int t) { hi = cs[2 * i][t]; lo = cs[2 * i + 1][t]; }
  template <int TPB>
  __device__ __forceinline__ void store(F2 (*cs)[TPB], int i, int t) const { cs[2 * i][t] = hi; cs[2 * i + 1][t] = lo; }
  __device__ __forceinline__ void merge(F2 t) {
    const F2 s = hi + t;
    const F2 bp = s - hi;
    const F2 err = (hi - (s - bp)) + (t - bp);
    hi = s;
    lo = lo + err;
  }
  __device__ __forceinline__ float2 partial(int k) const {
    return make_float2((float)VT<F2>::lane(hi, k), (float)VT<F2>::lane(lo, k));
  }
};
template <> struct Comp<double> {
  static constexpr int kWords = 1;
  double hi;
  __device__ __forceinline__ void zero() { hi = 0.0; }
  template <int TPB>
  __device__ __forceinline__ void load(const double (*cs)[TPB], int i, int t) { hi = cs[i][t]; }
  template <int TPB>
  __device__ __forceinline__ void store(double (*cs)[TPB], int i, int t) const { cs[i][t] = hi; }
  __device__ __forceinline__ void merge(double t) { hi += t; }
  __device__ __forceinline__ double partial(int) const { return hi; }
};

// Ops whose compensated sums stay in registers (few accumulators: measured faster there) declare
// `static constexpr bool kCompInRegisters = true;`.
template <class Op, class = void>
struct CompInRegisters : std::false_type {};
template <class Op>
struct CompInRegisters<Op, std::void_t<decltype(Op::kCompInRegisters)>> : std::bool_constant<Op::kCompInRegisters> {};

__device__ __forceinline__ double partial_value(float2 p) { return (double)p.x + (double)p.y; }
__device__ __forceinline__ double partial_value(double p) { return p; }

__device__ __forceinline__ double fma(double a, double b, double c) { return ::fma(a, b, c); }

// Kernel families (the `kernel` argument of the C ABI): 0 = Gaussian, 16 + q = Laplacian (Matern) of order q <= 4,
// K(r) = P_q(r / sigma) exp(-r / sigma) (base/kernelFunctions_util.py:20-52 lapPol / lapPolDiff / lapPolDiff2).
enum KernelFamily : int { kGauss = 0, kLaplacian0 = 16, kLaplacianMax = 20 };

// Geometry shared by every op: centred, pre-scaled coordinates, and the radial profile of the kernel.
struct Frame {
  double o0, o1, o2;  // origin subtracted before scaling
  int own;            // no origin given: the split kernels' blocks take one of their own (segment_origin)
  double s;           // coordinate scale (Gaussian: kScale / sigma; Laplacian: log2(e) / sigma)
  double kappa;       // 1 / (s sigma^2): turns a scaled difference into (y - x) / sigma^2
  double inv_s2;      // 1 / sigma^2
  int family;         // KernelFamily
  // Laplacian profile in the scaled radius u' = |d|: K0 = P0(u') E, K1 = P1(u') E, K2 = P2(u') E with
  // E = 2^-u' (coefficients rescaled). grad_y K = -K1 kappa d, Hessian = kappa^2 K2 d d^T
  // - K1/sigma^2 I. Row r holds the coefficients of P_r in increasing degree (zeros past the order).
  float lc[3][5];
  double dc[3][5];
};

// Radial factors of one pair: K0 (value), K1 (first-derivative factor), K2 (second-derivative factor). For the
// Gaussian all three are exp(-|d|^2); unused ones are removed by the compiler.
template <typename V>
struct KV {
  V k0, k1, k2;
};

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// kCullR2<V>: a scaled squared distance beyond which every radial factor is exactly zero in the arithmetic of V
// (FP32: ex2.approx.ftz of an argument below -126 flushes to +0; FP64: exp2_neg is zero from 1022 on), with a
// margin for the FP32 rounding of the box test that uses it.
struct Gauss {
  template <typename V>
  static __device__ __forceinline__ KV<V> eval(const Frame&, V r2) {
    const V e = VT<V>::expneg(r2);
    return {e, e, e};
  }
  template <typename V>
  static constexpr float kCullR2 = VT<V>::kLanes == 2 ? 127.0f : 1024.0f;
};

// Orders up to D (the degree of the value's polynomial P0). Two instances: 3 covers the default order and those below,
// 4 the last one; one Horner step less per profile is 8% of a step (order 3, 40,962 points: forward step 1220 -> 1120
// us, adjoint 2217 -> 2156, first-order adjoint 1301 -> 1219, K a 676 -> 628).
template <int D>
struct LaplacianT {
  template <typename V>
  static __device__ __forceinline__ KV<V> eval(const Frame& f, V r2) {
    if constexpr (std::is_same<V, F2>::value)
      return eval_f2(f, r2);
    else
      return eval_f64(f, r2);
  }
  static __device__ __forceinline__ KV<F2> eval_f2(const Frame& f, F2 r2);
  static __device__ __forceinline__ KV<double> eval_f64(const Frame& f, double r2);
  template <typename V>
  static constexpr float kCullR2 = VT<V>::kLanes == 2 ? 127.0f * 127.0f : 1024.0f * 1024.0f;  // the radius u = |d|
};
using Laplacian3 = LaplacianT<3>;
using Laplacian4 = LaplacianT<4>;

// fn(Fam{}) with the profile type of a kernel family.
template <class Fn>
inline auto by_family(int family, Fn fn) {
  if (family == kGauss) return fn(Gauss{});
  if (family <= kLaplacian0 + 3) return fn(Laplacian3{});
  return fn(Laplacian4{});
}

// Axis-aligned box of the scaled coordinates held by a block of threads: per-thread (lo, hi), reduced over the
// block through `red` (6 x warps floats). Every thread ends with the block's box; callers separate reuses of `red`
// by a barrier.
template <int TPB>
__device__ __forceinline__ void block_box(float lo[3], float hi[3], float (*red)[TPB / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      red[c][warp] = lo[c];
      red[3 + c][warp] = hi[c];
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[c] = red[c][0];
    hi[c] = red[3 + c][0];
#pragma unroll
    for (int w = 1; w < TPB / 32; ++w) {
      lo[c] = fminf(lo[c], red[c][w]);
      hi[c] = fmaxf(hi[c], red[3 + c][w]);
    }
  }
}

// Squared distance between two boxes (0 when they overlap).
__device__ __forceinline__ float box_gap2(const float alo[3], const float ahi[3], const float blo[3],
                                          const float bhi[3]) {
  float d2 = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float g = fmaxf(0.f, fmaxf(blo[c] - ahi[c], alo[c] - bhi[c]));
    d2 = fmaf(g, g, d2);
  }
  return d2;
}

// c_0 + c_1 u + ... + c_D u^D. The profile P_r of a derivative of order r has degree q - r (make_frame).
template <int D>
__device__ __forceinline__ float horner(const float* c, float u) {
  float v = c[D];
#pragma unroll
  for (int k = D - 1; k >= 0; --k) v = fmaf(v, u, c[k]);
  return v;
}
template <int D>
__device__ __forceinline__ double horner(const double* c, double u) {
  double v = c[D];
#pragma unroll
  for (int k = D - 1; k >= 0; --k) v = ::fma(v, u, c[k]);
  return v;
}

template <int D>
__device__ __forceinline__ KV<F2> LaplacianT<D>::eval_f2(const Frame& f, F2 r2) {
  float a, b;
  split(r2, a, b);
  const float ua = sqrt_approx(a), ub = sqrt_approx(b);
  const float ea = ex2neg(ua), eb = ex2neg(ub);
  KV<F2> k;
  k.k0 = f2(ea * horner<D>(f.lc[0], ua), eb * horner<D>(f.lc[0], ub));
  k.k1 = f2(ea * horner<D - 1>(f.lc[1], ua), eb * horner<D - 1>(f.lc[1], ub));
  k.k2 = f2(ea * horner<D - 2>(f.lc[2], ua), eb * horner<D - 2>(f.lc[2], ub));
  return k;
}
template <int D>
__device__ __forceinline__ KV<double> LaplacianT<D>::eval_f64(const Frame& f, double r2) {
  const double u = sqrt(r2), e = exp2_neg(u);
  return {e * horner<D>(f.dc[0], u), e * horner<D - 1>(f.dc[1], u), e * horner<D - 2>(f.dc[2], u)};
}

// Shared-memory unit: two source fields (each a duplicated FP32 pair or one FP64 value), 16 bytes.
template <typename V>
struct alignas(16) Unit {
  V a, b;
};

// Per-target loaders: field values of targets i0, i1 packed into one V (V = double ignores i1).
template <typename V>
__device__ __forceinline__ V tgt_coord(const double* __restrict__ p, int i0, int i1, int c, double o, double s) {
  return VT<V>::pack((p[3 * i0 + c] - o) * s, (p[3 * i1 + c] - o) * s);
}
template <typename V>
__device__ __forceinline__ V tgt_field(const double* __restrict__ p, int stride, int i0, int i1, int c,
                                       double scale = 1.0) {
  return VT<V>::pack(scale * p[(size_t)stride * i0 + c], scale * p[(size_t)stride * i1 + c]);
}

// ---------------------------------------------------------------------------------------------------------
// Stream-K style launch plan. The work of one all-pairs sum is W = gx * TT units (gx target blocks of TPB*RT
// targets, TT source tiles of TPB sources). C = min(W, one resident wave) CTAs each take the contiguous unit range
// [start(c), start(c+1)), start(c) = floor(c W / C): every SM gets the same number of pair evaluations (to one
// tile), whatever n and m are. A CTA walks its range as segments (one target block, a run of tiles) and writes
// one compensated partial per segment; the partials of target block tb come from CTAs cta_of(tb TT) ..
// cta_of((tb+1) TT - 1) and are stored in slot (c - cta_of(tb TT)), so the epilogue reduces them in a fixed order.
// ---------------------------------------------------------------------------------------------------------
struct SKPlan {
  int gx = 0, TT = 0, C = 0, S = 0;  // S = max partial slots per target block
  long long W = 0;
  size_t box_off = 0;   // byte offset of the (gx + TT) coordinate boxes after the partial slots
  size_t ws_bytes = 0;
};

// a / b of non-negative values, in 32 bits where both fit (all but the largest problems): every CTA and every target of
// an epilogue divides before its first load, and a 64-bit division is some hundred dependent instructions. With one
// quotient per index instead of up to five of 64 bits: a step's two kernels 14.8 -> 13.2 us (forward, 2,562 points),
// 11.2 -> 10.1 (adjoint, 642 points).
__host__ __device__ __forceinline__ long long sk_quot(long long a, long long b) {
  if (((a | b) >> 32) == 0) return (unsigned)a / (unsigned)b;
  return a / b;
}

// CTA c takes the units [sk_start(c), sk_start(c + 1)); unit u belongs to the last c with c W / C < u + 1.
__host__ __device__ __forceinline__ long long sk_start(long long c, long long W, long long C) {
  return sk_quot(c * W, C);
}
__host__ __device__ __forceinline__ int sk_cta_of(long long u, long long W, long long C) {
  return (int)sk_quot((u + 1) * C - 1, W);
}

int device_sm_count();

__host__ __device__ __forceinline__ long long sym_tri(long long j) { return j * (j - 1) / 2; }

// The unit triangle for row blocks of B points and tiles of TPB: B a multiple of TPB (a row block spans kSpan tiles)
// or a divisor of it (a tile holds kShare row blocks). Row i takes the tiles from its own first one on; the tiles that
// overlap its own superblock of K = max(B, TPB) points are diagonal (rows only).
template <int TPB, int B>
struct SymGeom {
  static_assert(B % TPB == 0 || TPB % B == 0, "row blocks and tiles must nest");
  static constexpr int kSpan = B >= TPB ? B / TPB : 1, kShare = B < TPB ? TPB / B : 1;
  static constexpr int K = B >= TPB ? B : TPB;
  static __host__ __device__ __forceinline__ int first_tile(int i) { return B >= TPB ? i * kSpan : i / kShare; }
  // first unit of row i: the sum of TT - first_tile over the rows before it
  static __host__ __device__ __forceinline__ long long row_off(long long i, long long TT) {
    if (B >= TPB) return i * TT - kSpan * sym_tri(i);
    const long long q = i / kShare, r = i - q * kShare;
    return i * TT - (kShare * sym_tri(q) + q * r);
  }
  // column partials: superblock J receives one per row block before it (kShare J of them), K points each; offset of
  // the first one (in units of K points)
  static __host__ __device__ __forceinline__ long long col_first(long long J) { return kShare * sym_tri(J); }

  static __device__ __forceinline__ int row_of(long long u, int nblk, long long TT) {
    int lo = 0, hi = nblk - 1;  // largest i with row_off(i) <= u
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (row_off(mid, TT) <= u) lo = mid; else hi = mid - 1;
    }
    return lo;
  }
};

// Ops whose sum over all targets is all that is used (the energies) declare `static constexpr bool kTriangle = true;`.
// Their sources begin with the targets themselves (Op::self_count(P) of them, padded to whole tiles), and a term of
// that part is symmetric in the pair: target block i takes the self tiles from its own first one on, with weight 1 on
// its own superblock and 2 beyond it (Op::weigh), and every other source. A quarter of the pairs of an energy |S|^2 -
// 2 <S, S1> between surfaces of like size goes, half of those of a norm.
template <class Op, class = void>
struct Triangle : std::false_type {};
template <class Op>
struct Triangle<Op, std::void_t<decltype(Op::kTriangle)>> : std::bool_constant<Op::kTriangle> {};

// The units of an ordered sum: target blocks of B, source tiles of TPB, row-major; a triangle op's rows begin at their
// own first tile.
template <class Op, int TPB, int B>
struct Units {
  static constexpr bool kTri = Triangle<Op>::value;
  using Geo = SymGeom<TPB, B>;
  static __host__ __device__ __forceinline__ long long row_off(long long i, long long TT) {
    return kTri ? Geo::row_off(i, TT) : i * TT;
  }
  static __device__ __forceinline__ int row_of(long long u, int gx, long long TT) {
    return kTri ? Geo::row_of(u, gx, TT) : (int)sk_quot(u, TT);
  }
  static __device__ __forceinline__ int first_tile(int i) { return kTri ? Geo::first_tile(i) : 0; }
  // source of thread `tid` in tile j (whether there is one in `live`), and its weight for target block i
  static __device__ __forceinline__ int source(const typename Op::Params& P, int i, int j, int m, bool& live,
                                               double& weight) {
    weight = 1.0;
    if constexpr (kTri) {
      const int self = Op::self_count(P), ts = (self + TPB - 1) / TPB;
      if (j < ts) {
        const int l = j * TPB + (int)threadIdx.x;
        live = l < self;
        if (j >= Geo::first_tile(i) + Geo::kSpan) weight = 2.0;
        return l;
      }
      const int l = self + (j - ts) * TPB + (int)threadIdx.x;
      live = l < m;
      return l;
    } else {
      const int l = j * TPB + (int)threadIdx.x;
      live = l < m;
      return l;
    }
  }
  static inline int64_t tiles(const typename Op::Params& P, int64_t m) {
    if constexpr (kTri) {
      const int64_t self = Op::self_count(P);
      return (self + TPB - 1) / TPB + (m - self + TPB - 1) / TPB;
    } else {
      return (m + TPB - 1) / TPB;
    }
  }
};

// Most CTAs that a window of `len` consecutive units of W meets when C CTAs divide them evenly, the partial slots of a
// target block: sk_cta_of(u + len - 1) - sk_cta_of(u) is at most ceil((len - 1) C / W).
inline int sk_max_slots(long long len, long long W, long long C) { return (int)(((len - 1) * C + W - 1) / W + 1); }

// Slots times targets of an ordered sum, at most, over all problems of up to n targets and `tiles` source tiles (blocks
// of B targets, `wave` resident CTAs): a problem of W <= wave units has a slot per tile and tiles x blocks <= wave; a
// larger one has at most (wave / blocks) + 2 slots (W >= blocks x tiles).
inline int64_t sk_slot_targets_upto(int64_t n, int64_t tiles, int64_t B, int64_t wave) {
  const int64_t b = wave * B + 2 * n;
  return n * tiles < b ? n * tiles : b;
}

// `boxes`: reserve the coordinate boxes of exact culling (ops with Culled<Op>); other ops never read them, so their
// scratch is the partial slots alone (at most (C / gx + 2) * na * n partials, whatever m is).
template <class Op, int TPB, int B>
inline SKPlan make_plan(int64_t n, int64_t tiles, int na, size_t partial_bytes, int ctas_per_sm, bool boxes = true) {
  SKPlan p;
  if (n <= 0) return p;
  p.gx = (int)((n + B - 1) / B);
  if (tiles <= 0) return p;
  p.TT = (int)tiles;
  p.W = Units<Op, TPB, B>::row_off(p.gx, p.TT);
  const long long wave = (long long)device_sm_count() * (ctas_per_sm > 0 ? ctas_per_sm : 1);
  p.C = (int)(p.W < wave ? p.W : wave);
  p.S = sk_max_slots(p.TT, p.W, p.C);
  p.box_off = ((size_t)p.S * (size_t)na * (size_t)n * partial_bytes + 255) & ~(size_t)255;
  p.ws_bytes = p.box_off + (boxes ? (size_t)(p.gx + p.TT) * 6 * sizeof(float) : 0);
  return p;
}

// ---------------------------------------------------------------------------------------------------------
// Generic tiled all-pairs kernel.
//   Op::NS         number of source fields (scalars) staged per source (NU = ceil(NS/2) 16-byte units)
//   Op::NA         number of accumulators per target
//   Op::template Tgt<V>                                  per-lane-group register state
//   Op::template load_target<V>(P, i0, i1, tgt)          (i0, i1 < n; i1 ignored for V = double)
//   Op::source_fields(P, l, double* f)                   the NS source fields of source l (l < m), FP64
//   Op::template pair<V, Fam>(const Frame&, tgt, const V* s, V* acc)   (Fam: Gauss or Laplacian)
// Output: ws[(slot * NA + c) * n + i] = compensated partial of accumulator c of target i for one segment.
// ---------------------------------------------------------------------------------------------------------
// Ops may ask for a minimum number of resident CTAs per SM (`static constexpr int kMinCtas`), which caps the
// registers the compiler may use (65536 / (TPB * kMinCtas)).
// The cap applies to the FP32 (F2) kernels only.
template <class Op, typename V, class = void>
struct MinCtas : std::integral_constant<int, LDDMM_MIN_CTAS> {};
template <class Op>
struct MinCtas<Op, F2, std::void_t<decltype(Op::kMinCtas)>> : std::integral_constant<int, Op::kMinCtas> {};

// Ops may set their own unroll depth of the per-source loop (`static constexpr int kUnroll`); the default is
// LDDMM_SOURCE_UNROLL.
template <class Op, class = void>
struct UnrollOf : std::integral_constant<int, kSourceUnroll> {};
template <class Op>
struct UnrollOf<Op, std::void_t<decltype(Op::kUnroll)>> : std::integral_constant<int, Op::kUnroll> {};

// Ops whose sums are culled declare `static constexpr bool kCull = true;`: the surface data terms, whose faces are
// stored in a spatially coherent order by mesh generators and whose widths are often small against the shape.
// Elsewhere the box pre-pass and the per-tile test cost 2-3% and seldom pay (vertex orders are less coherent, and
// deformation widths large), so the other ops evaluate every tile.
template <class Op, class = void>
struct Culled : std::false_type {};
template <class Op>
struct Culled<Op, std::void_t<decltype(Op::kCull)>> : std::bool_constant<LDDMM_CULL != 0 && Op::kCull> {};

// Ops with an expanded-distance form of their Gaussian FP32 sums (pairs_kernel_x) declare
// `static constexpr bool kExpand = true;` and provide
//   NP                                   payload fields per source (staged after the coordinates)
//   target_point(P, i, double* c)        raw (unscaled) coordinates of target i
//   source_point(P, l, double* c, double* pay)   raw coordinates and the NP payload fields of source l
//   template TgtX<V>, load_target_x<V>(P, i0, i1, TgtX&)   per-lane-group target state besides the coordinates
//   accumulate<V>(const TgtX&, V e, const V* pay, V* acc)  the pair's contribution from its kernel value e
template <class Op, class = void>
struct Expanded : std::false_type {};
template <class Op>
struct Expanded<Op, std::void_t<decltype(Op::kExpand)>> : std::bool_constant<LDDMM_EXPAND != 0 && Op::kExpand> {};
template <class Op, typename V, class Fam>
constexpr bool kUseExpanded = Expanded<Op>::value && std::is_same<V, F2>::value && std::is_same<Fam, Gauss>::value;
// pairs_kernel_x's launch shape: 8 targets per thread (4 packed lane groups per source read) with the compensated
// sums in shared memory (136 registers, 3 CTAs per SM) measured 3-6% faster than the light ops' 4 targets per thread
// with sums in registers (applyK at levels 6 and 7, varifold energy at level 6)
#ifndef LDDMM_RT_X
#define LDDMM_RT_X 8  // targets per thread of pairs_kernel_x (0: the caller's launch shape)
#endif
#ifndef LDDMM_X_COMP_SMEM
#define LDDMM_X_COMP_SMEM 1  // 0: pairs_kernel_x keeps its compensated sums in registers
#endif
// Targets per thread of the kernel that runs an op (the plan, the launch and the epilogue all use it).
// Optional members of an expanded op: kRtX (its targets per thread, default LDDMM_RT_X), NAX (accumulators of the
// expanded form, default NA) with x_partial(expand, y, sums, out) mapping them to the NA sums the epilogue reads,
// and kExpandR2 (its bound on a block's radius^2, default kExpandR2 below).
template <class Op, class = void>
struct RtXOf : std::integral_constant<int, LDDMM_RT_X> {};
template <class Op>
struct RtXOf<Op, std::void_t<decltype(Op::kRtX)>> : std::integral_constant<int, Op::kRtX> {};
template <class Op, class = void>
struct NAXOf : std::integral_constant<int, Op::NA> {};
template <class Op>
struct NAXOf<Op, std::void_t<decltype(Op::NAX)>> : std::integral_constant<int, Op::NAX> {};
template <class Op, typename V, int RT, class Fam>
constexpr int kRunRT = (kUseExpanded<Op, V, Fam> && RtXOf<Op>::value > 0) ? RtXOf<Op>::value : RT;

// Origin of a target block's coordinates in the split self-sums: the caller's, or a middle of the block's own points, so
// that a caller whose points live on the device need not read a centroid back (one synchronisation per call before).
// Coordinate by coordinate, on FP32 offsets of 32 points of the block from a reference (the median of its first, middle
// and last point): the mean of the middle two of four lanes eight apart, the same of four neighbouring groups, and the
// mean of both halves. Far or non-finite points do not move it unless two of four are, several times over; a run of far
// points in storage order, up to a quarter of the 32 (or of a shorter block), never does (with groups of four
// neighbouring lanes six far points at 1e5 in a block of 32 moved it to 1.2e4: FP64 sums of the near ones 2e-13 instead
// of 1e-16). In a block of a scattered set it lies within an eighth of the half extent from the centre, so that
// coordinates round as about a common centroid (Gaussian sums and steps of cubes of 32 widths in random order, 700 to
// 12,000 points: 0.99 of the errors about the centroid; with the median of three points alone, 0.45 of the half extent,
// 1.2-1.5). A reference that is not finite leaves the block in the caller's frame. It costs 0.2 us of a step (forward
// step of 2,562 points 12.37 -> 12.57 us), where reading a centroid back costs a call 15. In the unsplit kernels, whose
// calls are long against that, the six more registers cost 1-4% (forward step at 40,962 points 783 -> 792 us, FP64
// first-order adjoint step 2458 -> 2569).

// the mean of the middle two of the values of lanes l, l ^ A, l ^ B and l ^ A ^ B
template <int A, int B>
__device__ __forceinline__ float middle4_lanes(float v) {
  const float w = __shfl_xor_sync(0xffffffffu, v, A);
  const float lo = fminf(v, w), hi = fmaxf(v, w);
  const float lo2 = __shfl_xor_sync(0xffffffffu, lo, B), hi2 = __shfl_xor_sync(0xffffffffu, hi, B);
  return 0.5f * (fmaxf(lo, lo2) + fminf(hi, hi2));
}
// coordinate c of it for points first .. last, by one whole warp (the same in every lane); x: that of a point of the lane,
// 32 different ones in the warp if `full`
__device__ __forceinline__ double segment_origin(const Frame& f, const double* __restrict__ points, int first, int last,
                                                 int c, bool full, double x) {
  const double given = c == 0 ? f.o0 : c == 1 ? f.o1 : f.o2;
  if (!f.own) return given;
  const int count = last - first + 1;
  const double* p = points + c;
  // fewer than 32 points: spread evenly, so that lanes eight apart have different ones from four points on
  if (!full) x = p[3 * (size_t)(first + (((int)(threadIdx.x & 31) * count) >> 5))];
  const double r0 = p[3 * (size_t)first], r1 = p[3 * (size_t)(first + (last - first) / 2)], r2 = p[3 * (size_t)last];
  const float f0 = (float)r0, f1 = (float)r1, f2 = (float)r2;
  const float fm = fmaxf(fminf(f0, f1), fminf(fmaxf(f0, f1), f2));
  const double m = fm == f0 ? r0 : fm == f1 ? r1 : r2;
  float v = middle4_lanes<1, 2>(middle4_lanes<8, 16>((float)(x - m)));
  v = 0.5f * (v + __shfl_xor_sync(0xffffffffu, v, 4));
  if (!isfinite(m)) return given;
  return count >= 4 && isfinite(v) ? m + (double)v : m;
}
// The op's parameters with the segment's origin (kept in shared memory).
template <class Params>
__device__ __forceinline__ Params with_origin(const Params& P, const double* org) {
  Params q = P;
  q.f.o0 = org[0];
  q.f.o1 = org[1];
  q.f.o2 = org[2];
  return q;
}

// SPLIT (problems too small to fill the GPU): the warps of a CTA share its 32 RT targets and take a quarter of every
// source tile each, instead of TPB RT targets and whole tiles; their sums meet in shared memory when a segment ends.
template <class Op, typename V, int TPB, int RT, class Fam, bool SPLIT>
__global__ void __launch_bounds__(TPB, MinCtas<Op, V>::value)
    pairs_kernel(const typename Op::Params P, int n, int m, int TT, long long W, int C,
                 typename VT<V>::Partial* __restrict__ ws, const float* __restrict__ boxes) {
  constexpr int L = VT<V>::kLanes;
  constexpr int G = RT / L;  // lane groups per thread
  constexpr int NU = (Op::NS + 1) / 2;
  constexpr int kUnroll = UnrollOf<Op>::value;
  static_assert(RT % L == 0, "targets per thread must be a multiple of the lane count");
  __shared__ Unit<V> sm[NU][TPB];
  // The segment's compensated sums live in shared memory (one private column per thread: no barrier needed) unless
  // the op keeps them in registers; shared memory frees 2-4 registers per accumulator for more resident warps.
  constexpr bool kSm = LDDMM_COMP_SMEM && !CompInRegisters<Op>::value;
  __shared__ V cs[kSm || SPLIT ? G * Op::NA * Comp<V>::kWords : 1][TPB];
  constexpr int TW = SPLIT ? 32 : TPB;  // targets a lane-group index apart
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Exact culling (ops with Culled<Op>): a (target block, source tile) unit whose coordinate boxes (box_kernel) are
  // farther apart than the distance at which the kernel's radial factors are exactly zero in this arithmetic
  // contributes exactly nothing, and is skipped by the whole CTA.
  constexpr float kZeroR2 = Fam::template kCullR2<V>;
  using Un = Units<Op, TPB, TW * RT>;
  const int gx = (n + TW * RT - 1) / (TW * RT);
  __shared__ float tbox[6];  // the segment's target box, in shared memory (re-read per tile, not held in registers)
  VT<V>::setup();
  chain_wait();

  const long long u_end = sk_start(blockIdx.x + 1, W, C);
  long long u = sk_start(blockIdx.x, W, C);
  int tb = u < u_end ? Un::row_of(u, gx, TT) : 0;
  while (u < u_end) {
    const long long off = Un::row_off(tb, TT);
    const int first = Un::first_tile(tb);
    const int j0 = first + (int)(u - off);
    const int j1 = first + (int)((u_end - off) < TT - first ? (u_end - off) : TT - first);
    const int slot = (int)blockIdx.x - sk_cta_of(off, W, C);

    typename Op::template Tgt<V> tgt[G];
    Comp<V> cmp[G][Op::NA];   // used when !kSm
    // target of (group g, lane k): base + (g * L + k) * TW
    const int base = tb * (TW * RT) + (SPLIT ? lane : (int)threadIdx.x);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      int i0 = base + (g * L) * TW, i1 = base + (g * L + L - 1) * TW;
      i0 = i0 < n ? i0 : n - 1;
      i1 = i1 < n ? i1 : n - 1;
      Op::template load_target<V>(P, i0, i1, tgt[g]);
#pragma unroll
      for (int c = 0; c < Op::NA; ++c) {
        cmp[g][c].zero();
        if constexpr (kSm) cmp[g][c].template store<TPB>(cs, g * Op::NA + c, threadIdx.x);
      }
    }
    if constexpr (Culled<Op>::value) {
      __syncthreads();  // the previous segment's last tile test has read tbox
      if (threadIdx.x < 6) tbox[threadIdx.x] = boxes[6 * tb + threadIdx.x];
      __syncthreads();
    }

    for (int j = j0; j < j1; ++j) {
      if constexpr (Culled<Op>::value) {
        const float* sbox = boxes + 6 * (gx + j);
        if (box_gap2(tbox, tbox + 3, sbox, sbox + 3) > kZeroR2) continue;  // uniform over the CTA
      }
      {
        bool live;
        double weight;
        const int l = Un::source(P, tb, j, m, live, weight);
        double f[2 * NU];
#pragma unroll
        for (int q = 0; q < 2 * NU; ++q) f[q] = 0.0;
        if (live) Op::source_fields(P, l, f);
        if constexpr (Un::kTri) Op::weigh(f + 3, weight);
#pragma unroll
        for (int q = 0; q < NU; ++q) {
          Unit<V> w;
          w.a = VT<V>::dup(f[2 * q]);
          w.b = VT<V>::dup(f[2 * q + 1]);
          sm[q][threadIdx.x] = w;
        }
      }
      __syncthreads();
      V acc[G][Op::NA];
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < Op::NA; ++c) acc[g][c] = VT<V>::zero();
#pragma unroll kUnroll
      for (int jj = 0; jj < TW; ++jj) {
        V s[2 * NU];
#pragma unroll
        for (int q = 0; q < NU; ++q) {
          const Unit<V> w = sm[q][SPLIT ? warp * 32 + jj : jj];
          s[2 * q] = w.a;
          s[2 * q + 1] = w.b;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) Op::template pair<V, Fam>(P.f, tgt[g], s, acc[g]);
      }
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < Op::NA; ++c) {
          if constexpr (kSm) cmp[g][c].template load<TPB>(cs, g * Op::NA + c, threadIdx.x);
          cmp[g][c].merge(acc[g][c]);
          if constexpr (kSm) cmp[g][c].template store<TPB>(cs, g * Op::NA + c, threadIdx.x);
        }
      __syncthreads();
    }

    if (SPLIT && u + (j1 - j0) >= u_end) chain_go();
    if constexpr (SPLIT) {
      if constexpr (!kSm) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int c = 0; c < Op::NA; ++c) cmp[g][c].template store<TPB>(cs, g * Op::NA + c, threadIdx.x);
      }
      __syncthreads();
      // sum c of the lanes' targets by warp c mod W, over the W warps in order
#pragma unroll
      for (int g = 0; g < G; ++g)
        for (int c = warp; c < Op::NA; c += TPB / 32) {
          double sum[L];
#pragma unroll
          for (int k = 0; k < L; ++k) sum[k] = 0.0;
#pragma unroll
          for (int w = 0; w < TPB / 32; ++w) {
            Comp<V> m;
            m.template load<TPB>(cs, g * Op::NA + c, w * 32 + lane);
#pragma unroll
            for (int k = 0; k < L; ++k) sum[k] += partial_value(m.partial(k));
          }
#pragma unroll
          for (int k = 0; k < L; ++k) {
            const int i = base + (g * L + k) * TW;
            if (i < n) ws[((size_t)slot * Op::NA + c) * (size_t)n + i] = VT<V>::to_partial(sum[k]);
          }
        }
      __syncthreads();  // the next segment clears the sums
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const int i = base + (g * L + k) * TW;
          if (i < n) {
#pragma unroll
            for (int c = 0; c < Op::NA; ++c) {
              if constexpr (kSm) cmp[g][c].template load<TPB>(cs, g * Op::NA + c, threadIdx.x);
              ws[((size_t)slot * Op::NA + c) * (size_t)n + i] = cmp[g][c].partial(k);
            }
          }
        }
    }
    u += j1 - j0;
    ++tb;
  }
}

// ---------------------------------------------------------------------------------------------------------
// Expanded-distance Gaussian pair kernel (FP32; ops with Expanded<Op>).
//
// With the coordinates of a segment taken relative to the centre o of its target block (the midpoint of the
// block's coordinate box, scaled units),
//     2^-|y - x|^2 = 2^-|y|^2 * 2^-(|x|^2 - 2 y.x),
// and the bracket costs three packed FMAs per pair from the staged fields X = -2 x and q = |x|^2 (the difference
// form costs three subtractions, a multiply and two FMAs): 6 FP32 lane-ops and one ex2 per pair for K a instead
// of 9, which leaves the pair loop bound by the MUFU (ex2) pipe instead of the FP32 pipe. The factor 2^-|y|^2 is
// common to every term of a target and multiplies the segment's compensated sums once, in FP64, when they are
// written. The identity is exact for the FP32-rounded relative coordinates; the rounding of the bracket grows with
// |y|^2 and |x|^2 (far sources have a large |x|^2 but terms that are smaller still), so a block is evaluated in the
// expanded form only when its radius^2 (scaled) is at most kExpandR2, which keeps the relative L2 error of the
// sums near 1e-6 (FP32 emulation with targets in a ball of that radius: 7e-7 at 32, 1.2e-6 at 64; the difference
// form: 5e-8); other blocks (point sets in no spatial order, widths small against a block) use the difference form,
// which costs ~20% more per pair (and, stream-K balancing units rather than time, the kernel waits for the CTAs that
// drew such blocks). Both forms share the launch plan and the epilogue of pairs_kernel.
// ---------------------------------------------------------------------------------------------------------
constexpr float kExpandR2 = 64.0f;
template <class Op, class = void>
struct ExpandR2Of {
  static constexpr float value = kExpandR2;
};
template <class Op>
struct ExpandR2Of<Op, std::void_t<decltype(Op::kExpandR2)>> {
  static constexpr float value = Op::kExpandR2;
};
template <class Op, class = void>
struct HasXPartial : std::false_type {};
template <class Op>
struct HasXPartial<Op, std::void_t<decltype(&Op::x_partial)>> : std::true_type {};

template <class Op, int TPB, int RT, bool SPLIT>
__global__ void __launch_bounds__(TPB, MinCtas<Op, F2>::value)
    pairs_kernel_x(const typename Op::Params P, int n, int m, int TT, long long W, int C,
                   float2* __restrict__ ws, const float* __restrict__ boxes) {
  constexpr int L = 2;
  constexpr int G = RT / L;
  constexpr int NF = 4 + Op::NP;  // staged fields: X or x (3), q (1), payload (NP)
  constexpr int NU = (NF + 1) / 2;
  constexpr int TW = SPLIT ? 32 : TPB;   // targets a lane-group index apart (SPLIT: as in pairs_kernel)
  constexpr int NAX = NAXOf<Op>::value;  // accumulators of the expanded form
  constexpr int kUnroll = UnrollOf<Op>::value;
  static_assert(RT % L == 0, "targets per thread must be a multiple of the lane count");
  __shared__ Unit<F2> sm[NU][TPB];
  __shared__ float red[6][TPB / 32];
  constexpr bool kSm = SPLIT || LDDMM_X_COMP_SMEM != 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ F2 cs[kSm ? G * NAX * 2 : 1][TPB];
  const Frame& f = P.f;
  const double fo[3] = {f.o0, f.o1, f.o2};
  using Un = Units<Op, TPB, TW * RT>;
  const int gx = (n + TW * RT - 1) / (TW * RT);
  chain_wait();

  const long long u_end = sk_start(blockIdx.x + 1, W, C);
  long long u = sk_start(blockIdx.x, W, C);
  int tb = u < u_end ? Un::row_of(u, gx, TT) : 0;
  while (u < u_end) {
    const long long off = Un::row_off(tb, TT);
    const int first = Un::first_tile(tb);
    const int j0 = first + (int)(u - off);
    const int j1 = first + (int)((u_end - off) < TT - first ? (u_end - off) : TT - first);
    const int slot = (int)blockIdx.x - sk_cta_of(off, W, C);
    const int base = tb * (TW * RT) + (SPLIT ? lane : (int)threadIdx.x);

    // the block's box and centre (every CTA working on block tb derives the same ones)
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int t = 0; t < RT; ++t) {
      int i = base + t * TW;
      i = i < n ? i : n - 1;
      double y[3];
      Op::target_point(P, i, y);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float v = (float)((y[c] - fo[c]) * f.s);
        lo[c] = fminf(lo[c], v);
        hi[c] = fmaxf(hi[c], v);
      }
    }
    block_box<TPB>(lo, hi, red);  // its barrier also orders the previous segment's last tile reads
    float ob[3], rb2 = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ob[c] = 0.5f * (lo[c] + hi[c]);
      const float h = 0.5f * (hi[c] - lo[c]);
      rb2 = fmaf(h, h, rb2);
    }
    const bool expand = rb2 <= ExpandR2Of<Op>::value;  // uniform over the CTA

    F2 yt[G][3];  // relative scaled target coordinates, lanes = targets (g L, g L + 1) of the thread
    typename Op::template TgtX<F2> tx[G];
    Comp<F2> cmp[G][NAX];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      int i0 = base + (g * L) * TW, i1 = base + (g * L + 1) * TW;
      i0 = i0 < n ? i0 : n - 1;
      i1 = i1 < n ? i1 : n - 1;
      double y0[3], y1[3];
      Op::target_point(P, i0, y0);
      Op::target_point(P, i1, y1);
#pragma unroll
      for (int c = 0; c < 3; ++c)
        yt[g][c] = f2((float)((y0[c] - fo[c]) * f.s - (double)ob[c]), (float)((y1[c] - fo[c]) * f.s - (double)ob[c]));
      Op::template load_target_x<F2>(P, i0, i1, tx[g]);
#pragma unroll
      for (int c = 0; c < NAX; ++c) {
        cmp[g][c].zero();
        if constexpr (kSm) cmp[g][c].template store<TPB>(cs, g * NAX + c, threadIdx.x);
      }
    }

    for (int j = j0; j < j1; ++j) {
      if constexpr (Culled<Op>::value) {
        // the same test as pairs_kernel: every term of the unit is exactly zero in the difference form; in the
        // expanded form each would be below 2^-127 of its payload
        const float* sbox = boxes + 6 * (gx + j);
        if (box_gap2(lo, hi, sbox, sbox + 3) > Gauss::kCullR2<F2>) continue;  // uniform over the CTA
      }
      {
        bool live;
        double weight;
        const int l = Un::source(P, tb, j, m, live, weight);
        double fl[2 * NU];
#pragma unroll
        for (int q = 0; q < 2 * NU; ++q) fl[q] = 0.0;
        if (live) {
          double xr[3], r2 = 0.0;
          Op::source_point(P, l, xr, fl + 4);
          if constexpr (Un::kTri) Op::weigh_x(fl + 4, weight);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float xc = (float)((xr[c] - fo[c]) * f.s - (double)ob[c]);
            r2 += (double)xc * (double)xc;
            fl[c] = expand ? -2.0 * (double)xc : (double)xc;
          }
          fl[3] = r2;
        }
#pragma unroll
        for (int q = 0; q < NU; ++q) {
          Unit<F2> w;
          w.a = VT<F2>::dup(fl[2 * q]);
          w.b = VT<F2>::dup(fl[2 * q + 1]);
          sm[q][threadIdx.x] = w;
        }
      }
      __syncthreads();
      F2 acc[G][NAX];
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < NAX; ++c) acc[g][c] = VT<F2>::zero();
      if (expand) {
#pragma unroll kUnroll
        for (int jj = 0; jj < TW; ++jj) {
          F2 s[2 * NU];
#pragma unroll
          for (int q = 0; q < NU; ++q) {
            const Unit<F2> w = sm[q][SPLIT ? warp * 32 + jj : jj];
            s[2 * q] = w.a;
            s[2 * q + 1] = w.b;
          }
#pragma unroll
          for (int g = 0; g < G; ++g) {
            F2 arg = fma(yt[g][2], s[2], s[3]);  // |x|^2 - 2 y.x
            arg = fma(yt[g][1], s[1], arg);
            arg = fma(yt[g][0], s[0], arg);
            Op::template accumulate<true>(tx[g], yt[g], VT<F2>::expneg(arg), s, acc[g]);
          }
        }
      } else {
#pragma unroll kUnroll
        for (int jj = 0; jj < TW; ++jj) {
          F2 s[2 * NU];
#pragma unroll
          for (int q = 0; q < NU; ++q) {
            const Unit<F2> w = sm[q][SPLIT ? warp * 32 + jj : jj];
            s[2 * q] = w.a;
            s[2 * q + 1] = w.b;
          }
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const F2 d0 = yt[g][0] - s[0], d1 = yt[g][1] - s[1], d2 = yt[g][2] - s[2];
            Op::template accumulate<false>(tx[g], yt[g], VT<F2>::expneg(fma(d2, d2, fma(d1, d1, d0 * d0))), s, acc[g]);
          }
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < NAX; ++c) {
          if constexpr (kSm) cmp[g][c].template load<TPB>(cs, g * NAX + c, threadIdx.x);
          cmp[g][c].merge(acc[g][c]);
          if constexpr (kSm) cmp[g][c].template store<TPB>(cs, g * NAX + c, threadIdx.x);
        }
      __syncthreads();
    }

    if (SPLIT && u + (j1 - j0) >= u_end) chain_go();
    if constexpr (SPLIT) __syncthreads();  // every warp's sums are in shared memory (also when no tile was evaluated)
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const int i = base + (g * L + k) * TW;
        // SPLIT: target g L + k of the lanes by warp (g L + k) mod W, over the W warps in order
        if (i < n && (!SPLIT || (g * L + k) % (TPB / 32) == warp)) {
          double yr[3], y2 = 0.0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            yr[c] = VT<F2>::lane(yt[g][c], k);
            y2 += yr[c] * yr[c];
          }
          const double fac = expand ? exp2(-y2) : 1.0;
          double v[NAX], o[Op::NA];
#pragma unroll
          for (int c = 0; c < NAX; ++c) {
            if constexpr (SPLIT) {
              v[c] = 0.0;
#pragma unroll
              for (int w = 0; w < TPB / 32; ++w) {
                Comp<F2> m;
                m.template load<TPB>(cs, g * NAX + c, w * 32 + lane);
                v[c] += partial_value(m.partial(k));
              }
            } else {
              if constexpr (kSm) cmp[g][c].template load<TPB>(cs, g * NAX + c, threadIdx.x);
              v[c] = partial_value(cmp[g][c].partial(k));
            }
          }
          if constexpr (HasXPartial<Op>::value) {
            Op::x_partial(expand, yr, v, o);
          } else {
#pragma unroll
            for (int c = 0; c < Op::NA; ++c) o[c] = v[c];
          }
#pragma unroll
          for (int c = 0; c < Op::NA; ++c) {
            ws[((size_t)slot * Op::NA + c) * (size_t)n + i] = VT<F2>::to_partial(o[c] * fac);
          }
        }
      }
    if constexpr (SPLIT) __syncthreads();  // the next segment clears the sums
    u += j1 - j0;
    ++tb;
  }
}

// Coordinate boxes for exact culling, from the same scaled coordinates the pair kernel uses: block b < gx covers
// target block b (its TPB * RT targets), block gx + j source tile j. boxes[6 b ..] = (lo xyz, hi xyz).
template <class Op, typename V, int TPB, int RT, bool SPLIT>
__global__ void __launch_bounds__(TPB) box_kernel(const typename Op::Params P, int n, int m, int gx,
                                                  float* __restrict__ boxes) {
  constexpr int L = VT<V>::kLanes;
  constexpr int G = RT / L;
  constexpr int NU = (Op::NS + 1) / 2;
  constexpr int TW = SPLIT ? 32 : TPB;
  __shared__ float red[6][TPB / 32];
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  const int b = blockIdx.x;
  chain_wait();
  if (b < gx) {
    const int base = b * (TW * RT) + (int)threadIdx.x % TW;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      int i0 = base + (g * L) * TW, i1 = base + (g * L + L - 1) * TW;
      i0 = i0 < n ? i0 : n - 1;
      i1 = i1 < n ? i1 : n - 1;
      typename Op::template Tgt<V> t;
      Op::template load_target<V>(P, i0, i1, t);
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const float y[3] = {(float)VT<V>::lane(t.y0, k), (float)VT<V>::lane(t.y1, k), (float)VT<V>::lane(t.y2, k)};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          lo[c] = fminf(lo[c], y[c]);
          hi[c] = fmaxf(hi[c], y[c]);
        }
      }
    }
  } else {
    bool live;
    double weight;
    const int l = Units<Op, TPB, TW * RT>::source(P, 0, b - gx, m, live, weight);
    if (live) {
      double f[2 * NU];
      Op::source_fields(P, l, f);
#pragma unroll
      for (int c = 0; c < 3; ++c) lo[c] = hi[c] = (float)f[c];
    }
  }
  block_box<TPB>(lo, hi, red);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      boxes[6 * b + c] = lo[c];
      boxes[6 * b + 3 + c] = hi[c];
    }
  }
}

// Epilogue: reduce the partial slots of target i (its block's CTAs) in FP64, then Op::finalize. `tpp` threads per
// target (a power of two <= 32): thread j sums the slots j, j + tpp, ... and the tpp sums are added in the order j = 0,
// 1, ... from shared memory, so the order of every addition is fixed. With one thread per target its slots are one
// serial chain (surface gradient of 2,990 against 3,534 faces: 41 us for 47 slots of 8 sums).
constexpr int kFinThreads = 256;

// The NV sums of point p over its tpp threads (thread j of np * tpp holds v), in the order j = 0, 1, ...: field c by
// thread c mod tpp, returned to thread 0.
template <int NV>
__device__ __forceinline__ void finalize_meet(double (*red)[kFinThreads], int np, int tpp, int p, int j, double* v) {
  if (tpp == 1) return;
#pragma unroll
  for (int c = 0; c < NV; ++c) red[c][threadIdx.x] = v[c];
  __syncthreads();
  for (int c = j; c < NV; c += tpp) {
    double sum = red[c][p];
    for (int k = 1; k < tpp; ++k) sum += red[c][k * np + p];
    red[c][p] = sum;
  }
  __syncthreads();
  if (j == 0)
#pragma unroll
    for (int c = 0; c < NV; ++c) v[c] = red[c][p];
}

template <class Op, typename V, int TPB, int B>
__global__ void __launch_bounds__(kFinThreads)
    finalize_kernel(const typename Op::Params P, int n, int TT, long long W, int C,
                    const typename VT<V>::Partial* __restrict__ ws, int tpp) {
  __shared__ double red[Op::NA][kFinThreads];
  const int np = kFinThreads / tpp;
  const int p = threadIdx.x % np, j = threadIdx.x / np;
  const int i = blockIdx.x * np + p;
  using Un = Units<Op, TPB, B>;
  const int tb = i / B;
  const int nslot =
      i < n && W > 0 ? sk_cta_of(Un::row_off(tb + 1, TT) - 1, W, C) - sk_cta_of(Un::row_off(tb, TT), W, C) + 1 : 0;
  chain_wait();
  double acc[Op::NA];
#pragma unroll
  for (int c = 0; c < Op::NA; ++c) acc[c] = 0.0;
  for (int s = j; s < nslot; s += tpp)
#pragma unroll
    for (int c = 0; c < Op::NA; ++c) acc[c] += partial_value(ws[((size_t)s * Op::NA + c) * (size_t)n + i]);
  finalize_meet<Op::NA>(red, np, tpp, p, j, acc);
  if (i < n && j == 0) Op::finalize(P, i, acc);
}

// Threads per point of an epilogue: enough to split a chain of slots into pieces of about four, at most 8.
inline int finalize_tpp(int chain) {
  int t = 1;
  while (t < 8 && chain > 4 * t) t <<= 1;
  return t;
}
inline int finalize_grid(int64_t n, int tpp) {
  const int64_t np = kFinThreads / tpp;
  return (int)((n + np - 1) / np);
}

// Deterministic single-block sum of `count` doubles: out[0] = (accumulate ? out[0] : 0) + scale * sum(v).
__global__ void ordered_sum_kernel(const double* __restrict__ v, int count, double scale, double* out, int accumulate);

int resident_ctas(const void* kernel, int threads, size_t dynamic_smem = 0);

template <class Op, typename V, int TPB, int RT, class Fam, bool SPLIT>
inline int ctas_per_sm() {
  static int cached = 0;
  if (cached == 0) {
    const void* k;
    if constexpr (kUseExpanded<Op, V, Fam>)
      k = reinterpret_cast<const void*>(&pairs_kernel_x<Op, TPB, kRunRT<Op, V, RT, Fam>, SPLIT>);
    else
      k = reinterpret_cast<const void*>(&pairs_kernel<Op, V, TPB, RT, Fam, SPLIT>);
    int c = resident_ctas(k, TPB);
    cached = c > 0 ? c : 4;
  }
  return cached;
}

// Ops that never split declare `static constexpr bool kNoSplit = true;`.
template <class Op, class = void>
struct CanSplit : std::true_type {};
template <class Op>
struct CanSplit<Op, std::void_t<decltype(Op::kNoSplit)>> : std::bool_constant<!Op::kNoSplit> {};

template <class Op, typename V, int TPB, int RT, class Fam, bool SPLIT>
inline SKPlan pairs_plan(int64_t n, int64_t tiles) {
  return make_plan<Op, TPB, (SPLIT ? 32 : TPB) * kRunRT<Op, V, RT, Fam>>(
      n, tiles, Op::NA, sizeof(typename VT<V>::Partial), ctas_per_sm<Op, V, TPB, RT, Fam, SPLIT>(), Culled<Op>::value);
}

// Whether a problem splits: its whole-tile units would fill less than a third of one resident wave (FP32), or less than
// two and a half waves (FP64, whose units are several times longer). us, unsplit | split, n = m: FP32 K a 162: 12.7 |
// 8.5, 1,500: 15.8 | 10.6, 2,562 (0.14 waves): 16.0 | 12.8, 6,000 (0.64): 23.3 | 27.6; applyDiffKT 2,562 (0.21): 13.6 |
// 13.1, 6,000 (0.95): 32.3 | 35.5; DDK 1,500 (0.16): 11.7 | 10.3, 2,562 (0.5): 16.0 | 19.0; varifold gradient 1,280
// faces: 33.6 | 30.4, 5,120 (1.8): 79.3 | 81.4. FP64 K a 642: 13.6 | 8.0, applyDiffKT 2,562 (0.4): 25.8 | 22.7, 6,000
// (1.9): 93 | 82, varifold gradient 5,120 (2.7): 159 | 162, K a 20,000 (21): 577 | 597.
template <class Op, typename V, int TPB, int RT, class Fam>
inline bool pairs_split(int64_t n, int64_t tiles) {
  constexpr int64_t B = (int64_t)TPB * kRunRT<Op, V, RT, Fam>;
  const int64_t units = ((n + B - 1) / B) * tiles;
  const int64_t wave = (int64_t)device_sm_count() * ctas_per_sm<Op, V, TPB, RT, Fam, false>();
  return std::is_same<V, F2>::value ? 3 * units < wave : 2 * units < 5 * wave;
}

template <class Op, typename V, int TPB, int RT, class Fam, bool SPLIT>
inline int launch_pairs(const typename Op::Params& P, int64_t n, int64_t m, void* ws, size_t ws_bytes,
                        cudaStream_t stream) {
  constexpr int R = kRunRT<Op, V, RT, Fam>;
  const SKPlan plan = pairs_plan<Op, V, TPB, RT, Fam, SPLIT>(n, Units<Op, TPB, TPB>::tiles(P, m));
  if (plan.ws_bytes > ws_bytes) return kWorkspaceTooSmall;
  if (plan.ws_bytes > 0 && ws == nullptr) return kInvalidArgument;
  auto* part = reinterpret_cast<typename VT<V>::Partial*>(ws);
  if (plan.W > 0) {
    float* boxes = Culled<Op>::value ? reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + plan.box_off) : nullptr;
    if (Culled<Op>::value)
      launch_chained(box_kernel<Op, V, TPB, R, SPLIT>, plan.gx + plan.TT, TPB, 0, stream, P, (int)n, (int)m, plan.gx,
                     boxes);
    if constexpr (kUseExpanded<Op, V, Fam>) {
      launch_chained(pairs_kernel_x<Op, TPB, R, SPLIT>, plan.C, TPB, 0, stream, P, (int)n, (int)m, plan.TT, plan.W,
                     plan.C, part, boxes);
    } else {
      launch_chained(pairs_kernel<Op, V, TPB, RT, Fam, SPLIT>, plan.C, TPB, 0, stream, P, (int)n, (int)m, plan.TT,
                     plan.W, plan.C, part, boxes);
    }
  }
  const int tpp = finalize_tpp(plan.S);
  launch_chained(finalize_kernel<Op, V, TPB, (SPLIT ? 32 : TPB) * R>, finalize_grid(n, tpp), kFinThreads, 0, stream, P,
                 (int)n, plan.TT, plan.W, plan.C, part, tpp);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

template <class Op, typename V, int TPB, int RT, class Fam = Gauss>
inline int run_pairs(const typename Op::Params& P, int64_t n, int64_t m, void* ws, size_t ws_bytes,
                     cudaStream_t stream) {
  if (n <= 0) return kOk;
  if (n > INT32_MAX / 4 || m > INT32_MAX / 4) return kInvalidArgument;
  if constexpr (CanSplit<Op>::value) {
    if (pairs_split<Op, V, TPB, RT, Fam>(n, Units<Op, TPB, TPB>::tiles(P, m)))
      return launch_pairs<Op, V, TPB, RT, Fam, true>(P, n, m, ws, ws_bytes, stream);
  }
  return launch_pairs<Op, V, TPB, RT, Fam, false>(P, n, m, ws, ws_bytes, stream);
}

// Scratch of n targets and m sources (the larger of both shapes'). A triangle op's sources are n targets and m - n
// others, each padded to whole tiles.
template <class Op, typename V, int TPB, int RT, class Fam = Gauss>
inline size_t pairs_ws_bytes(int64_t n, int64_t m) {
  const int64_t tiles = Triangle<Op>::value ? (n + TPB - 1) / TPB + (m - n + TPB - 1) / TPB : (m + TPB - 1) / TPB;
  size_t b = pairs_plan<Op, V, TPB, RT, Fam, false>(n, tiles).ws_bytes;
  if constexpr (CanSplit<Op>::value) {
    const size_t s = pairs_plan<Op, V, TPB, RT, Fam, true>(n, tiles).ws_bytes;
    b = s > b ? s : b;
  }
  return b;
}

// Scratch that holds every problem of up to n targets and m sources: the slots of a plan are not monotone in either
// (as many as tiles while every unit has a CTA of its own, half as many where two units go to one).
template <class Op, typename V, int TPB, int RT, class Fam, bool SPLIT>
inline size_t pairs_shape_ws_upto(int64_t n, int64_t m) {
  static_assert(!Triangle<Op>::value, "an energy's scratch is asked for its own face counts");
  if (n <= 0 || m <= 0) return 0;
  constexpr int64_t B = (int64_t)(SPLIT ? 32 : TPB) * kRunRT<Op, V, RT, Fam>;
  const int64_t tiles = (m + TPB - 1) / TPB;
  const int64_t wave = (int64_t)device_sm_count() * ctas_per_sm<Op, V, TPB, RT, Fam, SPLIT>();
  const size_t rows = (size_t)sk_slot_targets_upto(n, tiles, B, wave) * Op::NA * sizeof(typename VT<V>::Partial);
  const size_t boxes = Culled<Op>::value ? (size_t)((n + B - 1) / B + tiles) * 6 * sizeof(float) : 0;
  return ((rows + 255) & ~(size_t)255) + boxes;
}
template <class Op, typename V, int TPB, int RT, class Fam = Gauss>
inline size_t pairs_ws_upto(int64_t n, int64_t m) {
  size_t b = pairs_shape_ws_upto<Op, V, TPB, RT, Fam, false>(n, m);
  if constexpr (CanSplit<Op>::value) {
    const size_t s = pairs_shape_ws_upto<Op, V, TPB, RT, Fam, true>(n, m);
    b = s > b ? s : b;
  }
  return b;
}

// The same for every kernel family (the largest of their plans).
template <class Fn>
inline size_t largest_by_family(Fn bytes) {
  size_t b = 0;
  for (const int family : {(int)kGauss, (int)kLaplacian0, (int)kLaplacianMax}) {
    const size_t v = by_family(family, bytes);
    b = v > b ? v : b;
  }
  return b;
}
template <class Op, typename V, int TPB, int RT>
inline size_t pairs_ws_bytes_any(int64_t n, int64_t m) {
  return largest_by_family([&](auto fam) { return pairs_ws_bytes<Op, V, TPB, RT, decltype(fam)>(n, m); });
}
template <class Op, typename V, int TPB, int RT>
inline size_t pairs_ws_upto_any(int64_t n, int64_t m) {
  return largest_by_family([&](auto fam) { return pairs_ws_upto<Op, V, TPB, RT, decltype(fam)>(n, m); });
}

inline bool bad_kernel(int kernel) { return !(kernel == kGauss || (kernel >= kLaplacian0 && kernel <= kLaplacianMax)); }

// Frame of one kernel width. Coordinates are scaled so that the kernel's exponential is a power of two.
inline Frame make_frame(const double* origin, double sigma, int kernel) {
  Frame f = {};
  f.family = kernel;
  f.own = origin == nullptr;
  f.o0 = origin ? origin[0] : 0.0;
  f.o1 = origin ? origin[1] : 0.0;
  f.o2 = origin ? origin[2] : 0.0;
  constexpr double kLog2e = 1.44269504088896340736;
  if (kernel == kGauss) {
    f.s = kScale / sigma;
  } else {
    // P0 = lapPol of the order (Matern polynomial); P1 = (P0 - P0') / u and P2 = (P1 - P1') / u when the division
    // is exact (the constant terms cancel), else zero -- the reference's derivative tables for orders 0 and 1.
    static const double kP0[5][5] = {{1, 0, 0, 0, 0},
                                     {1, 1, 0, 0, 0},
                                     {1, 1, 1.0 / 3, 0, 0},
                                     {1, 1, 0.4, 1.0 / 15, 0},
                                     {1, 1, 3.0 / 7, 2.0 / 21, 1.0 / 105}};
    const int q = kernel - kLaplacian0;
    double c[3][5] = {};
    for (int k = 0; k < 5; ++k) c[0][k] = kP0[q][k];
    for (int r = 1; r < 3; ++r) {
      double d[5] = {};  // c[r-1] - derivative of c[r-1]
      for (int k = 0; k < 5; ++k) d[k] = c[r - 1][k] - (k + 1 < 5 ? (k + 1) * c[r - 1][k + 1] : 0.0);
      if (d[0] > -1e-12 && d[0] < 1e-12)  // exact in rationals; rounding leaves ~1e-17
        for (int k = 0; k < 4; ++k) c[r][k] = d[k + 1];
    }
    f.s = kLog2e / sigma;  // u' = log2(e) u, E = 2^-u'
    double pw = 1.0;
    for (int k = 0; k < 5; ++k) {
      for (int r = 0; r < 3; ++r) {
        f.dc[r][k] = c[r][k] * pw;
        f.lc[r][k] = (float)(c[r][k] * pw);
      }
      pw /= kLog2e;
    }
  }
  f.kappa = 1.0 / (f.s * sigma * sigma);
  f.inv_s2 = 1.0 / (sigma * sigma);
  return f;
}

// Launch an op with the pair kernel of its frame's family (P.f.family).
template <class Op, typename V, int TPB, int RT>
inline int run_pairs_k(const typename Op::Params& P, int64_t n, int64_t m, void* ws, size_t ws_bytes,
                       cudaStream_t stream) {
  return by_family(P.f.family, [&](auto fam) {
    return run_pairs<Op, V, TPB, RT, decltype(fam)>(P, n, m, ws, ws_bytes, stream);
  });
}

inline bool bad_sigma(double sigma) { return !(sigma > 0.0) || !(sigma < 1e300); }

// Source point in the frame (FP64 before the per-path conversion).
__device__ __forceinline__ void src_point(const double* __restrict__ p, int l, const Frame& f, double* o) {
  o[0] = (p[3 * l + 0] - f.o0) * f.s;
  o[1] = (p[3 * l + 1] - f.o1) * f.s;
  o[2] = (p[3 * l + 2] - f.o2) * f.s;
}

}  // namespace lddmm
