// Symmetric all-pairs kernel for self-interaction sums (targets and sources are the same n points).
//
// A sum out_k = sum_l f(k, l) over the same point set evaluates every unordered pair twice in pairs_kernel. When
// f(l, k) follows from the quantities of f(k, l) (the kernel value, the dot products and the difference vector, up to
// a sign), each unordered pair can be evaluated once and credited to both points. This kernel does that:
//
//  * The points are cut into blocks of B = TPB * RT (the target blocks of pairs_kernel) and tiles of TPB (its source
//    tiles); block j holds tiles RT j .. RT j + RT - 1. A unit is (target block i, source tile t) with t in a block
//    j >= i: the upper triangle in blocks. Units with j == i ("diagonal") evaluate their ordered pairs for the rows
//    only, like pairs_kernel; units with j > i evaluate each pair once and credit the row k (registers, as in
//    pairs_kernel) and the column l.
//  * Column credit without atomics: the warps of a CTA take the chunks of a tile in turn (one barrier per phase), and
//    lane λ processes record (λ + s) mod 32 of its chunk at step s: the 32 lanes read 32 different records. A record
//    is two sources in FP32, one in FP64 (SymStage). The record's column sums (over the lane's RT targets) are added to
//    an accumulator that moves one lane down after every step, so it follows its record around the warp; after 32
//    steps lane λ holds the warp's column sums of record λ of the chunk and adds them to the tile's column accumulators
//    in shared memory. At the end of the unit those hold the unit's column sums (TPB sources x NC), written as one
//    partial per (block i, source).
//  * Stream-K over the units in row-major order (as pairs_kernel over its units): a CTA's run of units of one row i
//    is a segment with compensated row sums (one partial slot, as in pairs_kernel). Point l of block b then has the
//    row slots of block b and b column partials (one from each block i < b); the epilogue sums both in a fixed order
//    in FP64 and hands them to Op::finalize_sym. Deterministic, no atomics.
//
// Units are balanced in count, not time: a column unit costs ~1.3x a diagonal one, and diagonal units are 1 in
// (number of blocks) per row, so the imbalance is a few percent. Padded targets (past n) carry zero payload fields,
// so their column credit is zero; padded sources carry zero fields, so their row credit is zero.
//
// Op interface (besides Params, finalize_sym):
//   NSS                                  source fields staged per source (scaled coordinates 0-2 first)
//   NR, NC                               row and column accumulators per point
//   SymTgt<V>                            register state of one target (V = F2: in both lanes)
//   load_target_sym<V>(P, i0, i1, v0, v1, SymTgt<V>&)  lanes from points i0, i1 (< n; the same here); v0 / v1 false =
//                                        padding (zero payload)
//   source_fields_sym(P, l, double* f)   NSS fields of source l (FP64)
//   pair_sym<COL, Fam, V>(const Frame&, const SymTgt<V>&, const V* s, V* row, V* col)
//   finalize_sym(P, i, const double* row, const double* col)
//
// FP64 (V = double): one source to a record, staged as doubles, row sums, column sums and column partials
// in FP64; the rotating accumulator costs two shuffles per field. What it saves is the exponential (about a third of
// an FP64 pair) and the shared products, on a pipe of half the FP32 rate.
#pragma once
#include "launch_config.cuh"
#include "lddmm_common.cuh"

#ifndef LDDMM_SYM
#define LDDMM_SYM 1  // 0: self-interaction sums evaluate every ordered pair (pairs_kernel)
#endif
#ifndef LDDMM_SYMX_UNROLL
#define LDDMM_SYMX_UNROLL 8  // unroll depth of pairs_kernel_symx's source loop (8: 1% faster than 4 at level 6)
#endif
#ifndef LDDMM_SYM_UNROLL
#define LDDMM_SYM_UNROLL 4  // unroll depth of the 32-step source loop of a chunk (4: 1% faster than 2 at level 6)
#endif

namespace lddmm {

constexpr int kSymUnroll = LDDMM_SYM_UNROLL;
constexpr int kSymxUnroll = LDDMM_SYMX_UNROLL;

// Shared-memory record of a staged source tile, and the column sums that ride around the warp while a chunk of sources
// is evaluated. In the symmetric kernels the lanes of a warp read different sources at every step (no broadcast), so
// what a load costs is its record.
//  * FP64: a record is one source; its column sums go around R = 32 lanes in 32 steps.
//  * FP32: the lanes of a packed value are two sources (r and r + R of a chunk of 2 R), and a 16-byte unit is two fields
//    of both, so an operand is used as it is loaded and a column sum moves as it is. With two targets to a value every
//    field is duplicated after its load, and every column sum is made a packed operand and its lanes added, at every
//    step: some 30 instructions per 4 targets that the pair does not need (40,962 points: forward / adjoint /
//    first-order adjoint step 772 / 1602 / 951 us, with two sources to a value 735 / 1478 / 840). The targets are the
//    duplicated side, once per segment, at the price of their registers.
//    R = 32 where a CTA's warps take all chunks of a tile in turn. R = 16 where each takes one chunk of 32 (SPLIT): the
//    column sums go around each half of the warp, and the halves, which hold different targets, meet at the end (whole
//    tiles with R = 16: 750 / 1503 / 862 us).
template <typename V, bool SPLIT>
constexpr int kSymRing = std::is_same<V, F2>::value && SPLIT ? 16 : 32;
template <int NF, int TPB, typename V, int R>
struct SymStage;
template <int NF, int TPB, int R>
struct SymStage<NF, TPB, double, R> {
  static constexpr int NQ = (NF + 1) / 2;  // 16-byte units
  static constexpr int kSlots = TPB;       // records of a tile
  static constexpr int kFields = 2 * NQ;   // size of the FP64 field buffer and of the operand array
  using T = double2;
  static __device__ __forceinline__ void store(T (*sm)[kSlots], int t, const double* fl) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) sm[q][t] = make_double2(fl[2 * q], fl[2 * q + 1]);
  }
  static __device__ __forceinline__ void load(const T (*sm)[kSlots], int rec, double* sv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double2 w = sm[q][rec];
      sv[2 * q] = w.x;
      sv[2 * q + 1] = w.y;
    }
  }
};
template <int NF, int TPB, int R>
struct SymStage<NF, TPB, F2, R> {
  static_assert(TPB % (2 * R) == 0, "tiles of whole chunks");
  static constexpr int NQ = (NF + 1) / 2;
  static constexpr int kSlots = TPB / 2;
  static constexpr int kFields = 2 * NQ;
  using T = float4;
  static __device__ __forceinline__ void store(T (*sm)[kSlots], int t, const double* fl) {
    const int rec = t / (2 * R) * R + t % R, half = t / R & 1;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      float* w = reinterpret_cast<float*>(&sm[q][rec]) + half;
      w[0] = (float)fl[2 * q];
      w[2] = (float)fl[2 * q + 1];
    }
  }
  static __device__ __forceinline__ void load(const T (*sm)[kSlots], int rec, F2* sv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const float4 w = sm[q][rec];
      sv[2 * q] = f2(w.x, w.y);
      sv[2 * q + 1] = f2(w.z, w.w);
    }
  }
};
// one step of the ring: `from` is the next lane of the R
template <int R>
__device__ __forceinline__ int ring_next(int lane) {
  return ((lane + 1) & (R - 1)) | (lane & ~(R - 1));
}
__device__ __forceinline__ double ring_move(double v, int from) { return __shfl_sync(0xffffffffu, v, from); }
__device__ __forceinline__ F2 ring_move(F2 v, int from) {
  float a, b;
  split(v, a, b);
  return f2(__shfl_sync(0xffffffffu, a, from), __shfl_sync(0xffffffffu, b, from));
}
// SPLIT, after the last step: the warp's column sum of source `lane` of its chunk of 32
__device__ __forceinline__ double ring_total(double v, int) { return v; }
__device__ __forceinline__ float ring_total(F2 v, int lane) {
  float a, b;
  split(v, a, b);
  const bool low = lane < 16;
  return (low ? a : b) + __shfl_xor_sync(0xffffffffu, low ? b : a, 16);
}
// whole tiles, after the last step: the sums added to the accumulators of chunk `chunk`
template <int TPB>
__device__ __forceinline__ void ring_add(double (&acc)[TPB], double v, int chunk, int lane) {
  acc[chunk * 32 + lane] += v;
}
template <int TPB>
__device__ __forceinline__ void ring_add(float (&acc)[TPB], F2 v, int chunk, int lane) {
  float a, b;
  split(v, a, b);
  acc[chunk * 64 + lane] += a;
  acc[chunk * 64 + 32 + lane] += b;
}
// Column accumulators of a CTA of whole tiles: warps that take the same chunk at the same time have their own.
template <typename V, int TPB>
struct SymChunks {
  static constexpr int kCount = TPB / (32 * VT<V>::kLanes);  // chunks of a tile
  static constexpr int kCopies = (TPB / 32) / kCount;
};

// Row sums of a tile as the compensated values hold them: FP32 two targets to a value (the lanes of each added), FP64
// one.
template <typename V, int RT>
struct SymRows;
template <int RT>
struct SymRows<double, RT> {
  static constexpr int kValues = RT;
  template <int NR>
  static __device__ __forceinline__ double value(const double (&acc)[RT][NR], int h, int c) { return acc[h][c]; }
};
template <int RT>
struct SymRows<F2, RT> {
  static constexpr int kValues = (RT + 1) / 2;
  template <int NR>
  static __device__ __forceinline__ F2 value(const F2 (&acc)[RT][NR], int h, int c) {
    return f2(VT<F2>::hsum(acc[2 * h][c]), 2 * h + 1 < RT ? VT<F2>::hsum(acc[2 * h + 1 < RT ? 2 * h + 1 : 0][c]) : 0.f);
  }
};

struct SymPlan {
  int nblk = 0, TT = 0, C = 0, S = 0;
  long long U = 0, wave = 1;  // units, resident CTAs
  size_t col_off = 0, ws_bytes = 0;
};

// row_bytes, col_bytes: size of one row / column partial
template <int TPB, int B>
inline SymPlan make_sym_plan(int64_t n, int nr, int nc, int ctas_per_sm, size_t row_bytes, size_t col_bytes) {
  using Geo = SymGeom<TPB, B>;
  SymPlan p;
  if (n <= 0) return p;
  p.nblk = (int)((n + B - 1) / B);
  p.TT = (int)((n + TPB - 1) / TPB);
  p.U = Geo::row_off(p.nblk, p.TT);
  const long long wave = p.wave = (long long)device_sm_count() * (ctas_per_sm > 0 ? ctas_per_sm : 1);
  // one resident wave of CTAs; up to half a wave more units run as one CTA each, so that no CTA takes two units while
  // others take one (forward step at 6,000 points, 576 units, 444 resident CTAs: 41.4 -> 31.7 us)
  p.C = (int)(2 * p.U < 3 * wave ? p.U : wave);
  p.S = sk_max_slots(p.TT, p.U, p.C);  // the longest row has TT units
  p.col_off = ((size_t)p.S * (size_t)nr * (size_t)n * row_bytes + 255) & ~(size_t)255;
  p.ws_bytes =
      p.col_off + (size_t)Geo::col_first((n + Geo::K - 1) / Geo::K) * (size_t)nc * (size_t)Geo::K * col_bytes;
  return p;
}

// Scratch that holds the plans of every n in (lo, hi]. A plan's slots are not monotone in n. With U units in nblk rows
// of at most TT (U >= nblk TT / 2) they are TT while every unit has a CTA of its own (2 U < 3 wave: slots x points <= TT
// nblk B <= 2 U B), and at most (TT - 1) wave / U + 2 beyond (slots x points <= 2 wave B + 2 n).
template <int TPB, int B>
inline size_t sym_plan_upto(int64_t lo, int64_t hi, int nr, int nc, int ctas_per_sm, size_t row_bytes,
                            size_t col_bytes) {
  if (hi <= lo) return 0;
  const SymPlan first = make_sym_plan<TPB, B>(lo + 1, nr, nc, ctas_per_sm, row_bytes, col_bytes);
  const SymPlan last = make_sym_plan<TPB, B>(hi, nr, nc, ctas_per_sm, row_bytes, col_bytes);
  int64_t points = 2 * first.wave * B + 2 * hi;
  if (2 * first.U < 3 * first.wave && points < 3 * first.wave * B) points = 3 * first.wave * B;
  if ((int64_t)last.TT * hi < points) points = (int64_t)last.TT * hi;
  const size_t rows = (size_t)points * (size_t)nr * row_bytes;
  return ((rows + 255) & ~(size_t)255) + (last.ws_bytes - last.col_off);
}

// Unroll depth of the source loop: the op's for the Gaussian in FP32, where it has one.
template <class Op, class = void>
struct SymUnrollOf : std::integral_constant<int, kSymUnroll> {};
template <class Op>
struct SymUnrollOf<Op, std::void_t<decltype(Op::kSymUnrollG)>> : std::integral_constant<int, Op::kSymUnrollG> {};
template <class Op, class Fam, typename V>
constexpr int kSymSteps =
    std::is_same<V, F2>::value && std::is_same<Fam, Gauss>::value ? SymUnrollOf<Op>::value : kSymUnroll;

// Ops whose column terms of a step are added up before they join the ring (Laplacian, whole tiles): a column sum of 4
// targets is a chain of 128 additions without that, and the second-order adjoint's error grew with it (pa-increment at
// 40,962 points 1.06 of what 2 targets to a packed value gave with 3 targets per thread, 0.75 with this and 4; 1917 and
// 1922 us).
template <class Op, class = void>
struct SymFresh : std::false_type {};
template <class Op>
struct SymFresh<Op, std::void_t<decltype(Op::kSymFresh)>> : std::bool_constant<Op::kSymFresh> {};

// One chunk of sources against the warp's targets; the column sums are back where they started in col.
template <class Op, int TPB, int RT, int R, bool COL, class Fam, typename V>
__device__ __forceinline__ void sym_chunk(const Frame& f, const typename Op::template SymTgt<V> (&tgt)[RT],
                                          const typename SymStage<Op::NSS, TPB, V, R>::T (*sm)[SymStage<Op::NSS, TPB, V, R>::kSlots],
                                          int chunk, V (&acc)[RT][Op::NR], V (&col)[Op::NC]) {
  using St = SymStage<Op::NSS, TPB, V, R>;
  constexpr bool FRESH = SymFresh<Op>::value && std::is_same<V, F2>::value && R == 32 && !std::is_same<Fam, Gauss>::value;
  constexpr int kUnroll = kSymSteps<Op, Fam, V>;
  const int lane = threadIdx.x & 31, from = ring_next<R>(lane);
#pragma unroll
  for (int c = 0; c < Op::NC; ++c) col[c] = VT<V>::zero();
#pragma unroll kUnroll
  for (int s = 0; s < R; ++s) {
    V sv[St::kFields];
    St::load(sm, chunk * R + ((lane + s) & (R - 1)), sv);
    if constexpr (COL && FRESH) {
      V step[Op::NC];
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) step[c] = VT<V>::zero();
#pragma unroll
      for (int g = 0; g < RT; ++g) Op::template pair_sym<COL, Fam, V>(f, tgt[g], sv, acc[g], step);
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) col[c] = ring_move(col[c] + step[c], from);
    } else {
#pragma unroll
      for (int g = 0; g < RT; ++g) Op::template pair_sym<COL, Fam, V>(f, tgt[g], sv, acc[g], col);
      if constexpr (COL) {
#pragma unroll
        for (int c = 0; c < Op::NC; ++c) col[c] = ring_move(col[c], from);
      }
    }
  }
}

template <class Op, int TPB, int RT, bool COL, class Fam, typename V>
__device__ __forceinline__ void sym_tile(const Frame& f, const typename Op::template SymTgt<V> (&tgt)[RT],
                                         const typename SymStage<Op::NSS, TPB, V, 32>::T (*sm)[SymStage<Op::NSS, TPB, V, 32>::kSlots],
                                         typename VT<V>::Scalar (*colacc)[Op::NC][TPB], V (&acc)[RT][Op::NR]) {
  using Ch = SymChunks<V, TPB>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int ph = 0; ph < Ch::kCount; ++ph) {
    const int chunk = (warp + ph) % Ch::kCount;
    V col[Op::NC];
    sym_chunk<Op, TPB, RT, 32, COL, Fam, V>(f, tgt, sm, chunk, acc, col);
    if constexpr (COL) {
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) ring_add<TPB>(colacc[warp / Ch::kCount][c], col[c], chunk, lane);
    }
    __syncthreads();  // the next phase hands this chunk (and its column accumulators) to another warp
  }
}

// minimum resident CTAs per SM: the op's for FP32, 2 (255 registers) from 6 targets per thread on; no register cap in
// FP64
template <class Op, typename V, int RT>
constexpr int kSymCtas = !std::is_same<V, F2>::value ? 1 : RT >= 6 ? 2 : Op::kSymMinCtas;

// SPLIT (small point sets): the warps of a CTA share its 32 RT targets and take one chunk of every tile each, instead
// of TPB RT targets and all chunks in turn. A unit is TPB / 32 times shorter and the triangle has that many times more
// units, which is what a set too small to fill the GPU needs: at 2,562 points a forward step's longest chain falls
// from 128 pair evaluations to 32 and its 462 units occupy every SM. The warps' row sums meet in shared memory at the
// end of a segment; a chunk's column sums are one warp's and go straight to the column partial.
template <class Op, int TPB, int RT, class Fam, typename V, bool SPLIT>
__global__ void __launch_bounds__(TPB, kSymCtas<Op, V, RT>)
    pairs_kernel_sym(const typename Op::Params P, int n, int nblk, int TT, long long U, int C,
                     typename VT<V>::Partial* __restrict__ row_ws, typename VT<V>::Scalar* __restrict__ col_ws) {
  constexpr int R = kSymRing<V, SPLIT>;
  using St = SymStage<Op::NSS, TPB, V, R>;
  using Rows = SymRows<V, RT>;
  constexpr int NR = Op::NR, NC = Op::NC, W = TPB / 32, H = Rows::kValues, L = VT<V>::kLanes;
  constexpr int TW = SPLIT ? 32 : TPB;  // targets a lane-group index apart
  constexpr int B = TW * RT;
  using Geo = SymGeom<TPB, B>;
  constexpr int K = Geo::K;
  static_assert(TPB % 32 == 0, "launch shape");
  __shared__ typename St::T sm[St::NQ][St::kSlots];
  constexpr int kCopies = SymChunks<V, TPB>::kCopies;
  __shared__ typename VT<V>::Scalar colacc[SPLIT ? 1 : kCopies][NC][SPLIT ? 1 : TPB];
  // compensated row sums of the segment, one private column per thread (H * NR * Comp<V>::kWords rows of TPB): dynamic
  // shared memory, so that 8 targets per thread may take more than the 48 KiB of static shared memory
  extern __shared__ __align__(16) unsigned char sym_dyn_smem[];
  V (*cs)[TPB] = reinterpret_cast<V (*)[TPB]>(sym_dyn_smem);
  __shared__ double org[3];
  const Frame& f = P.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  VT<V>::setup();  // the staging barrier of the first tile follows
  chain_wait();

  const long long u_end = sk_start(blockIdx.x + 1, U, C);
  long long u = sk_start(blockIdx.x, U, C);
  int i = u < u_end ? Geo::row_of(u, nblk, TT) : 0;
  while (u < u_end) {
    const long long off = Geo::row_off(i, TT);
    const int first = Geo::first_tile(i), cnt = TT - first;
    const int t0 = (int)(u - off);
    const int t1 = (int)((u_end - off) < cnt ? (u_end - off) : cnt);
    const int slot = (int)blockIdx.x - sk_cta_of(off, U, C);
    const int base = i * B + (SPLIT ? lane : (int)threadIdx.x);

    typename Op::template SymTgt<V> tgt[RT];
    // SPLIT: raw coordinates, loaded before the other fields; with nine of those (the second-order adjoint) and more than
    // two targets they are loaded again when the origin is known (us held | again: adjoint of 2,562 points, 4 targets,
    // 17.8 | 17.5, of 642, 2 targets, 9.5 | 9.75; forward of 2,562 12.4 | 13.0)
    constexpr bool kHold = SPLIT && (Op::NSS < 12 || RT <= 2);
    double xt[kHold ? RT : 1][3];
    if constexpr (kHold) {
#pragma unroll
      for (int g = 0; g < RT; ++g) {
        const int k = base + g * TW, kc = k < n ? k : n - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) xt[g][c] = P.x[3 * (size_t)kc + c];
      }
    }
#pragma unroll
    for (int g = 0; g < RT; ++g) {
      const int k = base + g * TW, kc = k < n ? k : n - 1;
      Op::template load_target_sym<V>(P, kc, kc, k < n, k < n, tgt[g]);
    }
    if constexpr (SPLIT) {
      // the segment's origin, a coordinate per warp, while the targets' other fields arrive; then their coordinates
      static_assert(W >= 3, "a warp per coordinate");
      if (warp < 3) {
        const int last = i * B + B < n ? i * B + B - 1 : n - 1, count = last - i * B + 1;
        constexpr int M = RT / 2;  // the middle 32 points, of a short block the first
        const bool mid = count >= 32 * (M + 1);
        double x;
        if constexpr (kHold) {
          const double x0 = warp == 0 ? xt[0][0] : warp == 1 ? xt[0][1] : xt[0][2];
          const double xm = warp == 0 ? xt[M][0] : warp == 1 ? xt[M][1] : xt[M][2];
          x = mid ? xm : x0;
        } else {
          const int k = base + (mid ? M * TW : 0);
          x = P.x[3 * (size_t)(k < n ? k : n - 1) + warp];
        }
        const double o = segment_origin(f, P.x, i * B, last, warp, count >= 32, x);
        if (lane == 0) org[warp] = o;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < RT; ++g) {
        if constexpr (kHold) {
          tgt[g].y0 = VT<V>::dup((xt[g][0] - org[0]) * f.s);
          tgt[g].y1 = VT<V>::dup((xt[g][1] - org[1]) * f.s);
          tgt[g].y2 = VT<V>::dup((xt[g][2] - org[2]) * f.s);
        } else {
          const int k = base + g * TW, kc = k < n ? k : n - 1;
          tgt[g].y0 = tgt_coord<V>(P.x, kc, kc, 0, org[0], f.s);
          tgt[g].y1 = tgt_coord<V>(P.x, kc, kc, 1, org[1], f.s);
          tgt[g].y2 = tgt_coord<V>(P.x, kc, kc, 2, org[2], f.s);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < H * NR; ++c) {
      Comp<V> z;
      z.zero();
      z.template store<TPB>(cs, c, threadIdx.x);
    }

    for (int tt = t0; tt < t1; ++tt) {
      const int t = first + tt;                // absolute source tile
      const bool diag = tt < Geo::kSpan;       // tile of the block's own superblock: rows only
      {
        const int l = t * TPB + threadIdx.x;
        double fl[St::kFields];
#pragma unroll
        for (int q = 0; q < St::kFields; ++q) fl[q] = 0.0;
        if (l < n) {
          if constexpr (SPLIT)
            Op::source_fields_sym(with_origin(P, org), l, fl);
          else
            Op::source_fields_sym(P, l, fl);
        }
        St::store(sm, threadIdx.x, fl);
        if constexpr (!SPLIT) {
#pragma unroll
          for (int w = 0; w < kCopies; ++w)
#pragma unroll
            for (int c = 0; c < NC; ++c) colacc[w][c][threadIdx.x] = 0;
        }
      }
      __syncthreads();
      V acc[RT][NR];
#pragma unroll
      for (int g = 0; g < RT; ++g)
#pragma unroll
        for (int c = 0; c < NR; ++c) acc[g][c] = VT<V>::zero();
      // column partial of (row block i, tile t), field stride K. Held over the tile, except where the six sums and the
      // order-4 profile leave no register for it (40,962 points: forward step 1216 -> 1197 us, first-order adjoint
      // 1299 -> 1286; held elsewhere: at 20,000 points of order 3 the first-order adjoint is 309 us against 324).
      auto column_base = [&]() {
        const int J = (int)(t * (long long)TPB / K);
        return (size_t)(Geo::col_first(J) + i) * NC * K + (size_t)(t * (long long)TPB - (long long)K * J) + threadIdx.x;
      };
      constexpr bool kHeld = SPLIT || NC < 6 || VT<V>::kLanes == 1 || !std::is_same<Fam, Laplacian4>::value;
      const size_t cb = kHeld ? column_base() : 0;
      if constexpr (SPLIT) {
        V col[NC];
        if (diag) {
          sym_chunk<Op, TPB, RT, R, false, Fam, V>(f, tgt, sm, warp, acc, col);
        } else {
          sym_chunk<Op, TPB, RT, R, true, Fam, V>(f, tgt, sm, warp, acc, col);
#pragma unroll
          for (int c = 0; c < NC; ++c) col_ws[cb + (size_t)c * K] = ring_total(col[c], lane);
        }
      } else if (diag) {
        sym_tile<Op, TPB, RT, false, Fam, V>(f, tgt, sm, colacc, acc);
      } else {
        sym_tile<Op, TPB, RT, true, Fam, V>(f, tgt, sm, colacc, acc);
      }
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          Comp<V> m;
          m.template load<TPB>(cs, h * NR + c, threadIdx.x);
          m.merge(Rows::value(acc, h, c));
          m.template store<TPB>(cs, h * NR + c, threadIdx.x);
        }
      if constexpr (SPLIT) {
        __syncthreads();  // every warp has read the tile and left its row sums
      } else if (!diag) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          typename VT<V>::Scalar v = colacc[0][c][threadIdx.x];
#pragma unroll
          for (int w = 1; w < kCopies; ++w) v += colacc[w][c][threadIdx.x];
          col_ws[(kHeld ? cb : column_base()) + (size_t)c * K] = v;
        }
      }
      // (not SPLIT) the last phase barrier of sym_tile orders every read of sm and colacc before the next staging
    }

    if (SPLIT && u + (t1 - t0) >= u_end) chain_go();
    if constexpr (SPLIT) {
      // the block's row sums: field c of the lanes' targets by warp c mod W, over the W warps in order
#pragma unroll
      for (int h = 0; h < H; ++h)
        for (int c = warp; c < NR; c += W) {
          double sum[L];
#pragma unroll
          for (int k = 0; k < L; ++k) sum[k] = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            Comp<V> m;
            m.template load<TPB>(cs, h * NR + c, w * 32 + lane);
#pragma unroll
            for (int k = 0; k < L; ++k) sum[k] += partial_value(m.partial(k));
          }
#pragma unroll
          for (int k = 0; k < L; ++k) {
            const int idx = base + (h * L + k) * TW;
            if (h * L + k < RT && idx < n)
              row_ws[((size_t)slot * NR + c) * (size_t)n + idx] = VT<V>::to_partial(sum[k]);
          }
        }
      __syncthreads();  // the next segment clears the sums
    } else {
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const int idx = base + (h * L + k) * TW;
          if (h * L + k < RT && idx < n) {
#pragma unroll
            for (int c = 0; c < NR; ++c) {
              Comp<V> m;
              m.template load<TPB>(cs, h * NR + c, threadIdx.x);
              row_ws[((size_t)slot * NR + c) * (size_t)n + idx] = m.partial(k);
            }
          }
        }
    }
    u += t1 - t0;
    ++i;
  }
}

// Epilogue: the row slots of the point's block and its column partials, in FP64, summed by TPP threads per point
// (TPP a power of two <= 32). A CTA of kFinThreads threads takes P = kFinThreads / TPP consecutive points; thread
// (j, p) -- p = threadIdx % P, j = threadIdx / P -- sums slots j, j + TPP, ... and column partials j, j + TPP, ...
// of point p (consecutive threads read consecutive points: coalesced), and thread (0, p) adds the TPP sums in the
// order j = 0, 1, ... from shared memory and applies the op's epilogue. Every addition's order is fixed by (point,
// TPP): deterministic. With one thread per point, a point's slots and partials are one serial chain of up to tens
// of dependent loads (at 2,562 points: 11 CTAs, ~11 us, latency-bound); several threads shorten the chain and
// spread the points over more CTAs.
template <class Op, int TPB, int B, typename V>
__global__ void __launch_bounds__(kFinThreads)
    finalize_sym_kernel(const typename Op::Params P, int n, int nblk, int TT, long long U, int C,
                        const typename VT<V>::Partial* __restrict__ row_ws,
                        const typename VT<V>::Scalar* __restrict__ col_ws, int tpp) {
  using Geo = SymGeom<TPB, B>;
  constexpr int NV = Op::NR + Op::NC, K = Geo::K;
  __shared__ double red[NV][kFinThreads];
  const int np = kFinThreads / tpp;
  const int p = threadIdx.x % np, j = threadIdx.x / np;
  const int idx = blockIdx.x * np + p;
  const bool live = idx < n;
  const int b = live ? idx / B : 0, J = live ? idx / K : 0, r = live ? idx - J * K : 0;
  const int nslot =
      live ? sk_cta_of(Geo::row_off(b + 1, TT) - 1, U, C) - sk_cta_of(Geo::row_off(b, TT), U, C) + 1 : 0;
  const int ncol = live ? J * Geo::kShare : 0;
  const size_t cfirst = (size_t)Geo::col_first(J) * Op::NC * K + r;
  chain_wait();
  double v[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) v[c] = 0.0;
  for (int s = j; s < nslot; s += tpp)
#pragma unroll
    for (int c = 0; c < Op::NR; ++c) v[c] += partial_value(row_ws[((size_t)s * Op::NR + c) * (size_t)n + idx]);
  for (int q = j; q < ncol; q += tpp)
#pragma unroll
    for (int c = 0; c < Op::NC; ++c) v[Op::NR + c] += (double)col_ws[cfirst + ((size_t)q * Op::NC + c) * K];
  finalize_meet<NV>(red, np, tpp, p, j, v);
  if (live && j == 0) Op::finalize_sym(P, idx, v, v + Op::NR);
}

// The chain a point's epilogue sums: its block's slots and the column partials of the blocks before it.
inline int sym_finalize_tpp(const SymPlan& p) { return finalize_tpp(p.S + p.nblk); }

// Dynamic shared memory of pairs_kernel_sym (its compensated row sums).
template <class Op, int TPB, int RT, typename V>
constexpr size_t sym_dyn_smem_bytes() {
  return (size_t)SymRows<V, RT>::kValues * Op::NR * Comp<V>::kWords * TPB * sizeof(V);
}

// Declare the kernel's dynamic shared memory, once per device (the attribute belongs to the device's context):
// without it static + dynamic shared memory may not exceed 48 KiB. Returns false when the device refuses.
template <class Op, int TPB, int RT, class Fam = Gauss, typename V = F2, bool SPLIT = false>
inline bool sym_prepare() {
  static signed char state[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (dev < 0 || dev >= 64) return false;
  if (state[dev] == 0) {
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&pairs_kernel_sym<Op, TPB, RT, Fam, V, SPLIT>),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sym_dyn_smem_bytes<Op, TPB, RT, V>());
    if (e != cudaSuccess) cudaGetLastError();
    state[dev] = e == cudaSuccess ? 1 : -1;
  }
  return state[dev] > 0;
}

template <class Op, int TPB, int RT, class Fam = Gauss, typename V = F2, bool SPLIT = false>
inline int sym_ctas_per_sm() {
  static int cached = 0;
  if (cached == 0) {
    sym_prepare<Op, TPB, RT, Fam, V, SPLIT>();
    int c = resident_ctas(reinterpret_cast<const void*>(&pairs_kernel_sym<Op, TPB, RT, Fam, V, SPLIT>), TPB,
                          sym_dyn_smem_bytes<Op, TPB, RT, V>());
    cached = c > 0 ? c : 2;
  }
  return cached;
}

template <class Op, int TPB, int RT, class Fam = Gauss, typename V = F2, bool SPLIT = false>
inline SymPlan sym_plan(int64_t n) {
  return make_sym_plan<TPB, (SPLIT ? 32 : TPB) * RT>(n, Op::NR, Op::NC, sym_ctas_per_sm<Op, TPB, RT, Fam, V, SPLIT>(),
                                sizeof(typename VT<V>::Partial), sizeof(typename VT<V>::Scalar));
}

template <class Op, int TPB, int RT, class Fam = Gauss, typename V = F2, bool SPLIT = false>
inline size_t sym_ws_bytes(int64_t n) {
  return sym_plan<Op, TPB, RT, Fam, V, SPLIT>(n).ws_bytes;
}

template <class Op, int TPB, int RT, class Fam = Gauss, typename V = F2, bool SPLIT = false>
inline int run_pairs_sym(const typename Op::Params& P, int64_t n, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (n <= 0) return kOk;
  if (n > INT32_MAX / 4) return kInvalidArgument;
  const SymPlan plan = sym_plan<Op, TPB, RT, Fam, V, SPLIT>(n);
  if (plan.ws_bytes > ws_bytes) return kWorkspaceTooSmall;
  if (ws == nullptr) return kInvalidArgument;
  if (!sym_prepare<Op, TPB, RT, Fam, V, SPLIT>()) return kLaunchFailure;
  auto* row_ws = reinterpret_cast<typename VT<V>::Partial*>(ws);
  auto* col_ws = reinterpret_cast<typename VT<V>::Scalar*>(reinterpret_cast<char*>(ws) + plan.col_off);
  launch_chained(pairs_kernel_sym<Op, TPB, RT, Fam, V, SPLIT>, plan.C, TPB, sym_dyn_smem_bytes<Op, TPB, RT, V>(),
                 stream, P, (int)n, plan.nblk, plan.TT, plan.U, plan.C, row_ws, col_ws);
  const int tpp = sym_finalize_tpp(plan);
  launch_chained(finalize_sym_kernel<Op, TPB, (SPLIT ? 32 : TPB) * RT, V>, finalize_grid(n, tpp), kFinThreads, 0,
                 stream, P, (int)n, plan.nblk, plan.TT, plan.U, plan.C, row_ws, col_ws, tpp);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}


// Launch shapes. Each symmetric op names its rule (Op::Shape): up to where 4 targets per thread with the split are used
// in FP32 (8 follow), the targets per thread of whole tiles (0: another kernel has them), each for the Gaussian and the
// Laplacian, and the FP64 shape of whole tiles (launch_config.cuh has the measurements).
template <int SPLIT4_N, int SPLIT4_N_LAP, int RT, int RT_LAP, int TPB64, int RT64>
struct SymRule {
  static constexpr int64_t kSplit4 = SPLIT4_N, kSplit4Lap = SPLIT4_N_LAP;
  static constexpr int kRt = RT, kRtLap = RT_LAP, kTpb64 = TPB64, kRt64 = RT64;
};
template <int TPB, int RT, bool SPLIT>
struct SymShape {
  static constexpr int kTpb = TPB, kRt = RT;
  static constexpr bool kSplit = SPLIT;
};

// Whether the units of a plan fill its resident CTAs: at least 95% of the rounds that they take.
inline bool sym_full(const SymPlan& p) {
  const long long rounds = (p.U + p.wave - 1) / p.wave;
  return 20 * p.U >= 19 * rounds * p.wave;
}
// Whole tiles or the split, in FP32: see kSplitN.
template <class PlanFn>
inline bool sym_whole(int64_t n, PlanFn plan) {
  return n > kSplitN || (n > kWholeN && sym_full(plan()));
}

// fn(SymShape{}) with the shape of n points.
template <class Op, typename V, class Fam, class Fn>
inline auto sym_shape(int64_t n, Fn fn) {
  using R = typename Op::Shape;
  constexpr bool kG = std::is_same<Fam, Gauss>::value;
  if constexpr (std::is_same<V, double>::value) {
    if (n <= kSplit1N64) return fn(SymShape<128, 1, true>{});
    if (n <= (kG ? kSplit2N64 : kSplit2N64Lap)) return fn(SymShape<128, 2, true>{});
    return fn(SymShape<R::kTpb64, R::kRt64, false>{});
  } else {
    constexpr int kRt = kG ? R::kRt : R::kRtLap;
    constexpr int64_t kSplit4 = kG ? R::kSplit4 : R::kSplit4Lap;
    if (n <= kSplit2N) return fn(SymShape<128, 2, true>{});
    if constexpr (kRt > 0) {
      if (sym_whole(n, [&] { return sym_plan<Op, 128, kRt, Fam, V, false>(n); }))
        return fn(SymShape<128, kRt, false>{});
    }
    if constexpr (kSplit4 < kSplitN) {
      if (n > kSplit4) return fn(SymShape<128, 8, true>{});
    }
    return fn(SymShape<128, 4, true>{});
  }
}

// Whether a self-sum takes the symmetric kernel: always in FP32. In FP64 the column partials of the unsplit shape are
// bounded at 2 GiB (150,000 points for the six-field steps): they grow with n^2, and larger sets keep the ordered-pair
// kernel, whose scratch does not.
constexpr int64_t kSym64MaxColBytes = int64_t(2) << 30;
template <class Op, typename V>
inline int64_t sym_max_n() {
  if (LDDMM_SYM == 0) return 0;
  if (std::is_same<V, F2>::value) return INT32_MAX / 4;
  constexpr int64_t B = Op::Shape::kTpb64 * Op::Shape::kRt64;
  constexpr int64_t tri = kSym64MaxColBytes / (int64_t)(Op::NC * B * sizeof(double));  // blocks: tri(nblk) <= this
  static const int64_t nblk = [] {
    int64_t k = 1;
    while (sym_tri(k + 1) <= tri) ++k;
    return k;
  }();
  return nblk * B;
}
template <class Op, typename V>
inline bool sym_takes(int64_t n) {
  return n > 0 && n <= sym_max_n<Op, V>();
}

template <class Op, typename V, class Fam>
inline size_t sym_scratch_fam(int64_t n) {
  return sym_shape<Op, V, Fam>(n, [&](auto sh) {
    return sym_ws_bytes<Op, decltype(sh)::kTpb, decltype(sh)::kRt, Fam, V, decltype(sh)::kSplit>(n);
  });
}
// Scratch of one launch.
template <class Op, typename V>
inline size_t sym_scratch(int64_t n, int family) {
  return by_family(family, [&](auto fam) { return sym_scratch_fam<Op, V, decltype(fam)>(n); });
}
// Scratch for every point count up to n: each shape over the range that it may be launched in (between kWholeN and
// kSplitN either shape may be the one).
template <class Op, typename V, class Fam>
inline size_t sym_scratch_upto_fam(int64_t n) {
  using R = typename Op::Shape;
  constexpr bool kG = std::is_same<Fam, Gauss>::value;
  n = n < sym_max_n<Op, V>() ? n : sym_max_n<Op, V>();
  size_t b = 0;
  auto range = [&](auto sh, int64_t lo, int64_t hi) {
    using Sh = decltype(sh);
    const size_t v = sym_plan_upto<Sh::kTpb, (Sh::kSplit ? 32 : Sh::kTpb) * Sh::kRt>(
        lo, n < hi ? n : hi, Op::NR, Op::NC, sym_ctas_per_sm<Op, Sh::kTpb, Sh::kRt, Fam, V, Sh::kSplit>(),
        sizeof(typename VT<V>::Partial), sizeof(typename VT<V>::Scalar));
    b = v > b ? v : b;
  };
  if constexpr (std::is_same<V, double>::value) {
    constexpr int64_t kSplit2 = kG ? kSplit2N64 : kSplit2N64Lap;
    range(SymShape<128, 1, true>{}, 0, kSplit1N64);
    range(SymShape<128, 2, true>{}, kSplit1N64, kSplit2);
    range(SymShape<R::kTpb64, R::kRt64, false>{}, kSplit2, n);
  } else {
    constexpr int kRt = kG ? R::kRt : R::kRtLap;
    constexpr int64_t kSplit4 = kG ? R::kSplit4 : R::kSplit4Lap;
    range(SymShape<128, 2, true>{}, 0, kSplit2N);
    if constexpr (kRt > 0) {
      range(SymShape<128, kRt, false>{}, kWholeN, kSplitN);
      range(SymShape<128, kRt, false>{}, kSplitN, n);
    }
    if constexpr (kSplit4 < kSplitN) range(SymShape<128, 8, true>{}, kSplit4, kSplitN);
    range(SymShape<128, 4, true>{}, kSplit2N, kSplit4);
  }
  return b;
}
template <class Op, typename V>
inline size_t sym_scratch_upto(int64_t n) {
  return largest_by_family([&](auto fam) { return sym_scratch_upto_fam<Op, V, decltype(fam)>(n); });
}

template <class Op, typename V, class Fam>
inline int run_sym_fam(const typename Op::Params& P, int64_t n, void* ws, size_t wsb, cudaStream_t st) {
  return sym_shape<Op, V, Fam>(n, [&](auto sh) {
    return run_pairs_sym<Op, decltype(sh)::kTpb, decltype(sh)::kRt, Fam, V, decltype(sh)::kSplit>(P, n, ws, wsb, st);
  });
}
// Launch of a symmetric op, for the kernel family of its frame.
template <class Op, typename V>
inline int run_sym(const typename Op::Params& P, int64_t n, void* ws, size_t wsb, cudaStream_t st) {
  return by_family(P.f.family, [&](auto fam) { return run_sym_fam<Op, V, decltype(fam)>(P, n, ws, wsb, st); });
}

// ---------------------------------------------------------------------------------------------------------
// Expanded-distance form of the symmetric kernel, for sums whose pair term is the kernel value times a payload of
// the source (K a over one point set: out_k = sum_l e_kl a_l, so the mirrored term of l is e_kl a_k).
//
// As in pairs_kernel_x, the coordinates of a unit are taken relative to the centre of its row block i (box centre
// of the block's TPB * RT points, scaled): e_kl = f_k w_kl with f_k = 2^-|y_k|^2 and w_kl = 2^-(|x_l|^2 - 2 y_k.x_l),
// the bracket being three packed FMAs from the staged fields (-2 x_l, |x_l|^2). The row sums of k accumulate
// w_kl a_l and are multiplied by f_k (FP64) when the segment's partial is written; the column payload of target k is
// f_k a_k, so the column sums accumulate w_kl f_k a_k = e_kl a_k directly. 9 FP32 lane-ops and one ex2 per
// unordered pair (against 6 + 1 per ordered pair, i.e. 12 + 2, for pairs_kernel_x). Row blocks whose radius^2
// (scaled units) exceeds kExpandR2 use the difference form (e from |y - x|^2, payload a_k; 12 + 1), chosen per
// segment. Everything else -- the unit triangle, the rotating column accumulators, the stream-K split, the partial
// layouts and finalize_sym_kernel -- is pairs_kernel_sym's.
//
// Op interface: Params, NP (payload fields; NR = NC = NP), kSymMinCtas, point(P, i, double* c) (coordinates of
// point i), payload(P, i, double* p), finalize_sym(P, i, row, col).
// ---------------------------------------------------------------------------------------------------------
template <class Op, int TPB, int RT, bool COL, bool X>
__device__ __forceinline__ void symx_tile(const F2 (&yt)[RT][3], const F2 (&tp)[RT][Op::NP],
                                          const float4 (*sm)[TPB / 2], float (*colacc)[Op::NP][TPB],
                                          F2 (&acc)[RT][Op::NP]) {
  using St = SymStage<4 + Op::NP, TPB, F2, 32>;
  using Ch = SymChunks<F2, TPB>;
  constexpr int NP = Op::NP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int ph = 0; ph < Ch::kCount; ++ph) {
    const int chunk = (warp + ph) % Ch::kCount;
    const int from = ring_next<32>(lane);
    F2 col[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c) col[c] = VT<F2>::zero();
#pragma unroll kSymxUnroll
    for (int s = 0; s < 32; ++s) {
      F2 sv[St::kFields];
      St::load(sm, chunk * 32 + ((lane + s) & 31), sv);
#pragma unroll
      for (int g = 0; g < RT; ++g) {
        F2 arg;
        if constexpr (X) {
          arg = fma(yt[g][2], sv[2], sv[3]);  // |x|^2 - 2 y.x
          arg = fma(yt[g][1], sv[1], arg);
          arg = fma(yt[g][0], sv[0], arg);
        } else {
          const F2 d0 = yt[g][0] - sv[0], d1 = yt[g][1] - sv[1], d2 = yt[g][2] - sv[2];
          arg = fma(d2, d2, fma(d1, d1, d0 * d0));
        }
        const F2 e = VT<F2>::expneg(arg);
#pragma unroll
        for (int c = 0; c < NP; ++c) acc[g][c] = fma(e, sv[4 + c], acc[g][c]);
        if constexpr (COL) {
#pragma unroll
          for (int c = 0; c < NP; ++c) col[c] = fma(e, tp[g][c], col[c]);
        }
      }
      if constexpr (COL) {
#pragma unroll
        for (int c = 0; c < NP; ++c) col[c] = ring_move(col[c], from);
      }
    }
    if constexpr (COL) {
#pragma unroll
      for (int c = 0; c < NP; ++c) ring_add<TPB>(colacc[warp / Ch::kCount][c], col[c], chunk, lane);
    }
    __syncthreads();  // the next phase hands this chunk (and its column accumulators) to another warp
  }
}

template <class Op, int TPB, int RT>
__global__ void __launch_bounds__(TPB, Op::kSymMinCtas)
    pairs_kernel_symx(const typename Op::Params P, int n, int nblk, int TT, long long U, int C,
                      float2* __restrict__ row_ws, float* __restrict__ col_ws) {
  using St = SymStage<4 + Op::NP, TPB, F2, 32>;
  using Rows = SymRows<F2, RT>;
  constexpr int NP = Op::NP, H = Rows::kValues;
  constexpr int B = TPB * RT;
  using Geo = SymGeom<TPB, B>;
  static_assert(TPB % 32 == 0, "launch shape");
  __shared__ float4 sm[St::NQ][TPB / 2];
  constexpr int kCopies = SymChunks<F2, TPB>::kCopies;
  __shared__ float colacc[kCopies][NP][TPB];
  __shared__ float red[6][TPB / 32];
  extern __shared__ __align__(16) unsigned char sym_dyn_smem[];
  F2 (*cs)[TPB] = reinterpret_cast<F2 (*)[TPB]>(sym_dyn_smem);  // compensated row sums, H * NP * 2 rows
  const Frame& f = P.f;
  const double fo[3] = {f.o0, f.o1, f.o2};
  chain_wait();

  const long long u_end = sk_start(blockIdx.x + 1, U, C);
  long long u = sk_start(blockIdx.x, U, C);
  int i = u < u_end ? Geo::row_of(u, nblk, TT) : 0;
  while (u < u_end) {
    const long long off = Geo::row_off(i, TT);
    const int cnt = TT - RT * i;
    const int t0 = (int)(u - off);
    const int t1 = (int)((u_end - off) < cnt ? (u_end - off) : cnt);
    const int slot = (int)blockIdx.x - sk_cta_of(off, U, C);
    const int base = i * B + threadIdx.x;

    // box and centre of row block i (every CTA working on it derives the same ones)
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int t = 0; t < RT; ++t) {
      int k = base + t * TPB;
      k = k < n ? k : n - 1;
      double y[3];
      Op::point(P, k, y);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float v = (float)((y[c] - fo[c]) * f.s);
        lo[c] = fminf(lo[c], v);
        hi[c] = fmaxf(hi[c], v);
      }
    }
    block_box<TPB>(lo, hi, red);  // its barrier also orders the previous segment's last reads of sm and cs
    float ob[3], rb2 = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ob[c] = 0.5f * (lo[c] + hi[c]);
      const float h = 0.5f * (hi[c] - lo[c]);
      rb2 = fmaf(h, h, rb2);
    }
    const bool expand = rb2 <= kExpandR2;  // uniform over the CTA

    F2 yt[RT][3], tp[RT][NP];
#pragma unroll
    for (int g = 0; g < RT; ++g) {
      const int k = base + g * TPB;
      double y[3], pay[NP], q = 0.0;
      Op::point(P, k < n ? k : n - 1, y);
      Op::payload(P, k < n ? k : n - 1, pay);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float r = (float)((y[c] - fo[c]) * f.s - (double)ob[c]);
        yt[g][c] = f2(r, r);
        q += (double)r * (double)r;
      }
      // column payload: f_k a_k (expanded form) or a_k; padded targets carry none
      const double fk = k < n ? (expand ? exp2(-q) : 1.0) : 0.0;
#pragma unroll
      for (int c = 0; c < NP; ++c) tp[g][c] = VT<F2>::dup(fk * pay[c]);
    }
#pragma unroll
    for (int c = 0; c < H * NP; ++c) {
      Comp<F2> z;
      z.zero();
      z.template store<TPB>(cs, c, threadIdx.x);
    }

    for (int tt = t0; tt < t1; ++tt) {
      const int t = RT * i + tt;  // absolute source tile
      const bool diag = tt < RT;  // tile of block i itself: rows only
      {
        const int l = t * TPB + threadIdx.x;
        double fl[St::kFields];
#pragma unroll
        for (int q = 0; q < St::kFields; ++q) fl[q] = 0.0;
        if (l < n) {
          double xr[3], r2 = 0.0;
          Op::point(P, l, xr);
          Op::payload(P, l, fl + 4);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float xc = (float)((xr[c] - fo[c]) * f.s - (double)ob[c]);
            r2 += (double)xc * (double)xc;
            fl[c] = expand ? -2.0 * (double)xc : (double)xc;
          }
          fl[3] = r2;
        }
        St::store(sm, threadIdx.x, fl);
#pragma unroll
        for (int w = 0; w < kCopies; ++w)
#pragma unroll
          for (int c = 0; c < NP; ++c) colacc[w][c][threadIdx.x] = 0.f;
      }
      __syncthreads();
      F2 acc[RT][NP];
#pragma unroll
      for (int g = 0; g < RT; ++g)
#pragma unroll
        for (int c = 0; c < NP; ++c) acc[g][c] = VT<F2>::zero();
      if (expand) {
        if (diag)
          symx_tile<Op, TPB, RT, false, true>(yt, tp, sm, colacc, acc);
        else
          symx_tile<Op, TPB, RT, true, true>(yt, tp, sm, colacc, acc);
      } else {
        if (diag)
          symx_tile<Op, TPB, RT, false, false>(yt, tp, sm, colacc, acc);
        else
          symx_tile<Op, TPB, RT, true, false>(yt, tp, sm, colacc, acc);
      }
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          Comp<F2> m;
          m.template load<TPB>(cs, h * NP + c, threadIdx.x);
          m.merge(Rows::value(acc, h, c));
          m.template store<TPB>(cs, h * NP + c, threadIdx.x);
        }
      if (!diag) {
        const int j = t / RT;
        const size_t cb = (size_t)(Geo::col_first(j) + i) * NP * B + (size_t)(t - RT * j) * TPB + threadIdx.x;
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          float v = colacc[0][c][threadIdx.x];
#pragma unroll
          for (int w = 1; w < kCopies; ++w) v += colacc[w][c][threadIdx.x];
          col_ws[cb + (size_t)c * B] = v;
        }
      }
      // the last phase barrier of symx_tile orders every read of sm and colacc before the next tile's staging
    }

#pragma unroll
    for (int g = 0; g < RT; ++g) {
      const int idx = base + g * TPB;
      if (idx < n) {
        double y2 = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double yr = VT<F2>::lane(yt[g][c], 0);
          y2 += yr * yr;
        }
        const double fac = expand ? exp2(-y2) : 1.0;
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          Comp<F2> m;
          m.template load<TPB>(cs, (g / 2) * NP + c, threadIdx.x);
          row_ws[((size_t)slot * NP + c) * (size_t)n + idx] = VT<F2>::to_partial(partial_value(m.partial(g & 1)) * fac);
        }
      }
    }
    u += t1 - t0;
    ++i;
  }
}

template <class Op, int TPB, int RT>
constexpr size_t symx_dyn_smem_bytes() {
  return (size_t)SymRows<F2, RT>::kValues * Op::NP * Comp<F2>::kWords * TPB * sizeof(F2);
}

template <class Op, int TPB, int RT>
inline bool symx_prepare() {
  static signed char state[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (dev < 0 || dev >= 64) return false;
  if (state[dev] == 0) {
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&pairs_kernel_symx<Op, TPB, RT>),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)symx_dyn_smem_bytes<Op, TPB, RT>());
    if (e != cudaSuccess) cudaGetLastError();
    state[dev] = e == cudaSuccess ? 1 : -1;
  }
  return state[dev] > 0;
}

template <class Op, int TPB, int RT>
inline int symx_ctas_per_sm() {
  static int cached = 0;
  if (cached == 0) {
    symx_prepare<Op, TPB, RT>();
    int c = resident_ctas(reinterpret_cast<const void*>(&pairs_kernel_symx<Op, TPB, RT>), TPB,
                          symx_dyn_smem_bytes<Op, TPB, RT>());
    cached = c > 0 ? c : 2;
  }
  return cached;
}

template <class Op, int TPB, int RT>
inline SymPlan symx_plan(int64_t n) {
  return make_sym_plan<TPB, TPB * RT>(n, Op::NP, Op::NP, symx_ctas_per_sm<Op, TPB, RT>(), sizeof(float2),
                                      sizeof(float));
}

template <class Op, int TPB, int RT>
inline int run_pairs_symx(const typename Op::Params& P, int64_t n, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (n <= 0) return kOk;
  if (n > INT32_MAX / 4) return kInvalidArgument;
  const SymPlan plan = symx_plan<Op, TPB, RT>(n);
  if (plan.ws_bytes > ws_bytes) return kWorkspaceTooSmall;
  if (ws == nullptr) return kInvalidArgument;
  if (!symx_prepare<Op, TPB, RT>()) return kLaunchFailure;
  auto* row_ws = reinterpret_cast<float2*>(ws);
  auto* col_ws = reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + plan.col_off);
  launch_chained(pairs_kernel_symx<Op, TPB, RT>, plan.C, TPB, symx_dyn_smem_bytes<Op, TPB, RT>(), stream, P, (int)n,
                 plan.nblk, plan.TT, plan.U, plan.C, row_ws, col_ws);
  const int tpp = sym_finalize_tpp(plan);
  launch_chained(finalize_sym_kernel<Op, TPB, TPB * RT, F2>, finalize_grid(n, tpp), kFinThreads, 0, stream, P, (int)n,
                 plan.nblk, plan.TT, plan.U, plan.C, row_ws, col_ws, tpp);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

// K(x, x) a: the FP32 Gaussian sum of a set beyond the split shapes runs the expanded form (OpX), everything else the
// difference form (OpD).
template <class OpX, typename V>
inline bool ksym_expanded(int64_t n, int family) {
  return std::is_same<V, F2>::value && family == kGauss && n > kSplitN;
}
template <class OpX, class OpD, typename V>
inline int run_ksym(const typename OpD::Params& P, int64_t n, void* ws, size_t wsb, cudaStream_t st) {
  if (ksym_expanded<OpX, V>(n, P.f.family)) return run_pairs_symx<OpX, kTpbKSym, kRtKSym>(P, n, ws, wsb, st);
  return run_sym<OpD, V>(P, n, ws, wsb, st);
}
template <class OpX, class OpD, typename V>
inline size_t ksym_scratch(int64_t n, int family) {
  if (ksym_expanded<OpX, V>(n, family)) return symx_plan<OpX, kTpbKSym, kRtKSym>(n).ws_bytes;
  return sym_scratch<OpD, V>(n, family);
}
template <class OpX, class OpD, typename V>
inline size_t ksym_scratch_upto(int64_t n) {
  size_t b = sym_scratch_upto<OpD, V>(n);
  if (ksym_expanded<OpX, V>(n, kGauss)) {
    const size_t v = sym_plan_upto<kTpbKSym, kTpbKSym * kRtKSym>(kSplitN, n, OpX::NP, OpX::NP,
                                                                 symx_ctas_per_sm<OpX, kTpbKSym, kRtKSym>(),
                                                                 sizeof(float2), sizeof(float));
    b = v > b ? v : b;
  }
  return b;
}

}  // namespace lddmm
