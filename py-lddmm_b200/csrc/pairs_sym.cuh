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
//  * Column credit without atomics: inside a tile, warp w of the CTA takes chunk (w + phase) mod W of 32 sources in
//    phase `phase` (one barrier per phase), and lane λ processes source (λ + s) mod 32 of the chunk at step s: the 32
//    lanes read 32 different sources (conflict-free 16-byte loads of the shared tile). The lane's column sum for its
//    source (its RT targets) is added to a rotating accumulator that moves one lane down after every step (one
//    shuffle per accumulator), so it follows its source around the warp; after 32 steps lane λ holds the warp's
//    column sum of source λ of the chunk and adds it to the tile's column accumulators in shared memory. At the end
//    of the unit those hold the unit's column sums (TPB sources x NC), written as one partial per (block i, source).
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
//   SymTgt<V>                            per-lane-group register state (V = F2: two targets, V = double: one)
//   load_target_sym<V>(P, i0, i1, v0, v1, SymTgt<V>&)  targets i0, i1 (< n); v0 / v1 false = padding (zero payload)
//   source_fields_sym(P, l, double* f)   NSS fields of source l (FP64)
//   pair_sym<COL, Fam, V>(const Frame&, const SymTgt<V>&, const V* s, V* row, V* col)
//   finalize_sym(P, i, const double* row, const double* col)
//
// FP64 (V = double): one target per lane group, sources staged as doubles, row sums, column sums and column partials
// in FP64; the rotating accumulator costs two shuffles per field. What it saves is the exponential (about a third of
// an FP64 pair) and the shared products, on a pipe of half the FP32 rate.
#pragma once
#include "launch_config.cuh"
#include "lddmm_common.cuh"

#ifndef LDDMM_SYM
#define LDDMM_SYM 1  // 0: self-interaction sums evaluate every ordered pair (pairs_kernel)
#endif
#ifndef LDDMM_SYM_COMPACT
#define LDDMM_SYM_COMPACT 1  // 0: the symmetric kernels stage sources in pairs_kernel's duplicated layout (measured
                             // 3-6% slower at level 6: twice the bytes per unshared load)
#endif
#ifndef LDDMM_SYMX_COL_SPLIT
#define LDDMM_SYMX_COL_SPLIT 0  // 1: pairs_kernel_symx accumulates the column terms of even and odd lane groups apart
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

// Shared-memory record of a staged source tile. In the symmetric kernels the 32 lanes of a warp read 32 different
// sources at every step (no broadcast), so the record size is what the loads cost: compact records hold each field
// once in FP32 (float4 groups) and the packed (f, f) operands are formed in registers; the duplicated layout of
// pairs_kernel (Unit<F2>: one 16-byte load gives two packed operands) reads twice the bytes.
template <int NF, int TPB, typename V>
struct SymStage;
template <int NF, int TPB>
struct SymStage<NF, TPB, double> {
  static constexpr int NQ = (NF + 1) / 2;  // 16-byte units of two fields
  using T = double2;
  static __device__ __forceinline__ void store(T (*sm)[TPB], int t, const double* fl) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) sm[q][t] = make_double2(fl[2 * q], fl[2 * q + 1]);
  }
  static __device__ __forceinline__ void load(const T (*sm)[TPB], int src, double* sv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double2 w = sm[q][src];
      sv[2 * q] = w.x;
      sv[2 * q + 1] = w.y;
    }
  }
  static constexpr int kFields = 2 * NQ;
};
template <int NF, int TPB>
struct SymStage<NF, TPB, F2> {
#if LDDMM_SYM_COMPACT
  static constexpr int NQ = (NF + 3) / 4;  // float4 groups
  using T = float4;
  static __device__ __forceinline__ void store(T (*sm)[TPB], int t, const double* fl) {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      sm[q][t] = make_float4((float)fl[4 * q], (float)fl[4 * q + 1], (float)fl[4 * q + 2], (float)fl[4 * q + 3]);
  }
  static __device__ __forceinline__ void load(const T (*sm)[TPB], int src, F2* sv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const float4 w = sm[q][src];
      sv[4 * q] = f2(w.x, w.x);
      sv[4 * q + 1] = f2(w.y, w.y);
      sv[4 * q + 2] = f2(w.z, w.z);
      sv[4 * q + 3] = f2(w.w, w.w);
    }
  }
#else
  static constexpr int NQ = (NF + 1) / 2;  // 16-byte units of two duplicated fields
  using T = Unit<F2>;
  static __device__ __forceinline__ void store(T (*sm)[TPB], int t, const double* fl) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      Unit<F2> w;
      w.a = VT<F2>::dup(fl[2 * q]);
      w.b = VT<F2>::dup(fl[2 * q + 1]);
      sm[q][t] = w;
    }
  }
  static __device__ __forceinline__ void load(const T (*sm)[TPB], int src, F2* sv) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const Unit<F2> w = sm[q][src];
      sv[2 * q] = w.a;
      sv[2 * q + 1] = w.b;
    }
  }
#endif
  static constexpr int kFields = 4 * ((NF + 3) / 4);  // size of the FP64 field buffer and of the operand array
};

struct SymPlan {
  int nblk = 0, TT = 0, C = 0, S = 0;
  long long U = 0;
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
  const long long wave = (long long)device_sm_count() * (ctas_per_sm > 0 ? ctas_per_sm : 1);
  // one resident wave of CTAs; up to half a wave more units run as one CTA each, so that no CTA takes two units while
  // others take one (forward step at 6,000 points, 576 units, 444 resident CTAs: 41.4 -> 31.7 us)
  p.C = (int)(2 * p.U < 3 * wave ? p.U : wave);
  p.S = sk_max_slots(p.TT, p.U, p.C);  // the longest row has TT units
  p.col_off = ((size_t)p.S * (size_t)nr * (size_t)n * row_bytes + 255) & ~(size_t)255;
  p.ws_bytes =
      p.col_off + (size_t)Geo::col_first((n + Geo::K - 1) / Geo::K) * (size_t)nc * (size_t)Geo::K * col_bytes;
  return p;
}

// One chunk of 32 sources against the warp's targets; lane λ returns the warp's column sums of source λ in cs.
template <class Op, int TPB, int RT, bool COL, class Fam, typename V>
__device__ __forceinline__ void sym_chunk(const Frame& f,
                                          const typename Op::template SymTgt<V> (&tgt)[RT / VT<V>::kLanes],
                                          const typename SymStage<Op::NSS, TPB, V>::T (*sm)[TPB], int chunk,
                                          V (&acc)[RT / VT<V>::kLanes][Op::NR],
                                          typename VT<V>::Scalar (&cs)[Op::NC]) {
  using St = SymStage<Op::NSS, TPB, V>;
  constexpr int G = RT / VT<V>::kLanes;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < Op::NC; ++c) cs[c] = 0;
#pragma unroll kSymUnroll
  for (int s = 0; s < 32; ++s) {
    const int src = chunk * 32 + ((lane + s) & 31);
    V sv[St::kFields];
    St::load(sm, src, sv);
    if constexpr (COL) {
      V col[Op::NC];
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) col[c] = VT<V>::first(cs[c]);
#pragma unroll
      for (int g = 0; g < G; ++g) Op::template pair_sym<true, Fam, V>(f, tgt[g], sv, acc[g], col);
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) cs[c] = __shfl_sync(0xffffffffu, VT<V>::hsum(col[c]), (lane + 1) & 31);
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g) Op::template pair_sym<false, Fam, V>(f, tgt[g], sv, acc[g], nullptr);
    }
  }
}

template <class Op, int TPB, int RT, bool COL, class Fam, typename V>
__device__ __forceinline__ void sym_tile(const Frame& f,
                                         const typename Op::template SymTgt<V> (&tgt)[RT / VT<V>::kLanes],
                                         const typename SymStage<Op::NSS, TPB, V>::T (*sm)[TPB],
                                         typename VT<V>::Scalar (*colacc)[TPB],
                                         V (&acc)[RT / VT<V>::kLanes][Op::NR]) {
  constexpr int W = TPB / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int ph = 0; ph < W; ++ph) {
    const int chunk = (warp + ph) % W;
    typename VT<V>::Scalar cs[Op::NC];
    sym_chunk<Op, TPB, RT, COL, Fam, V>(f, tgt, sm, chunk, acc, cs);
    if constexpr (COL) {
#pragma unroll
      for (int c = 0; c < Op::NC; ++c) colacc[c][chunk * 32 + lane] += cs[c];
    }
    __syncthreads();  // the next phase hands this chunk (and its column accumulators) to another warp
  }
}

// minimum resident CTAs per SM: the op's for FP32; no register cap in FP64
template <class Op, typename V>
constexpr int kSymCtas = std::is_same<V, F2>::value ? Op::kSymMinCtas : 1;

// SPLIT (small point sets): the warps of a CTA share its 32 RT targets and take one chunk of every tile each, instead
// of TPB RT targets and all chunks in turn. A unit is TPB / 32 times shorter and the triangle has that many times more
// units, which is what a set too small to fill the GPU needs: at 2,562 points a forward step's longest chain falls
// from 128 pair evaluations to 32 and its 462 units occupy every SM. The warps' row sums meet in shared memory at the
// end of a segment; a chunk's column sums are one warp's and go straight to the column partial.
template <class Op, int TPB, int RT, class Fam, typename V, bool SPLIT>
__global__ void __launch_bounds__(TPB, kSymCtas<Op, V>)
    pairs_kernel_sym(const typename Op::Params P, int n, int nblk, int TT, long long U, int C,
                     typename VT<V>::Partial* __restrict__ row_ws, typename VT<V>::Scalar* __restrict__ col_ws) {
  using St = SymStage<Op::NSS, TPB, V>;
  constexpr int L = VT<V>::kLanes, G = RT / L, NR = Op::NR, NC = Op::NC, W = TPB / 32;
  constexpr int TW = SPLIT ? 32 : TPB;  // targets a lane-group index apart
  constexpr int B = TW * RT;
  using Geo = SymGeom<TPB, B>;
  constexpr int K = Geo::K;
  static_assert(TPB % 32 == 0 && RT % L == 0, "launch shape");
  __shared__ typename St::T sm[St::NQ][TPB];
  __shared__ typename VT<V>::Scalar colacc[SPLIT ? 1 : NC][TPB];
  // compensated row sums of the segment, one private column per thread (G * NR * Comp<V>::kWords rows of TPB): dynamic
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

    if constexpr (SPLIT) {
      double o[3];
      segment_origin(f, P.x, i * B, i * B + B < n ? i * B + B - 1 : n - 1, o);
#pragma unroll
      for (int c = 0; c < 3; ++c) org[c] = o[c];
    }
    typename Op::template SymTgt<V> tgt[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int i0 = base + (g * L) * TW, i1 = base + (g * L + L - 1) * TW;
      if constexpr (SPLIT)
        Op::template load_target_sym<V>(with_origin(P, org), i0 < n ? i0 : n - 1, i1 < n ? i1 : n - 1, i0 < n, i1 < n,
                                        tgt[g]);
      else
        Op::template load_target_sym<V>(P, i0 < n ? i0 : n - 1, i1 < n ? i1 : n - 1, i0 < n, i1 < n, tgt[g]);
      Comp<V> z;
      z.zero();
#pragma unroll
      for (int c = 0; c < NR; ++c) z.template store<TPB>(cs, g * NR + c, threadIdx.x);
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
          for (int c = 0; c < NC; ++c) colacc[c][threadIdx.x] = 0;
        }
      }
      __syncthreads();
      V acc[G][NR];
#pragma unroll
      for (int g = 0; g < G; ++g)
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
        typename VT<V>::Scalar col[NC];
        if (diag) {
          sym_chunk<Op, TPB, RT, false, Fam, V>(f, tgt, sm, warp, acc, col);
        } else {
          sym_chunk<Op, TPB, RT, true, Fam, V>(f, tgt, sm, warp, acc, col);
#pragma unroll
          for (int c = 0; c < NC; ++c) col_ws[cb + (size_t)c * K] = col[c];
        }
      } else if (diag) {
        sym_tile<Op, TPB, RT, false, Fam, V>(f, tgt, sm, colacc, acc);
      } else {
        sym_tile<Op, TPB, RT, true, Fam, V>(f, tgt, sm, colacc, acc);
      }
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          Comp<V> m;
          m.template load<TPB>(cs, g * NR + c, threadIdx.x);
          m.merge(acc[g][c]);
          m.template store<TPB>(cs, g * NR + c, threadIdx.x);
        }
      if constexpr (SPLIT) {
        __syncthreads();  // every warp has read the tile and left its row sums
      } else if (!diag) {
#pragma unroll
        for (int c = 0; c < NC; ++c) col_ws[(kHeld ? cb : column_base()) + (size_t)c * K] = colacc[c][threadIdx.x];
      }
      // (not SPLIT) the last phase barrier of sym_tile orders every read of sm and colacc before the next staging
    }

    if (SPLIT && u + (t1 - t0) >= u_end) chain_go();
    if constexpr (SPLIT) {
      // the block's row sums: field c of the lanes' targets by warp c mod W, over the W warps in order
#pragma unroll
      for (int g = 0; g < G; ++g)
        for (int c = warp; c < NR; c += W) {
          double sum[L];
#pragma unroll
          for (int k = 0; k < L; ++k) sum[k] = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            Comp<V> m;
            m.template load<TPB>(cs, g * NR + c, w * 32 + lane);
#pragma unroll
            for (int k = 0; k < L; ++k) sum[k] += partial_value(m.partial(k));
          }
#pragma unroll
          for (int k = 0; k < L; ++k) {
            const int idx = base + (g * L + k) * TW;
            if (idx < n) row_ws[((size_t)slot * NR + c) * (size_t)n + idx] = VT<V>::to_partial(sum[k]);
          }
        }
      __syncthreads();  // the next segment clears the sums
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const int idx = base + (g * L + k) * TW;
          if (idx < n) {
#pragma unroll
            for (int c = 0; c < NR; ++c) {
              Comp<V> m;
              m.template load<TPB>(cs, g * NR + c, threadIdx.x);
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
  return (size_t)(RT / VT<V>::kLanes) * Op::NR * Comp<V>::kWords * TPB * sizeof(V);
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


// Launch shapes. Each symmetric op names its rule (Op::Shape): the FP32 lines between 2, 4 and 8 targets per thread
// with the split and the shape without it, and the FP64 shape (launch_config.cuh has the measurements).
template <int SPLIT2_N, int SPLIT4_N, int SPLIT8_N, int SPLIT4_N_LAP, int RT, int RT_LAP, int TPB64, int RT64>
struct SymRule {
  static constexpr int64_t kSplit2 = SPLIT2_N, kSplit4 = SPLIT4_N, kSplit8 = SPLIT8_N, kSplit4Lap = SPLIT4_N_LAP;
  static constexpr int kRt = RT, kRtLap = RT_LAP, kTpb64 = TPB64, kRt64 = RT64;
};
template <int TPB, int RT, bool SPLIT>
struct SymShape {
  static constexpr int kTpb = TPB, kRt = RT;
  static constexpr bool kSplit = SPLIT;
};

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
    if (n <= R::kSplit2) return fn(SymShape<128, 2, true>{});
    if (n <= (kG ? R::kSplit4 : R::kSplit4Lap)) return fn(SymShape<128, 4, true>{});
    if constexpr (kG && R::kSplit8 > R::kSplit4) {
      if (n <= R::kSplit8) return fn(SymShape<128, 8, true>{});
    }
    return fn(SymShape<128, kG ? R::kRt : R::kRtLap, false>{});
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
// Scratch for every point count up to n: the largest of each shape's range.
template <class Op, typename V>
inline size_t sym_scratch_upto(int64_t n) {
  using R = typename Op::Shape;
  size_t b = 0;
  for (const int64_t k : {R::kSplit2, R::kSplit4, R::kSplit8, R::kSplit4Lap, kSplit1N64, kSplit2N64, kSplit2N64Lap,
                          sym_max_n<Op, V>(), n}) {
    if (k > n || !sym_takes<Op, V>(k)) continue;
    for (const int family : {(int)kGauss, (int)kLaplacian0, (int)kLaplacianMax}) {
      const size_t v = sym_scratch<Op, V>(k, family);
      b = v > b ? v : b;
    }
  }
  return b;
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
__device__ __forceinline__ void symx_tile(const F2 (&yt)[RT / 2][3], const F2 (&tp)[RT / 2][Op::NP],
                                          const typename SymStage<4 + Op::NP, TPB, F2>::T (*sm)[TPB],
                                          float (*colacc)[TPB], F2 (&acc)[RT / 2][Op::NP]) {
  using St = SymStage<4 + Op::NP, TPB, F2>;
  constexpr int G = RT / 2, NP = Op::NP, W = TPB / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int ph = 0; ph < W; ++ph) {
    const int chunk = (warp + ph) % W;
    float cs[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c) cs[c] = 0.f;
#pragma unroll kSymxUnroll
    for (int s = 0; s < 32; ++s) {
      const int src = chunk * 32 + ((lane + s) & 31);
      F2 sv[St::kFields];
      St::load(sm, src, sv);
      F2 col[NP], col2[NP];
      if constexpr (COL) {
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          col[c] = f2(cs[c], 0.f);
          col2[c] = VT<F2>::zero();
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
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
          if (LDDMM_SYMX_COL_SPLIT != 0 && (g & 1)) {  // resolved at compile time (the loop is unrolled)
#pragma unroll
            for (int c = 0; c < NP; ++c) col2[c] = fma(e, tp[g][c], col2[c]);
          } else {
#pragma unroll
            for (int c = 0; c < NP; ++c) col[c] = fma(e, tp[g][c], col[c]);
          }
        }
      }
      if constexpr (COL) {
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          if constexpr (LDDMM_SYMX_COL_SPLIT != 0) col[c] = col[c] + col2[c];
          float lo, hi;
          split(col[c], lo, hi);
          cs[c] = __shfl_sync(0xffffffffu, lo + hi, (lane + 1) & 31);
        }
      }
    }
    if constexpr (COL) {
#pragma unroll
      for (int c = 0; c < NP; ++c) colacc[c][chunk * 32 + lane] += cs[c];
    }
    __syncthreads();  // the next phase hands this chunk (and its column accumulators) to another warp
  }
}

template <class Op, int TPB, int RT>
__global__ void __launch_bounds__(TPB, Op::kSymMinCtas)
    pairs_kernel_symx(const typename Op::Params P, int n, int nblk, int TT, long long U, int C,
                      float2* __restrict__ row_ws, float* __restrict__ col_ws) {
  using St = SymStage<4 + Op::NP, TPB, F2>;
  constexpr int L = 2, G = RT / L, NP = Op::NP;
  constexpr int B = TPB * RT;
  using Geo = SymGeom<TPB, B>;
  static_assert(TPB % 32 == 0 && RT % L == 0, "launch shape");
  __shared__ typename St::T sm[St::NQ][TPB];
  __shared__ float colacc[NP][TPB];
  __shared__ float red[6][TPB / 32];
  extern __shared__ __align__(16) unsigned char sym_dyn_smem[];
  F2 (*cs)[TPB] = reinterpret_cast<F2 (*)[TPB]>(sym_dyn_smem);  // compensated row sums, G * NP * 2 rows
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

    F2 yt[G][3], tp[G][NP];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int k0 = base + (g * L) * TPB, k1 = base + (g * L + 1) * TPB;
      double y0[3], y1[3], p0[NP], p1[NP];
      Op::point(P, k0 < n ? k0 : n - 1, y0);
      Op::point(P, k1 < n ? k1 : n - 1, y1);
      Op::payload(P, k0 < n ? k0 : n - 1, p0);
      Op::payload(P, k1 < n ? k1 : n - 1, p1);
      double q0 = 0.0, q1 = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float r0 = (float)((y0[c] - fo[c]) * f.s - (double)ob[c]);
        const float r1 = (float)((y1[c] - fo[c]) * f.s - (double)ob[c]);
        yt[g][c] = f2(r0, r1);
        q0 += (double)r0 * (double)r0;
        q1 += (double)r1 * (double)r1;
      }
      // column payload: f_k a_k (expanded form) or a_k; padded targets carry none
      const double f0 = k0 < n ? (expand ? exp2(-q0) : 1.0) : 0.0;
      const double f1 = k1 < n ? (expand ? exp2(-q1) : 1.0) : 0.0;
#pragma unroll
      for (int c = 0; c < NP; ++c) tp[g][c] = f2((float)(f0 * p0[c]), (float)(f1 * p1[c]));
      Comp<F2> z;
      z.zero();
#pragma unroll
      for (int c = 0; c < NP; ++c) z.template store<TPB>(cs, g * NP + c, threadIdx.x);
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
        for (int c = 0; c < NP; ++c) colacc[c][threadIdx.x] = 0.f;
      }
      __syncthreads();
      F2 acc[G][NP];
#pragma unroll
      for (int g = 0; g < G; ++g)
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
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < NP; ++c) {
          Comp<F2> m;
          m.template load<TPB>(cs, g * NP + c, threadIdx.x);
          m.merge(acc[g][c]);
          m.template store<TPB>(cs, g * NP + c, threadIdx.x);
        }
      if (!diag) {
        const int j = t / RT;
        const size_t cb = (size_t)(Geo::col_first(j) + i) * NP * B + (size_t)(t - RT * j) * TPB + threadIdx.x;
#pragma unroll
        for (int c = 0; c < NP; ++c) col_ws[cb + (size_t)c * B] = colacc[c][threadIdx.x];
      }
      // the last phase barrier of symx_tile orders every read of sm and colacc before the next tile's staging
    }

#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const int idx = base + (g * L + k) * TPB;
        if (idx < n) {
          double y2 = 0.0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double yr = VT<F2>::lane(yt[g][c], k);
            y2 += yr * yr;
          }
          const double fac = expand ? exp2(-y2) : 1.0;
#pragma unroll
          for (int c = 0; c < NP; ++c) {
            Comp<F2> m;
            m.template load<TPB>(cs, g * NP + c, threadIdx.x);
            const float2 pp = m.partial(k);
            const double w = ((double)pp.x + (double)pp.y) * fac;
            const float h = (float)w;
            row_ws[((size_t)slot * NP + c) * (size_t)n + idx] = make_float2(h, (float)(w - (double)h));
          }
        }
      }
    u += t1 - t0;
    ++i;
  }
}

template <class Op, int TPB, int RT>
constexpr size_t symx_dyn_smem_bytes() {
  return (size_t)(RT / 2) * Op::NP * 2 * TPB * sizeof(F2);
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
inline size_t symx_ws_bytes(int64_t n) {
  return make_sym_plan<TPB, TPB * RT>(n, Op::NP, Op::NP, symx_ctas_per_sm<Op, TPB, RT>(), sizeof(float2), sizeof(float)).ws_bytes;
}

template <class Op, int TPB, int RT>
inline int run_pairs_symx(const typename Op::Params& P, int64_t n, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (n <= 0) return kOk;
  if (n > INT32_MAX / 4) return kInvalidArgument;
  const SymPlan plan = make_sym_plan<TPB, TPB * RT>(n, Op::NP, Op::NP, symx_ctas_per_sm<Op, TPB, RT>(), sizeof(float2), sizeof(float));
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
template <class OpX, class OpD, typename V>
inline int run_ksym(const typename OpD::Params& P, int64_t n, void* ws, size_t wsb, cudaStream_t st) {
  if (std::is_same<V, F2>::value && P.f.family == kGauss && n > OpD::Shape::kSplit8)
    return run_pairs_symx<OpX, kTpbKSym, kRtKSym>(P, n, ws, wsb, st);
  return run_sym<OpD, V>(P, n, ws, wsb, st);
}
template <class OpX, class OpD, typename V>
inline size_t ksym_scratch(int64_t n, int family) {
  if (std::is_same<V, F2>::value && family == kGauss && n > OpD::Shape::kSplit8)
    return symx_ws_bytes<OpX, kTpbKSym, kRtKSym>(n);
  return sym_scratch<OpD, V>(n, family);
}
template <class OpX, class OpD, typename V>
inline size_t ksym_scratch_upto(int64_t n) {
  const size_t b = sym_scratch_upto<OpD, V>(n), x = ksym_scratch<OpX, OpD, V>(n, kGauss);
  return sym_takes<OpD, V>(n) && x > b ? x : b;
}

}  // namespace lddmm
