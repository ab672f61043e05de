// Launch shapes of the all-pairs kernels (threads per CTA x targets per thread). The defaults were chosen by
// timing on the B200; each can be overridden at build time (-DLDDMM_RT_LIGHT=... etc.) for tuning sweeps.
#pragma once
#include <stdint.h>

#ifndef LDDMM_TPB_LIGHT
#define LDDMM_TPB_LIGHT 128
#endif
#ifndef LDDMM_RT_LIGHT
#define LDDMM_RT_LIGHT 4
#endif
#ifndef LDDMM_TPB_HEAVY
#define LDDMM_TPB_HEAVY 128
#endif
#ifndef LDDMM_RT_HEAVY
#define LDDMM_RT_HEAVY 2
#endif
#ifndef LDDMM_RT_ADJOINT
#define LDDMM_RT_ADJOINT 4
#endif
#ifndef LDDMM_RT_SYM_FWD
#define LDDMM_RT_SYM_FWD 6
#endif
#ifndef LDDMM_RT_FO_SYM
#define LDDMM_RT_FO_SYM 4
#endif
#ifndef LDDMM_RT_SYM_FWD_L
#define LDDMM_RT_SYM_FWD_L 4
#endif
#ifndef LDDMM_RT_ADJOINT_SYM_L
#define LDDMM_RT_ADJOINT_SYM_L 4
#endif
#ifndef LDDMM_RT_FO_SYM_L
#define LDDMM_RT_FO_SYM_L 4
#endif
#ifndef LDDMM_RT_KSYM_L
#define LDDMM_RT_KSYM_L 4
#endif
#ifndef LDDMM_TPB_KSYM
#define LDDMM_TPB_KSYM 128
#endif
#ifndef LDDMM_RT_KSYM
#define LDDMM_RT_KSYM 6
#endif
#ifndef LDDMM_TPB_64
#define LDDMM_TPB_64 128
#endif
#ifndef LDDMM_RT_64
#define LDDMM_RT_64 2
#endif

namespace lddmm {

// Light ops (<= 8 accumulators per target): several targets per thread amortise each broadcast LDS.
constexpr int kTpbLight = LDDMM_TPB_LIGHT;
constexpr int kRtLight = LDDMM_RT_LIGHT;
// Heavy ops (the 7-accumulator DDK): fewer targets per thread.
constexpr int kTpbHeavy = LDDMM_TPB_HEAVY;
constexpr int kRtHeavy = LDDMM_RT_HEAVY;
// The 12-accumulator second-order adjoint step: 4 targets per thread with its sums in registers (254 registers,
// 2 CTAs per SM) measured 4% faster than 2 targets per thread at 4 CTAs per SM (half the shared-memory reads per
// pair, two independent lane groups per source).
constexpr int kRtAdjoint = LDDMM_RT_ADJOINT;
// Symmetric sums, FP32, whole tiles: targets per thread. More of them share a source's loads and column shuffles; each
// takes two registers per value (both lanes of a packed operand are the target). us at 40,962 points, Gaussian, threads
// of 128 (the kernels with two targets to a packed value, at their best shape: forward 775, adjoint 1609, first-order
// adjoint 955, K a 381; Laplacian of order 3: 1114, 2047, 1215, 627):
//   forward step 4 | 6: 786 | 744          adjoint step 4 | 5: 1498 | 1525     first-order adjoint 4 | 5 | 6 at the
//   K a (expanded form) 4 | 6 | 8 | 10: 393 | 373 | 365 | 354                  better of two unroll depths: 845 | 826 | 842
//   Laplacian: forward step 4 | 6: 1051 | 1008, adjoint 4 | 5: 1830 | 1948, first-order adjoint 4 | 5 | 6: 1103 | 1105 |
//   1135, K a 4 | 6 | 8: 601 | 594 | 579
// A column sum is a chain of RT additions per step, and its rounding grows with RT: the shapes taken are the fastest
// whose errors against FP64 are not above those of the kernels before (K a of 30,001 points, sigma 0.3: 6.8e-8 before,
// with 6 | 8 | 10 targets 6.6e-8 | 7.3e-8 | 8.2e-8; the Laplacian's K a of 20,000 points with 4 | 6 | 8: 0.97 | 1.06 | 1.13
// of it, its forward step with 4 | 5 | 6: 0.97 | 1.02 | 1.05).
constexpr int kRtSymFwd = LDDMM_RT_SYM_FWD;
constexpr int kRtFoSym = LDDMM_RT_FO_SYM;
constexpr int kRtSymFwdL = LDDMM_RT_SYM_FWD_L;
constexpr int kRtAdjointSymL = LDDMM_RT_ADJOINT_SYM_L;
constexpr int kRtFoSymL = LDDMM_RT_FO_SYM_L;
constexpr int kRtKSymL = LDDMM_RT_KSYM_L;
// Small and middle point sets: the split symmetric kernel (pairs_kernel_sym with SPLIT: the four warps of a CTA share
// 32 RT targets and take a quarter of every tile each), with more targets per thread as the set grows. A small RT gives
// more units, a large one fewer loads, shuffles and partials per pair. us, launches overlapped (2 | 4 | 8 targets split
// / whole tiles; "-": the split kernel with two targets to a packed value at its best shape):
//   forward step     n = 1,300: 7.8 | 8.6 | 11.9 (- 8.8)   2,562: 13.3 | 11.8 | 12.8 (- 12.2)   6,000: 33.0 | 27.4 | 27.9
//                    (- 30.5)   10,242: 72.4 | 65.8 | 62.9 / 57.2 (- 67)   13,000: 110 | 95.8 | 88.9 / 106 (- 95.6)
//                    16,000: 161 | 140 | 132 / 130   20,000: 250 | 215 | 203 / 194
//   adjoint step     1,300: 9.0 | 11.6 (- 9.3)   2,562: 18.0 | 16.7 (- 17.2)   8,000: 79 | 72.3 / 74.9 (- 76.5)
//                    10,242: 122 | 115 / 109 (- 116)   13,000: 190 | 171 / 175 (- 188)   20,000: 437 | 388 / 377
//   first-order      1,300: 7.9 | 9.1 (- 9.5)   2,562: 14.1 | 12.5 (- 13.2)   6,000: 36.0 | 30.1 (- 33.9)   10,242: 80 |
//   adjoint step     72 / 66.4 (- 71.4)   13,000: 122 | 105 / 105 (- 115)   20,000: 278 | 235 / 224
//   K a              2,562: 9.5 | 8.7 | 8.8 (- 9.1)   6,000: 20.5 | 19.0 | 18.0 (- 18.9)   10,242: 46.5 | 39.7 | 36.9 /
//                    45.6 (- 38.4)   13,000: 67 | 56 | 52 / 53 (- 54)   16,000: 98 | 81 | 79 / 70 (- 78)
// and for the Laplacian of order 3: forward 10,242: 91 | 83 | 86 / 76 (- 82), 13,000: 139 | 123 | 122 / 141 (- 132);
// adjoint 13,000: 227 | 208 / 230 (- 239), 16,000: 335 | 308 / 319; K a 10,242: 56 | 51 | 48 / 59 (- 53).
// (Taken with a median of three points as a split block's origin; the middle of 32 adds 0.1-0.2 us to each split figure.)
// The bounds are in points, as measured on 148 SMs; on another chip they stay correct and may not be the fastest.
// 2 targets up to kSplit2N: there the units of 64 points still have an SM each. Whole tiles are faster per pair and
// their units four times longer, so between kWholeN and kSplitN they are taken where their units fill the resident CTAs
// (10,242 and 16,000 points above, not 13,000), beyond kSplitN always. K a of the Gaussian keeps the split up to
// kSplitN: its whole tiles centre a block on its box, the split on a point, which one far point does not move.
constexpr int64_t kSplit2N = 1408;
constexpr int64_t kSplit4N = 3600;   // 4 targets up to here in K a, then 8
constexpr int64_t kWholeN = 8192;    // (4 targets up to here in the Gaussian's forward step, then 8)
constexpr int64_t kSplitN = 16384;
constexpr int kTpbKSym = LDDMM_TPB_KSYM;
constexpr int kRtKSym = LDDMM_RT_KSYM;
// FP64 baseline path.
constexpr int kTpb64 = LDDMM_TPB_64;
constexpr int kRt64 = LDDMM_RT_64;
// FP64 symmetric sums (pairs_kernel_sym with V = double), threads per CTA x targets per thread. 64 x 4 for K a, the
// forward step and the first-order adjoint step, 128 x 2 for the adjoint step (measured with 17 values per target, 13
// since: 4 targets left 1 CTA per SM). us at n = 10,242 / 40,962, 64 x 4 | 128 x 2 | 128 x 4: K a 113 / 1486 | 120 / 1593 | 111 /
// 1494; adjoint step 302 / 4218 | 291 / 4100 | 299 / 4232 (every ordered pair with exp(): K a 227 / 3111, adjoint step
// 463 / 6606).
constexpr int kTpbSym64 = 64, kRtSym64 = 4;
constexpr int kTpbSym64Adj = 128, kRtSym64Adj = 2;
// Small sets split: 128 x 1, then 128 x 2 (us per step with 1 | 2 targets split, then the shape above: forward 642:
// 10.8 | 11.6 | 20, 1,500: 16.1 | 15.4 | 21, 2,562: 28.4 | 24.6 | 22.7; the Laplacian's 2,562: 36.4 | 34.6 | 48.7,
// 4,000: 62.8 | 55.3 | 55.6).
constexpr int64_t kSplit1N64 = 1280, kSplit2N64 = 2304, kSplit2N64Lap = 4096;

static_assert(kWholeN >= 8192 && kSplitN >= kWholeN && kSplit2N64 >= 2304,
              "every self-sum up to LDDMM_OWN_ORIGIN_POINTS runs a split kernel");

}  // namespace lddmm
