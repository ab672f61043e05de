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
#define LDDMM_RT_SYM_FWD 8
#endif
#ifndef LDDMM_RT_FO_SYM
#define LDDMM_RT_FO_SYM 4
#endif
#ifndef LDDMM_RT_SYM_FWD_L
#define LDDMM_RT_SYM_FWD_L 4
#endif
#ifndef LDDMM_RT_ADJOINT_SYM_L
#define LDDMM_RT_ADJOINT_SYM_L 2
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
#define LDDMM_RT_KSYM 8
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
// The symmetric second-order forward step (pairs_kernel_sym): 8 targets per thread (168 registers, 3 CTAs per SM,
// its compensated row sums in 48 KiB of dynamic shared memory) measured 15% faster at level 6 than 4 targets per
// thread (134 registers, 3 CTAs per SM): the per-step source loads and the column shuffles are shared by twice
// as many pairs, and four independent lane groups hide the latency of the ex2 chain.
constexpr int kRtSymFwd = LDDMM_RT_SYM_FWD;
// Small and middle point sets: the split symmetric kernel (pairs_kernel_sym with SPLIT: the four warps of a CTA share
// 32 RT targets and take a quarter of every tile each), with more targets per thread as the set grows. A small RT gives
// more units, a large one fewer loads, shuffles and partials per pair. Each line lies where the next shape starts to
// win; us per step, launches overlapped (2 | 4 | 8 targets split; "-": the shape that was used up to here):
//   forward step   n = 1,500: 11.5 | 11.1 | 14.4 (- 14.7)   2,562: 16.4 | 14.7 | 15.3 (- 15.5)   4,000: 23.2 | 20.9 |
//                  20.5 (- 20.9)   7,000: 50.9 | 40.2 | 41.0 (- 56.7)   10,242: 89 | 74.5 | 67.9 (- 80.3)
//                  16,000: 190 | 152 | 138 (- 174)   20,000: 301 | 236 | 221, without the split 223
//   adjoint step   642: 11.1 | 14.1 (- 18.7)   2,000: 14.9 | 15.0 (- 19.7)   3,200: 29.0 | 26.1 (- 30.0)   7,000: 77.0 |
//                  70.9 (- 83.4)   10,242: 139 | 129, without the split 120
//   K a            642: 8.1 | 9.0 | 10.1 (- 16.3)   2,562: 12.0 | 11.9 | 12.0 (- 20.1)   4,000: 17.1 | 15.3 | 14.9 (-
//                  20.1)   10,242: 55 | 45.5 | 41.0 (- 48.9)   16,000: 114 | 91 | 79.7 (- 79.9)
//   first-order    642: 9.5 | 11.8 (- 19.4)   2,562: 17.3 | 16.1 (- 20.6)   7,000: 55.5 | 44.6 (- 43.6)   8,000: 63 |
//   adjoint step   56 (- 74.8)   10,242: 97.7 | 83.0, without the split 74.6
// and for the Laplacian (2 | 4 split): forward 2,562: 18.3 | 16.7 (- 23.8), 6,000: 45.1 | 42.9 (- 46.7), 10,242: 110 |
// 98, without 91; adjoint 6,000: 75.9 | 63.7 (- 87.7); K a 10,242: 67 | 58.1 (- 63.6).
constexpr int64_t kSplit2N = 1280, kSplit2NAdj = 2048;  // 2 targets per thread up to here
constexpr int64_t kSplit4N = 3600;                      // 4 up to here, then 8 (forward step and K a, Gaussian)
constexpr int64_t kSplit4NLast = 8192;                  // 4 up to here, then no split (adjoint steps, Laplacian)
constexpr int64_t kSplit8N = 16384;                     // 8 up to here, then no split
// The symmetric K(x, x) a (pairs_kernel_symx): 8 targets per thread.
// The symmetric first-order adjoint step (pairs_kernel_sym): 4 targets per thread.
constexpr int kRtFoSym = LDDMM_RT_FO_SYM;
// The symmetric steps with the Laplacian family (its radial profile -- a square root and the polynomial -- takes
// registers that the Gaussian shapes spend on more targets per thread).
constexpr int kRtSymFwdL = LDDMM_RT_SYM_FWD_L;
constexpr int kRtAdjointSymL = LDDMM_RT_ADJOINT_SYM_L;
constexpr int kRtFoSymL = LDDMM_RT_FO_SYM_L;
constexpr int kRtKSymL = LDDMM_RT_KSYM_L;
constexpr int kTpbKSym = LDDMM_TPB_KSYM;
constexpr int kRtKSym = LDDMM_RT_KSYM;
// FP64 baseline path.
constexpr int kTpb64 = LDDMM_TPB_64;
constexpr int kRt64 = LDDMM_RT_64;
// FP64 symmetric sums (pairs_kernel_sym with V = double), threads per CTA x targets per thread. 64 x 4 for K a, the
// forward step and the first-order adjoint step, 128 x 2 for the adjoint step (17 target values per thread: 4 targets
// would leave 1 CTA per SM). us at n = 10,242 / 40,962, 64 x 4 | 128 x 2 | 128 x 4: K a 113 / 1486 | 120 / 1593 | 111 /
// 1494; adjoint step 302 / 4218 | 291 / 4100 | 299 / 4232 (every ordered pair with exp(): K a 227 / 3111, adjoint step
// 463 / 6606).
constexpr int kTpbSym64 = 64, kRtSym64 = 4;
constexpr int kTpbSym64Adj = 128, kRtSym64Adj = 2;
// Small sets split: 128 x 1, then 128 x 2 (us per step with 1 | 2 targets split, then the shape above: forward 642:
// 10.8 | 11.6 | 20, 1,500: 16.1 | 15.4 | 21, 2,562: 28.4 | 24.6 | 22.7; the Laplacian's 2,562: 36.4 | 34.6 | 48.7,
// 4,000: 62.8 | 55.3 | 55.6).
constexpr int64_t kSplit1N64 = 1280, kSplit2N64 = 2304, kSplit2N64Lap = 4096;

static_assert(kSplit4NLast >= 8192 && kSplit8N >= 8192 && kSplit2N64 >= 2304,
              "every self-sum up to LDDMM_OWN_ORIGIN_POINTS runs a split kernel");

}  // namespace lddmm
