// Kernels of the learned momentum proposal: a per-vertex MLP (BF16 weights and activations, FP32 accumulation) and
// its training step, plus the nearest-target displacement feature.
//
// GEMM: C = op(A) op(B) on the tensor cores with mma.sync.m16n8k16 (bf16 x bf16 -> f32). CTA tile 64x64x32, four
// warps of 32x32; operands staged in padded shared memory (row stride +16 B: conflict-free ldmatrix) by cp.async in a
// ring of four stages, transposed operands read with ldmatrix.trans, so one kernel covers forward (X W), input
// gradient (dY W^T) and weight gradient (X^T dY). Epilogues fuse bias, ReLU, the ReLU-derivative mask and the BF16 /
// FP32 store (BF16 tiles pass through shared memory: 16-byte stores and mask loads); the weight gradient is split over
// the (long) vertex dimension and reduced in a fixed order (deterministic), and sums the columns of dY, the bias
// gradient, from the tiles it stages anyway.
// At 41,984 rows a layer is 0.7 G multiply-adds (2.5 us at the measured 930 per clock and SM of mma.sync) against 21-32
// MB (3-5 us from HBM): bound by memory and latency, not by the tensor cores. The ring took the training step's
// eleven GEMMs from 186 to 117 us: without it every 32-deep slice was a load, a barrier and a few instructions in
// series.
// All dimensions are padded by the caller: M, N multiples of 64, K a multiple of 32.
#include <cuda_bf16.h>

#include "../../include/lddmm_b200.h"
#include "lddmm_common.cuh"

namespace lddmm {
namespace mlp {

using bf16 = __nv_bfloat16;

constexpr int BM = 64, BN = 64, BK = 32, PAD = 8, THREADS = 128, STAGES = 4;

enum Epilogue : int {
  kEpiF32 = 0,          // C (f32) = acc                      (split-K partials)
  kEpiBiasF32 = 1,      // C (f32) = acc + bias[n]
  kEpiBiasReluBf16 = 2, // C (bf16) = relu(acc + bias[n])
  kEpiBiasBf16 = 3,     // C (bf16) = acc + bias[n]
  kEpiMaskBf16 = 4,     // C (bf16) = mask[m][n] > 0 ? acc : 0  (ReLU derivative of the forward activation)
};

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const bf16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const bf16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Global layouts: A is [M][K] (TA = false) or stored transposed as [K][M] (TA = true);
//                 B is [K][N] (TB = false) or stored transposed as [N][K] (TB = true). C is [M][N] (+ split offset).
// COLSUM (TB = false): colp[split][n] = column sums of the split's rows of B, by the CTAs of the first row block.
template <bool TA, bool TB, int EPI, bool COLSUM>
__global__ void __launch_bounds__(THREADS) gemm_kernel(int M, int N, int K, int k_split, const bf16* __restrict__ A,
                                                       const bf16* __restrict__ B, const float* __restrict__ bias,
                                                       const bf16* __restrict__ mask, void* __restrict__ C,
                                                       float* __restrict__ colp) {
  struct Stage {
    bf16 a[TA ? BK : BM][(TA ? BM : BK) + PAD];
    bf16 b[TB ? BN : BK][(TB ? BK : BN) + PAD];
  };
  __shared__ __align__(16) Stage st[STAGES];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int kb = blockIdx.z * k_split;
  const int ke = min(K, kb + k_split);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  chain_wait();
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  float cs0 = 0.f, cs1 = 0.f;  // COLSUM: column pair `lane`, rows 8 warp .. 8 warp + 7 of every slice

  const int nk = (ke - kb + BK - 1) / BK;
  auto stage_load = [&](int i) {
    if (i < nk) {
      Stage& S = st[i % STAGES];
      const int k0 = kb + i * BK;
#pragma unroll
      for (int it = threadIdx.x; it < (BM * BK) / 8; it += THREADS) {
        if (!TA) {
          const int r = it / (BK / 8), c = (it % (BK / 8)) * 8;
          cp_async16(&S.a[r][c], &A[(size_t)(m0 + r) * K + k0 + c]);
        } else {
          const int r = it / (BM / 8), c = (it % (BM / 8)) * 8;
          cp_async16(&S.a[r][c], &A[(size_t)(k0 + r) * M + m0 + c]);
        }
      }
#pragma unroll
      for (int it = threadIdx.x; it < (BN * BK) / 8; it += THREADS) {
        if (!TB) {
          const int r = it / (BN / 8), c = (it % (BN / 8)) * 8;
          cp_async16(&S.b[r][c], &B[(size_t)(k0 + r) * N + n0 + c]);
        } else {
          const int r = it / (BK / 8), c = (it % (BK / 8)) * 8;
          cp_async16(&S.b[r][c], &B[(size_t)(n0 + r) * K + k0 + c]);
        }
      }
    }
    cp_async_commit();  // a group per slice, empty past the last: the wait below counts groups
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) stage_load(i);

  for (int i = 0; i < nk; ++i) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();  // slice i has arrived for every thread, and everyone is done with the stage that is loaded next
    stage_load(i + STAGES - 1);
    const Stage& S = st[i % STAGES];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t a[2][4], b[4][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const int mr = wm + mt * 16;
        if (!TA)
          ldsm_x4(a[mt], &S.a[mr + (lane & 15)][kk + (lane >> 4) * 8]);
        else
          ldsm_x4_t(a[mt], &S.a[kk + (lane & 7) + (lane >> 4) * 8][mr + ((lane >> 3) & 1) * 8]);
      }
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        const int nc = wn + np * 16;
        uint32_t r[4];
        if (!TB)
          ldsm_x4_t(r, &S.b[kk + (lane & 15)][nc + (lane >> 4) * 8]);
        else
          ldsm_x4(r, &S.b[nc + (lane & 7) + (lane >> 4) * 8][kk + ((lane >> 3) & 1) * 8]);
        b[2 * np][0] = r[0];
        b[2 * np][1] = r[1];
        b[2 * np + 1][0] = r[2];
        b[2 * np + 1][1] = r[3];
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[mt][nt], a[mt], b[nt]);
    }
    if constexpr (COLSUM) {
      static_assert(!TB && BK == 32 && BN == 64, "one column pair per lane, eight rows per warp");
      if (blockIdx.y == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&S.b[warp * 8 + r][2 * lane]);
          cs0 += __bfloat162float(v.x);
          cs1 += __bfloat162float(v.y);
        }
      }
    }
  }
  __syncthreads();  // the stages are free: the epilogue uses them

  if constexpr (COLSUM) {
    float2* red = reinterpret_cast<float2*>(&st[0]);  // 4 x 32
    if (blockIdx.y == 0) {
      red[warp * 32 + lane] = make_float2(cs0, cs1);
      __syncthreads();
      if (warp == 0) {
        float2 t = red[lane];
        for (int w = 1; w < 4; ++w) {
          t.x += red[w * 32 + lane].x;
          t.y += red[w * 32 + lane].y;
        }
        *reinterpret_cast<float2*>(&colp[(size_t)blockIdx.z * N + n0 + 2 * lane]) = t;
      }
    }
  }

  const int g = lane >> 2, t = lane & 3;
  constexpr bool kF32 = EPI == kEpiF32 || EPI == kEpiBiasF32;
  bf16(*tile)[BN + PAD] = reinterpret_cast<bf16(*)[BN + PAD]>(&st[0]);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int tr = wm + mt * 16 + g + 8 * h, tc = wn + nt * 8 + 2 * t;
        const int row = m0 + tr, col = n0 + tc;
        float v0 = acc[mt][nt][2 * h], v1 = acc[mt][nt][2 * h + 1];
        if (EPI == kEpiBiasF32 || EPI == kEpiBiasReluBf16 || EPI == kEpiBiasBf16) {
          v0 += bias[col];
          v1 += bias[col + 1];
        }
        if (EPI == kEpiBiasReluBf16) {
          v0 = fmaxf(v0, 0.f);
          v1 = fmaxf(v1, 0.f);
        }
        if constexpr (kF32) {
          float* Cf = reinterpret_cast<float*>(C) + (EPI == kEpiF32 ? (size_t)blockIdx.z * M * N : 0);
          *reinterpret_cast<float2*>(&Cf[(size_t)row * N + col]) = make_float2(v0, v1);
        } else {
          *reinterpret_cast<__nv_bfloat162*>(&tile[tr][tc]) = __floats2bfloat162_rn(v0, v1);
        }
      }
  if constexpr (!kF32) {
    __syncthreads();
    auto masked = [](bf16 v, bf16 m) { return __bfloat162float(m) > 0.f ? v : __float2bfloat16_rn(0.f); };
    // C and the mask need no more than the alignment of a column pair: 16 bytes at a time where both have it (rows are
    // multiples of 128 bytes)
    const uintptr_t at = reinterpret_cast<uintptr_t>(C) | (EPI == kEpiMaskBf16 ? reinterpret_cast<uintptr_t>(mask) : 0);
    if (at % 16 == 0) {
#pragma unroll
      for (int it = threadIdx.x; it < (BM * BN) / 8; it += THREADS) {
        const int r = it / (BN / 8), c = (it % (BN / 8)) * 8;
        uint4 v = *reinterpret_cast<const uint4*>(&tile[r][c]);
        const size_t o = (size_t)(m0 + r) * N + n0 + c;
        if (EPI == kEpiMaskBf16) {
          const uint4 mk = *reinterpret_cast<const uint4*>(&mask[o]);
          const bf16* mv = reinterpret_cast<const bf16*>(&mk);
          bf16* vv = reinterpret_cast<bf16*>(&v);
#pragma unroll
          for (int q = 0; q < 8; ++q) vv[q] = masked(vv[q], mv[q]);
        }
        *reinterpret_cast<uint4*>(&reinterpret_cast<bf16*>(C)[o]) = v;
      }
    } else {
      for (int it = threadIdx.x; it < (BM * BN) / 2; it += THREADS) {
        const int r = it / (BN / 2), c = (it % (BN / 2)) * 2;
        __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&tile[r][c]);
        const size_t o = (size_t)(m0 + r) * N + n0 + c;
        if (EPI == kEpiMaskBf16) {
          const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162*>(&mask[o]);
          v.x = masked(v.x, mk.x);
          v.y = masked(v.y, mk.y);
        }
        *reinterpret_cast<__nv_bfloat162*>(&reinterpret_cast<bf16*>(C)[o]) = v;
      }
    }
  }
}

// out[i] = sum_s partials[s][i], fixed order.
__global__ void splitk_reduce_kernel(const float* __restrict__ p, int S, size_t count, float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  float s = 0.f;
  for (int k = 0; k < S; ++k) s += p[(size_t)k * count + i];
  out[i] = s;
}

// db[n] = sum_m dy[m][n] (bf16 input, f32 output), one block per 32 columns, fixed order.
__global__ void colsum_kernel(const bf16* __restrict__ dy, int M, int N, float* __restrict__ db) {
  __shared__ float red[8][33];
  const int col = blockIdx.x * 32 + (threadIdx.x & 31);
  const int ry = threadIdx.x >> 5;
  float s = 0.f;
  if (col < N)
    for (int m = ry; m < M; m += 8) s += __bfloat162float(dy[(size_t)m * N + col]);
  red[ry][threadIdx.x & 31] = s;
  __syncthreads();
  if (ry == 0 && col < N) {
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += red[k][threadIdx.x & 31];
    db[col] = t;
  }
}

// Two-stage column sums for tall matrices: stage 1, one CTA per (32 columns, kColsumRows rows) writes the chunk's
// column sums (8 row lanes x 32 columns, then the 8 lanes in order) to partial[chunk][col]; stage 2 adds the chunks
// of each column in chunk order. Deterministic; the whole GPU takes part instead of N / 32 CTAs.
constexpr int kColsumRows = 256;
__global__ void colsum_partial_kernel(const bf16* __restrict__ dy, int M, int N, float* __restrict__ partial) {
  __shared__ float red[8][33];
  const int col = blockIdx.x * 32 + (threadIdx.x & 31);
  const int ry = threadIdx.x >> 5;
  const int r0 = blockIdx.y * kColsumRows;
  const int r1 = min(M, r0 + kColsumRows);
  float s = 0.f;
  if (col < N)
    for (int m = r0 + ry; m < r1; m += 8) s += __bfloat162float(dy[(size_t)m * N + col]);
  red[ry][threadIdx.x & 31] = s;
  __syncthreads();
  if (ry == 0 && col < N) {
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += red[k][threadIdx.x & 31];
    partial[(size_t)blockIdx.y * N + col] = t;
  }
}

__global__ void colsum_final_kernel(const float* __restrict__ partial, int chunks, int N, float* __restrict__ db) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= N) return;
  float t = 0.f;
  for (int c = 0; c < chunks; ++c) t += partial[(size_t)c * N + col];
  db[col] = t;
}

// Squared-error gradient of the first `nout` output columns: dy = 2 w (y - target) for rows < valid, 0 elsewhere;
// per-row losses go to `row_loss` (FP32) for a fixed-order reduction. One thread per (row, V columns): 16-byte stores
// at V = 8 (41,984 x 64: 42 us with one thread walking a row, 4.5 us).
template <int V>
__global__ void mse_grad_kernel(const float* __restrict__ y, int M, int N, const float* __restrict__ target, int nout,
                                int valid, float w, bf16* __restrict__ dy, float* __restrict__ row_loss) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  chain_wait();
  const int per = N / V;
  const int r = (int)(i / per), c0 = (int)(i - (long long)r * per) * V;
  if (r >= M) return;
  __align__(16) bf16 g[V];
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int c = c0 + q;
    float v = 0.f;
    if (c < nout && r < valid) v = 2.f * w * (y[(size_t)r * N + c] - target[(size_t)r * nout + c]);
    g[q] = __float2bfloat16_rn(v);
  }
  if constexpr (V == 8)
    *reinterpret_cast<uint4*>(&dy[(size_t)r * N + c0]) = *reinterpret_cast<const uint4*>(g);
  else
    dy[(size_t)r * N + c0] = g[0];
  if (c0 == 0) {
    float l = 0.f;
    if (r < valid)
      for (int c = 0; c < nout; ++c) {
        const float d = y[(size_t)r * N + c] - target[(size_t)r * nout + c];
        l += d * d;
      }
    row_loss[r] = l;
  }
}

int launch_mse(const float* y, int M, int N, const float* target, int nout, int valid, float w, bf16* dy,
               float* row_loss, cudaStream_t st) {
  if (N % 8 == 0 && reinterpret_cast<uintptr_t>(dy) % 16 == 0)
    launch_chained(mse_grad_kernel<8>, (int)(((long long)M * (N / 8) + 255) / 256), 256, 0, st, y, M, N, target, nout,
                   valid, w, dy, row_loss);
  else
    launch_chained(mse_grad_kernel<1>, (int)(((long long)M * N + 255) / 256), 256, 0, st, y, M, N, target, nout, valid,
                   w, dy, row_loss);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

// The last stage of a training step's gradients: the split-K partials of every layer's weight gradient and column sums
// (one element per thread, splits in order), and in the last CTA the loss, w times the sum of the row losses (FP64,
// fixed order).
constexpr int kMaxLayers = LDDMM_MLP_MAX_LAYERS;
struct GradReduce {
  const float* part[2 * kMaxLayers];
  float* out[2 * kMaxLayers];
  int count[2 * kMaxLayers], splits[2 * kMaxLayers], end[2 * kMaxLayers];  // end: running total of the counts
  int total;
  const float* row_loss;
  int rows;
  float w;
  float* loss;
};
__global__ void __launch_bounds__(256) grad_reduce_kernel(const GradReduce R) {
  chain_wait();
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < R.rows; i += 256) s += (double)R.row_loss[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
      if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
      __syncthreads();
    }
    if (threadIdx.x == 0) R.loss[0] = (float)(red[0] * (double)R.w);
    return;
  }
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= R.total) return;
  int k = 0;
  while (i >= R.end[k]) ++k;
  const int e = i - (k ? R.end[k - 1] : 0), S = R.splits[k], n = R.count[k];
  const float* p = R.part[k] + e;
  float s = 0.f;
#pragma unroll 8
  for (int q = 0; q < S; ++q) s += p[(size_t)q * n];
  R.out[k][e] = s;
}

// Adam on FP32 master weights; writes the BF16 copy used by the GEMMs. Several tensors in one launch.
struct AdamTensors {
  float *p[LDDMM_ADAM_MAX_TENSORS], *m1[LDDMM_ADAM_MAX_TENSORS], *m2[LDDMM_ADAM_MAX_TENSORS];
  const float* g[LDDMM_ADAM_MAX_TENSORS];
  bf16* pb[LDDMM_ADAM_MAX_TENSORS];
  long long end[LDDMM_ADAM_MAX_TENSORS];  // running total of the element counts
  int n;
};
__global__ void adam_kernel(const AdamTensors T, float lr, float b1, float b2, float eps, float c1, float c2, float wd) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  chain_wait();
  if (i >= T.end[T.n - 1]) return;
  int k = 0;
  while (i >= T.end[k]) ++k;
  if (k) i -= T.end[k - 1];
  float *p = T.p[k], *m1 = T.m1[k], *m2 = T.m2[k];
  const float gi = T.g[k][i] + wd * p[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float v = p[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
  p[i] = v;
  if (T.pb[k]) T.pb[k][i] = __float2bfloat16_rn(v);
}

// disp[k] = tgt[argmin_l |src_k - tgt_l|] - src_k (FP32 distances, FP64 output); ties -> lowest index.
__global__ void nearest_kernel(const double* __restrict__ src, int n, const double* __restrict__ tgt, int m,
                               double* __restrict__ disp) {
  __shared__ float4 sm[256];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int kk = k < n ? k : n - 1;
  const float y0 = (float)src[3 * kk], y1 = (float)src[3 * kk + 1], y2 = (float)src[3 * kk + 2];
  float best = 3.4e38f;
  int arg = 0;
  for (int l0 = 0; l0 < m; l0 += blockDim.x) {
    const int l = l0 + threadIdx.x;
    if (l < m) sm[threadIdx.x] = make_float4((float)tgt[3 * l], (float)tgt[3 * l + 1], (float)tgt[3 * l + 2], 0.f);
    __syncthreads();
    const int cnt = min((int)blockDim.x, m - l0);
    for (int j = 0; j < cnt; ++j) {
      const float4 q = sm[j];
      const float d0 = y0 - q.x, d1 = y1 - q.y, d2 = y2 - q.z;
      const float d = d0 * d0 + d1 * d1 + d2 * d2;
      if (d < best) {
        best = d;
        arg = l0 + j;
      }
    }
    __syncthreads();
  }
  if (k < n)
    for (int c = 0; c < 3; ++c) disp[3 * k + c] = tgt[3 * arg + c] - src[3 * k + c];
}

template <bool TA, bool TB, int EPI, bool COLSUM = false>
int launch_gemm(int M, int N, int K, int splits, const void* A, const void* B, const float* bias, const void* mask,
                void* C, cudaStream_t st, float* colp = nullptr) {
  const int k_split = ((K + splits * BK - 1) / (splits * BK)) * BK;
  const int gz = (K + k_split - 1) / k_split;
  dim3 grid(N / BN, M / BM, gz);
  launch_chained(gemm_kernel<TA, TB, EPI, COLSUM>, grid, THREADS, 0, st, M, N, K, k_split,
                 reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(B), bias,
                 reinterpret_cast<const bf16*>(mask), C, colp);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

// The splits that launch_gemm makes of K.
inline int gemm_splits(int64_t K, int splits) {
  const int64_t k_split = ((K + splits * BK - 1) / (splits * BK)) * BK;
  return (int)((K + k_split - 1) / k_split);
}

bool bad_dims(const int64_t* dims, int layers, int64_t M) {
  if (layers < 1 || layers > kMaxLayers || dims == nullptr || M <= 0 || M % BM || M > INT32_MAX / 2 || M / BM > 65535)
    return true;
  for (int i = 0; i <= layers; ++i)
    if (dims[i] <= 0 || dims[i] % BN || dims[i] > 4096) return true;
  return false;
}

// h_0 = x, h_{i+1} = relu(h_i W_i + b_i), y = h_{last} W + b (FP32)
int forward(const int64_t* dims, int layers, const void* x, int64_t M, const void* const* W, const float* const* b,
            void* const* acts, float* y, cudaStream_t st) {
  const void* h = x;
  for (int i = 0; i < layers; ++i) {
    const int rc = i + 1 < layers
                       ? launch_gemm<false, false, kEpiBiasReluBf16>((int)M, (int)dims[i + 1], (int)dims[i], 1, h, W[i],
                                                                     b[i], nullptr, acts[i], st)
                       : launch_gemm<false, false, kEpiBiasF32>((int)M, (int)dims[i + 1], (int)dims[i], 1, h, W[i], b[i],
                                                                nullptr, y, st);
    if (rc != kOk) return rc;
    if (i + 1 < layers) h = acts[i];
  }
  return kOk;
}

// Rows of a split of the weight-gradient GEMMs, and the most splits.
constexpr int kSplitRows = 512, kMaxSplits = 64;

struct GradLayout {
  size_t acts[kMaxLayers], y, d[2], loss, part[kMaxLayers], colp[kMaxLayers], total;
  int splits;
};
GradLayout grad_layout(const int64_t* dims, int layers, int64_t M) {
  GradLayout L = {};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 255) & ~(size_t)255;
    return at;
  };
  int64_t wide = 0;
  for (int i = 1; i <= layers; ++i) wide = dims[i] > wide ? dims[i] : wide;
  for (int i = 0; i + 1 < layers; ++i) L.acts[i] = take((size_t)M * dims[i + 1] * sizeof(bf16));
  L.y = take((size_t)M * dims[layers] * sizeof(float));
  L.d[0] = take((size_t)M * wide * sizeof(bf16));
  L.d[1] = take((size_t)M * wide * sizeof(bf16));
  L.loss = take((size_t)M * sizeof(float));
  const int64_t want = M / kSplitRows;
  L.splits = gemm_splits(M, (int)(want < 1 ? 1 : (want > kMaxSplits ? kMaxSplits : want)));
  for (int i = 0; i < layers; ++i) {
    L.part[i] = take((size_t)L.splits * dims[i] * dims[i + 1] * sizeof(float));
    L.colp[i] = take((size_t)L.splits * dims[i + 1] * sizeof(float));
  }
  L.total = o;
  return L;
}

}  // namespace mlp
}  // namespace lddmm

using namespace lddmm;
using namespace lddmm::mlp;

extern "C" {

int lddmm_bf16_gemm(int trans_a, int trans_b, int epilogue, int64_t M, int64_t N, int64_t K, const void* A,
                    const void* B, const float* bias, const void* mask, void* C, int splits, float* split_ws,
                    size_t split_ws_bytes, lddmm_stream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || M % BM || N % BN || K % BK || M > INT32_MAX / 2 || N > 65536 || K > INT32_MAX / 2)
    return kInvalidArgument;
  if (A == nullptr || B == nullptr || C == nullptr || epilogue < 0 || epilogue > 4) return kInvalidArgument;
  if ((epilogue == kEpiBiasF32 || epilogue == kEpiBiasReluBf16 || epilogue == kEpiBiasBf16) && bias == nullptr)
    return kInvalidArgument;
  if (epilogue == kEpiMaskBf16 && mask == nullptr) return kInvalidArgument;
  if (splits < 1 || M / BM > 65535) return kInvalidArgument;
  if (splits > 1 && (epilogue != kEpiF32 || split_ws == nullptr)) return kInvalidArgument;
  cudaStream_t st = (cudaStream_t)stream;
  const int k_split = (int)(((K + splits * BK - 1) / (splits * BK)) * BK);
  const int gz = (int)((K + k_split - 1) / k_split);
  void* out = C;
  if (gz > 1) {
    if (split_ws_bytes < (size_t)gz * M * N * sizeof(float)) return kWorkspaceTooSmall;
    out = split_ws;
  }
  const int m = (int)M, n = (int)N, k = (int)K;
  int rc;
#define LDDMM_GEMM_CASE(ta, tb, epi) \
  if (trans_a == ta && trans_b == tb && epilogue == epi) rc = launch_gemm<ta, tb, epi>(m, n, k, gz, A, B, bias, mask, out, st); else
  LDDMM_GEMM_CASE(0, 0, kEpiF32) LDDMM_GEMM_CASE(0, 0, kEpiBiasF32) LDDMM_GEMM_CASE(0, 0, kEpiBiasReluBf16)
  LDDMM_GEMM_CASE(0, 0, kEpiBiasBf16) LDDMM_GEMM_CASE(0, 0, kEpiMaskBf16)
  LDDMM_GEMM_CASE(0, 1, kEpiF32) LDDMM_GEMM_CASE(0, 1, kEpiBiasF32) LDDMM_GEMM_CASE(0, 1, kEpiBiasReluBf16)
  LDDMM_GEMM_CASE(0, 1, kEpiBiasBf16) LDDMM_GEMM_CASE(0, 1, kEpiMaskBf16)
  LDDMM_GEMM_CASE(1, 0, kEpiF32) LDDMM_GEMM_CASE(1, 0, kEpiBiasF32) LDDMM_GEMM_CASE(1, 0, kEpiBiasReluBf16)
  LDDMM_GEMM_CASE(1, 0, kEpiBiasBf16) LDDMM_GEMM_CASE(1, 0, kEpiMaskBf16)
  LDDMM_GEMM_CASE(1, 1, kEpiF32) LDDMM_GEMM_CASE(1, 1, kEpiBiasF32) LDDMM_GEMM_CASE(1, 1, kEpiBiasReluBf16)
  LDDMM_GEMM_CASE(1, 1, kEpiBiasBf16) LDDMM_GEMM_CASE(1, 1, kEpiMaskBf16)
  return kInvalidArgument;
#undef LDDMM_GEMM_CASE
  if (rc != kOk) return rc;
  if (gz > 1) {
    const size_t count = (size_t)M * N;
    splitk_reduce_kernel<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(split_ws, gz, count,
                                                                          reinterpret_cast<float*>(C));
    if (cudaPeekAtLastError() != cudaSuccess) return kLaunchFailure;
  }
  return kOk;
}

int lddmm_bf16_colsum(const void* dy, int64_t M, int64_t N, float* db, float* ws, size_t ws_bytes,
                      lddmm_stream_t stream) {
  if (M < 0 || N <= 0 || dy == nullptr || db == nullptr || M > INT32_MAX || N > INT32_MAX) return kInvalidArgument;
  const int64_t chunks = (M + kColsumRows - 1) / kColsumRows;
  cudaStream_t st = (cudaStream_t)stream;
  if (ws == nullptr || chunks <= 1) {
    colsum_kernel<<<(unsigned)((N + 31) / 32), 256, 0, st>>>(reinterpret_cast<const bf16*>(dy), (int)M, (int)N, db);
  } else {
    if (ws_bytes < (size_t)chunks * (size_t)N * sizeof(float)) return kWorkspaceTooSmall;
    if (chunks > 65535) return kInvalidArgument;
    colsum_partial_kernel<<<dim3((unsigned)((N + 31) / 32), (unsigned)chunks), 256, 0, st>>>(
        reinterpret_cast<const bf16*>(dy), (int)M, (int)N, ws);
    colsum_final_kernel<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(ws, (int)chunks, (int)N, db);
  }
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

int lddmm_mse_grad(const float* y, int64_t M, int64_t N, const float* target, int64_t nout, int64_t valid, float w,
                   void* dy, float* row_loss, lddmm_stream_t stream) {
  if (M <= 0 || N <= 0 || nout < 1 || nout > N || valid < 0 || valid > M || y == nullptr || target == nullptr ||
      dy == nullptr || row_loss == nullptr || M > INT32_MAX)
    return kInvalidArgument;
  if (M * N / 256 >= INT32_MAX) return kInvalidArgument;
  return launch_mse(y, (int)M, (int)N, target, (int)nout, (int)valid, w, reinterpret_cast<bf16*>(dy), row_loss,
                    (cudaStream_t)stream);
}

int lddmm_adam_steps(int tensors, float* const* param, const float* const* grad, float* const* m1, float* const* m2,
                     void* const* param_bf16, const int64_t* count, float lr, float beta1, float beta2, float eps,
                     int64_t step, float weight_decay, lddmm_stream_t stream) {
  if (tensors < 1 || tensors > LDDMM_ADAM_MAX_TENSORS || step < 1 || param == nullptr || grad == nullptr ||
      m1 == nullptr || m2 == nullptr || param_bf16 == nullptr || count == nullptr)
    return kInvalidArgument;
  AdamTensors T = {};
  long long total = 0;
  for (int k = 0; k < tensors; ++k) {
    if (count[k] < 0 || param[k] == nullptr || grad[k] == nullptr || m1[k] == nullptr || m2[k] == nullptr)
      return kInvalidArgument;
    total += count[k];
    T.p[k] = param[k];
    T.g[k] = grad[k];
    T.m1[k] = m1[k];
    T.m2[k] = m2[k];
    T.pb[k] = reinterpret_cast<bf16*>(param_bf16[k]);
    T.end[k] = total;
  }
  T.n = tensors;
  if (total == 0) return kOk;
  if (total / 256 >= INT32_MAX) return kInvalidArgument;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  launch_chained(adam_kernel, (int)((total + 255) / 256), 256, 0, (cudaStream_t)stream, T, lr, beta1, beta2, eps, c1, c2,
                 weight_decay);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

int lddmm_adam_step(float* param, const float* grad, float* m1, float* m2, void* param_bf16, int64_t count, float lr,
                    float beta1, float beta2, float eps, int64_t step, float weight_decay, lddmm_stream_t stream) {
  return lddmm_adam_steps(1, &param, &grad, &m1, &m2, &param_bf16, &count, lr, beta1, beta2, eps, step, weight_decay,
                          stream);
}

int lddmm_mlp_forward(const int64_t* dims, int layers, const void* x, int64_t M, const void* const* W,
                      const float* const* b, void* const* acts, float* y, lddmm_stream_t stream) {
  if (bad_dims(dims, layers, M) || x == nullptr || W == nullptr || b == nullptr || y == nullptr ||
      (layers > 1 && acts == nullptr))
    return kInvalidArgument;
  for (int i = 0; i < layers; ++i)
    if (W[i] == nullptr || b[i] == nullptr || (i + 1 < layers && acts[i] == nullptr)) return kInvalidArgument;
  return forward(dims, layers, x, M, W, b, acts, y, (cudaStream_t)stream);
}

size_t lddmm_mlp_workspace_bytes(const int64_t* dims, int layers, int64_t M) {
  return bad_dims(dims, layers, M) ? 0 : grad_layout(dims, layers, M).total;
}

int lddmm_mlp_gradients(const int64_t* dims, int layers, const void* x, int64_t M, const void* const* W,
                        const float* const* b, const float* target, int64_t nout, int64_t valid, float w,
                        float* const* dW, float* const* db, float* loss, void* workspace, size_t workspace_bytes,
                        lddmm_stream_t stream) {
  if (bad_dims(dims, layers, M) || x == nullptr || W == nullptr || b == nullptr || target == nullptr || dW == nullptr ||
      db == nullptr || loss == nullptr || nout < 1 || nout > dims[layers] || valid < 0 || valid > M)
    return kInvalidArgument;
  for (int i = 0; i < layers; ++i)
    if (W[i] == nullptr || b[i] == nullptr || dW[i] == nullptr || db[i] == nullptr) return kInvalidArgument;
  const GradLayout L = grad_layout(dims, layers, M);
  if (workspace == nullptr || workspace_bytes < L.total) return kWorkspaceTooSmall;
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = reinterpret_cast<char*>(workspace);
  void* acts[kMaxLayers] = {};
  for (int i = 0; i + 1 < layers; ++i) acts[i] = ws + L.acts[i];
  float* y = reinterpret_cast<float*>(ws + L.y);
  float* row_loss = reinterpret_cast<float*>(ws + L.loss);
  int rc = forward(dims, layers, x, M, W, b, acts, y, st);
  if (rc != kOk) return rc;
  rc = launch_mse(y, (int)M, (int)dims[layers], target, (int)nout, (int)valid, w, reinterpret_cast<bf16*>(ws + L.d[0]),
                  row_loss, st);
  if (rc != kOk) return rc;
  GradReduce R = {};
  int at = 0;
  auto segment = [&](const float* part, float* out, int64_t count) {
    R.part[at] = part;
    R.out[at] = out;
    R.count[at] = (int)count;
    R.splits[at] = L.splits;
    R.total += (int)count;
    R.end[at++] = R.total;
  };
  int cur = 0;
  for (int i = layers - 1; i >= 0; --i) {
    const void* h = i > 0 ? acts[i - 1] : x;
    void* dy = ws + L.d[cur];
    float* part = reinterpret_cast<float*>(ws + L.part[i]);
    float* colp = reinterpret_cast<float*>(ws + L.colp[i]);
    rc = launch_gemm<true, false, kEpiF32, true>((int)dims[i], (int)dims[i + 1], (int)M, L.splits, h, dy, nullptr,
                                                 nullptr, part, st, colp);
    if (rc != kOk) return rc;
    segment(part, dW[i], dims[i] * dims[i + 1]);
    segment(colp, db[i], dims[i + 1]);
    if (i > 0) {
      rc = launch_gemm<false, true, kEpiMaskBf16>((int)M, (int)dims[i], (int)dims[i + 1], 1, dy, W[i], nullptr,
                                                  acts[i - 1], ws + L.d[1 - cur], st);
      if (rc != kOk) return rc;
      cur = 1 - cur;
    }
  }
  R.row_loss = row_loss;
  R.rows = (int)M;
  R.w = w;
  R.loss = loss;
  launch_chained(grad_reduce_kernel, (R.total + 255) / 256 + 1, 256, 0, st, R);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

int lddmm_nearest_displacement(const double* src, int64_t n, const double* tgt, int64_t m, double* disp,
                               lddmm_stream_t stream) {
  if (n < 0 || m <= 0 || (n > 0 && (src == nullptr || disp == nullptr)) || tgt == nullptr || n > INT32_MAX / 4 ||
      m > INT32_MAX / 4)
    return kInvalidArgument;
  if (n == 0) return kOk;
  nearest_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(src, (int)n, tgt, (int)m, disp);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kLaunchFailure;
}

}  // extern "C"
