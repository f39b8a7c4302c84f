// Multilayer perceptron of the learned self-energy update: forward, backward and Adam as
// hand-written kernels.  Weights are BF16 in the forward pass (FP32 master copies for the
// optimiser); every product accumulates in FP32.
//
//   z1 = x W1^T + b1, h1 = tanh(z1); z2 = h1 W2^T + b2, h2 = tanh(z2); y = h2 W3^T + b3
//   loss = mean over the batch and outputs of (y - t)^2
#include <algorithm>
#include <cmath>
#include <numeric>
#include <random>
#include <vector>

#include "mlp.cuh"

namespace cq {

namespace {

template <typename T> __device__ __forceinline__ float ld(const T* p, int64_t i);
template <> __device__ __forceinline__ float ld<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) {
  return __bfloat162float(p[i]);
}
// four consecutive elements at an address aligned to four elements
__device__ __forceinline__ float4 ld4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u),
                     __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u));
}

enum Epi { kStore = 0, kBias = 1, kBiasTanh = 2, kTanhGrad = 3 };

constexpr int TK = 16;  // K step of the SIMT GEMM

// A TT x TK operand tile on its way from global memory to shared memory: KC says that the
// element stride along K is 1 (a thread takes consecutive K of one row), otherwise the stride
// along the row index is 1 (a thread takes four consecutive rows of one K).
template <typename T, int TT, bool KC> struct TileLoad {
  static constexpr int E = TT * TK / 256;  // elements per thread
  float v[E];
  // rows r0 .. r0 + TT of an operand with R rows and leading stride ld, K range [k0, kend)
  __device__ __forceinline__ void load(const T* __restrict__ X, int64_t ld_, int64_t r0, int64_t R,
                                       int64_t k0, int64_t kend, bool vec) {
    const int t = threadIdx.x;
#pragma unroll
    for (int e = 0; e < E; e += 4) {
      int64_t r, k, i;
      bool in;
      if (KC) {
        r = r0 + t % TT;
        k = k0 + (t / TT) * E + e;
        i = r * ld_ + k;
        in = r < R && k + 3 < kend;
      } else {
        r = r0 + (t % (TT / 4)) * 4;
        k = k0 + t / (TT / 4) + (e / 4) * (1024 / TT);
        i = k * ld_ + r;
        in = r + 3 < R && k < kend;
      }
      if (vec && in) {
        const float4 q = ld4(X + i);
        v[e] = q.x;
        v[e + 1] = q.y;
        v[e + 2] = q.z;
        v[e + 3] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool ok = KC ? (r < R && k + j < kend) : (r + j < R && k < kend);
          v[e + j] = ok ? ld<T>(X, i + j) : 0.f;
        }
      }
    }
  }
  __device__ __forceinline__ void store(float (*S)[TT + 4]) const {
    const int t = threadIdx.x;
#pragma unroll
    for (int e = 0; e < E; e += 4) {
      if (KC) {
#pragma unroll
        for (int j = 0; j < 4; ++j) S[(t / TT) * E + e + j][t % TT] = v[e + j];
      } else {
        *reinterpret_cast<float4*>(&S[t / (TT / 4) + (e / 4) * (1024 / TT)][(t % (TT / 4)) * 4]) =
            make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      }
    }
  }
};

// C[m][n] = sum_k A(m, k) B(k, n) over this z-slice's K range; AK / BK: the K index of A / B is
// the contiguous one (lda, ldb then stride the row / column index), otherwise the row / column
// index is.  Epilogue: kBias adds bias[n], kBiasTanh also applies tanh, kTanhGrad multiplies by
// (1 - aux[m][n]^2) (backward through tanh).  gridDim.z > 1 writes the partial sums of the K
// slices one after the other into C (kStore only); k_sum_parts adds them.
//
// Bound by the FP32 pipe: 256 threads hold TT / 16 x TT / 16 outputs each (8 x 8 at TT = 128: 16
// words from shared memory feed 64 multiply-adds, as 32 packed FFMA2), the next K step is in
// registers while this one is multiplied, two shared-memory buffers, one barrier per step.
// 65536 x 256 x 256 on one B200: 240 us, 36 TFLOP/s; as a weight gradient in 74 slices 202 us.
template <int TT, typename TB, int EPI, bool AK, bool BK>
__global__ void __launch_bounds__(256, 2)
    k_gemm(const float* __restrict__ A, int64_t lda, const TB* __restrict__ B, int64_t ldb,
           float* __restrict__ C, int64_t ldc, int64_t M, int64_t N, int64_t K, int64_t kslice,
           int va, int vb, const TB* __restrict__ bias, const float* __restrict__ aux) {
  constexpr int R = TT / 16, G = R / 4;  // outputs per thread and dimension, in groups of four
  __shared__ float As[2][TK][TT + 4];
  __shared__ float Bs[2][TK][TT + 4];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int64_t m0 = (int64_t)blockIdx.x * TT, n0 = (int64_t)blockIdx.y * TT;
  const int64_t kb = (int64_t)blockIdx.z * kslice;
  const int64_t ke = kb + kslice < K ? kb + kslice : K;
  float2 acc[R][R / 2];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
  TileLoad<float, TT, AK> la;
  TileLoad<TB, TT, BK> lb;
  la.load(A, lda, m0, M, kb, ke, va);
  lb.load(B, ldb, n0, N, kb, ke, vb);
  la.store(As[0]);
  lb.store(Bs[0]);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = kb; k0 < ke; k0 += TK, buf ^= 1) {
    const bool more = k0 + TK < ke;
    if (more) {
      la.load(A, lda, m0, M, k0 + TK, ke, va);
      lb.load(B, ldb, n0, N, k0 + TK, ke, vb);
    }
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float a[R];
      float2 b[R / 2];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 x = *reinterpret_cast<const float4*>(&As[buf][kk][64 * g + 4 * ty]);
        const float4 y = *reinterpret_cast<const float4*>(&Bs[buf][kk][64 * g + 4 * tx]);
        a[4 * g] = x.x;
        a[4 * g + 1] = x.y;
        a[4 * g + 2] = x.z;
        a[4 * g + 3] = x.w;
        b[2 * g] = make_float2(y.x, y.y);
        b[2 * g + 1] = make_float2(y.z, y.w);
      }
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R / 2; ++j)
          acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[i][j]);
    }
    if (more) {  // the other buffer was last read before the previous barrier
      la.store(As[buf ^ 1]);
      lb.store(Bs[buf ^ 1]);
      __syncthreads();
    }
  }
  float* Cz = C + (int64_t)blockIdx.z * M * N;
  const bool vc = (ldc % 4 == 0) && ((reinterpret_cast<uintptr_t>(Cz) & 15) == 0) &&
                  (EPI != kTanhGrad || (reinterpret_cast<uintptr_t>(aux) & 15) == 0);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int64_t m = m0 + 64 * (i / 4) + 4 * ty + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int64_t n = n0 + 64 * g + 4 * tx;
      float v[4] = {acc[i][2 * g].x, acc[i][2 * g].y, acc[i][2 * g + 1].x, acc[i][2 * g + 1].y};
      if (vc && n + 3 < N) {
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
        if (EPI == kTanhGrad) h = *reinterpret_cast<const float4*>(aux + m * ldc + n);
        const float hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (EPI == kBias || EPI == kBiasTanh) v[j] += ld<TB>(bias, n + j);
          if (EPI == kBiasTanh) v[j] = tanhf(v[j]);
          if (EPI == kTanhGrad) v[j] *= 1.f - hh[j] * hh[j];
        }
        *reinterpret_cast<float4*>(Cz + m * ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (n + j >= N) break;
          if (EPI == kBias || EPI == kBiasTanh) v[j] += ld<TB>(bias, n + j);
          if (EPI == kBiasTanh) v[j] = tanhf(v[j]);
          if (EPI == kTanhGrad) {
            const float h = aux[m * ldc + n + j];
            v[j] *= 1.f - h * h;
          }
          Cz[m * ldc + n + j] = v[j];
        }
      }
    }
  }
}

// out[i] = sum_p part[p * stride + i], i < n, added in a fixed order: 32 outputs per block, the
// parts over eight rows of threads
__global__ void __launch_bounds__(256) k_sum_parts(const float* __restrict__ part, int64_t nparts,
                                                   int64_t stride, int64_t n,
                                                   float* __restrict__ out) {
  __shared__ float red[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + x;
  float s = 0.f;
  if (i < n) {
#pragma unroll 4
    for (int64_t p = y; p < nparts; p += 8) s += part[p * stride + i];
  }
  red[y][x] = s;
  __syncthreads();
  if (y == 0 && i < n) {
    for (int j = 1; j < 8; ++j) s += red[j][x];
    out[i] = s;
  }
}
void sum_parts(const float* part, int64_t nparts, int64_t stride, int64_t n, float* out,
               cudaStream_t s) {
  k_sum_parts<<<(unsigned)((n + 31) / 32), 256, 0, s>>>(part, nparts, stride, n, out);
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
}

template <int TT, typename TB, int EPI, bool AK, bool BK>
void gemm_tt(const float* A, int64_t lda, const TB* B, int64_t ldb, float* C, int64_t ldc, int64_t M,
             int64_t N, int64_t K, int64_t slices, int64_t kslice, const TB* bias, const float* aux,
             cudaStream_t s) {
  const int va = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  const int vb = ldb % 4 == 0 && (reinterpret_cast<uintptr_t>(B) & (4 * sizeof(TB) - 1)) == 0;
  const dim3 grid((unsigned)((M + TT - 1) / TT), (unsigned)((N + TT - 1) / TT), (unsigned)slices);
  k_gemm<TT, TB, EPI, AK, BK><<<grid, 256, 0, s>>>(A, lda, B, ldb, C, ldc, M, N, K, kslice, va, vb,
                                                   bias, aux);
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
}

// Slices that the K of an M x N weight gradient is cut into (1: not cut): at least 256 long, two
// blocks of 128 x 128 outputs per SM.
constexpr int64_t kSms = 148;
int64_t gemm_slices(int64_t M, int64_t N, int64_t K) {
  const int64_t t128 = ((M + 127) / 128) * ((N + 127) / 128);
  return std::min((K + 255) / 256, (2 * kSms + t128 - 1) / t128);
}

// Tiles of 128 x 128 when they fill the GPU, else 64 x 64.  A weight gradient has few tiles and
// a long K (the batch): the partial sums of its slices go through `part` and are added in slice
// order.
template <typename TB, int EPI, bool AK, bool BK>
void gemm(const float* A, int64_t lda, const TB* B, int64_t ldb, float* C, int64_t ldc, int64_t M,
          int64_t N, int64_t K, const TB* bias, const float* aux, DevBuf<float>& part,
          cudaStream_t s) {
  const int64_t t128 = ((M + 127) / 128) * ((N + 127) / 128);
  if constexpr (EPI == kStore) {
    const int64_t slices = gemm_slices(M, N, K);
    if (slices > 1) {
      const int64_t kslice = ((K + slices - 1) / slices + TK - 1) / TK * TK;
      const int64_t nz = (K + kslice - 1) / kslice;
      part.ensure(nz * M * N);
      gemm_tt<128, TB, EPI, AK, BK>(A, lda, B, ldb, part.p, N, M, N, K, nz, kslice, bias, aux, s);
      CQ_REQUIRE(ldc == N, COQUI_B200_EINVAL, "split gemm: contiguous result expected");
      sum_parts(part.p, nz, M * N, M * N, C, s);
      return;
    }
  }
  if (t128 >= kSms)
    gemm_tt<128, TB, EPI, AK, BK>(A, lda, B, ldb, C, ldc, M, N, K, 1, K, bias, aux, s);
  else
    gemm_tt<64, TB, EPI, AK, BK>(A, lda, B, ldb, C, ldc, M, N, K, 1, K, bias, aux, s);
}

// per-block sums over rows of A (bias gradients): part[block][c]; summed by k_sum_parts
__global__ void __launch_bounds__(256) k_colsum(const float* __restrict__ A, int64_t rows,
                                                int64_t cols, float* __restrict__ part) {
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    float sum = 0.f;
    for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) sum += A[r * cols + c];
    part[blockIdx.x * cols + c] = sum;
  }
}
int64_t colsum_blocks(int64_t rows) { return std::min<int64_t>(rows, 296); }
void colsum(const float* A, int64_t rows, int64_t cols, float* out, DevBuf<float>& part,
            cudaStream_t s) {
  const int64_t blocks = colsum_blocks(rows);
  part.ensure(blocks * cols);
  k_colsum<<<(unsigned)blocks, 256, 0, s>>>(A, rows, cols, part.p);
  count_launch();
  sum_parts(part.p, blocks, cols, cols, out, s);
}

// Output layer of a network with width <= 256 and dout <= 4, one warp per sample: y = h2 W3^T +
// b3 and, with GRAD, dy = 2 (y - t) / nout, dz2 = (dy W3) (1 - h2^2) and this block's sums for
// dW3 = dy^T h2, db2 = sum dz2, db3 = sum dy and the loss, laid out as part[block][DO * H + H +
// DO + 1].  Bound by memory: h2 is read once and dz2 written once, where separate products, the
// loss and the bias sums read them five times.
template <int DO, bool GRAD>
__global__ void __launch_bounds__(512) k_mlp_out(const float* __restrict__ h2,
                                                 const __nv_bfloat16* __restrict__ W3,
                                                 const __nv_bfloat16* __restrict__ b3,
                                                 const float* __restrict__ t, int64_t B, int H,
                                                 float* __restrict__ y, float* __restrict__ dz2,
                                                 float* __restrict__ part) {
  constexpr int NV = 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float nout = (float)(B * DO);
  float w[DO][NV], bias[DO], gw[DO][NV], gb2[NV], gb3[DO], loss = 0.f;
#pragma unroll
  for (int d = 0; d < DO; ++d) {
    bias[d] = __bfloat162float(b3[d]);
    gb3[d] = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      w[d][i] = c < H ? __bfloat162float(W3[d * H + c]) : 0.f;
      gw[d][i] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) gb2[i] = 0.f;
  for (int64_t r = (int64_t)blockIdx.x * nw + warp; r < B; r += (int64_t)gridDim.x * nw) {
    float h[NV], o[DO];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = lane + 32 * i;
      h[i] = c < H ? h2[r * H + c] : 0.f;
    }
#pragma unroll
    for (int d = 0; d < DO; ++d) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) s = fmaf(h[i], w[d][i], s);
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, x);
      o[d] = s + bias[d];
    }
    if (!GRAD) {
#pragma unroll
      for (int d = 0; d < DO; ++d)
        if (lane == d) y[r * DO + d] = o[d];
      continue;
    }
    float dy[DO];
#pragma unroll
    for (int d = 0; d < DO; ++d) {
      const float e = o[d] - t[r * DO + d];
      dy[d] = 2.f * e / nout;
      loss += e * e;
      gb3[d] += dy[d];
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float z = 0.f;
#pragma unroll
      for (int d = 0; d < DO; ++d) {
        z = fmaf(dy[d], w[d][i], z);
        gw[d][i] = fmaf(dy[d], h[i], gw[d][i]);
      }
      z *= 1.f - h[i] * h[i];
      gb2[i] += z;
      const int c = lane + 32 * i;
      if (c < H) dz2[r * H + c] = z;
    }
  }
  if (!GRAD) return;
  // the warps' sums in warp order, one column group at a time
  __shared__ float red[16][33];
  float* p = part + (int64_t)blockIdx.x * (DO * H + H + DO + 1);
  auto reduce = [&](float v, int64_t at, bool ok) {  // valid in warp 0
    __syncthreads();
    red[warp][lane] = v;
    __syncthreads();
    if (warp == 0) {
      float s = 0.f;
      for (int j = 0; j < nw; ++j) s += red[j][lane];
      if (ok) p[at] = s;
    }
  };
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + 32 * i;
#pragma unroll
    for (int d = 0; d < DO; ++d) reduce(gw[d][i], d * H + c, c < H);
    reduce(gb2[i], DO * H + c, c < H);
  }
#pragma unroll
  for (int d = 0; d < DO; ++d) reduce(gb3[d], DO * H + H + d, lane == 0);
  reduce(loss, DO * H + H + DO, lane == 0);
}

// Input layer's gradients for din <= 8: part[block][c * din + d] = sum_r dz1[r][c] x[r][d], then
// the bias sums part[block][H * din + c], over this block's rows; one column per thread, so dz1
// is read once, coalesced.
__global__ void __launch_bounds__(256) k_mlp_in_grad(const float* __restrict__ dz1,
                                                     const float* __restrict__ x, int64_t B, int H,
                                                     int din, float* __restrict__ part) {
  float* p = part + (int64_t)blockIdx.x * (H * din + H);
  const int64_t per = (B + gridDim.x - 1) / gridDim.x;
  const int64_t r0 = blockIdx.x * per, r1 = r0 + per < B ? r0 + per : B;
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float g[8] = {}, gb = 0.f;
#pragma unroll 4
    for (int64_t r = r0; r < r1; ++r) {
      const float z = dz1[r * H + c];
      gb += z;
#pragma unroll
      for (int d = 0; d < 8; ++d)
        if (d < din) g[d] = fmaf(z, __ldg(x + r * din + d), g[d]);
    }
#pragma unroll
    for (int d = 0; d < 8; ++d)
      if (d < din) p[c * din + d] = g[d];
    p[H * din + c] = gb;
  }
}

// dy = 2 (y - t) / n and per-block partial sums of (y - t)^2
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ t, float* __restrict__ dy,
                      int64_t n, float* __restrict__ part) {
  __shared__ float red[256];
  float sum = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float d = y[i] - t[i];
    dy[i] = 2.f * d / (float)n;
    sum += d * d;
  }
  red[threadIdx.x] = sum;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_adam(float* __restrict__ w, __nv_bfloat16* __restrict__ wb,
                       const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float c1, float c2) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    wb[i] = __float2bfloat16(wi);
  }
}

__global__ void k_to_bf16(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    wb[i] = __float2bfloat16(w[i]);
}

__global__ void k_gather_rows(const float* __restrict__ src, const int64_t* __restrict__ idx,
                              float* __restrict__ dst, int64_t rows, int64_t cols) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * cols;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / cols, c = i % cols;
    dst[i] = src[idx[r] * cols + c];
  }
}

// features (d1/d2, d2/d3) of each sequence, clamped to [-4, 4]; valid flag where the
// differences are resolved
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  const double d = b.x * b.x + b.y * b.y;
  return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ double2 csub2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

__global__ void k_extrap_features(const double2* __restrict__ h, int64_t nel, float* __restrict__ X,
                                  unsigned char* __restrict__ ok) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double2 s0 = h[e], s1 = h[nel + e], s2 = h[2 * nel + e], s3 = h[3 * nel + e];
    const double2 d1 = csub2(s3, s2), d2 = csub2(s2, s1), d3 = csub2(s1, s0);
    const double a1 = hypot(d1.x, d1.y), a2 = hypot(d2.x, d2.y), a3 = hypot(d3.x, d3.y);
    const double scale = fmax(fmax(hypot(s3.x, s3.y), 1e-300), 1e-300);
    const bool valid = a1 > 1e-14 * scale && a2 > 1e-14 * scale && a3 > 1e-14 * scale;
    ok[e] = valid ? 1 : 0;
    double2 q1 = make_double2(0, 0), q2 = make_double2(0, 0);
    if (valid) {
      q1 = cdiv(d1, d2);
      q2 = cdiv(d2, d3);
    }
    X[4 * e + 0] = (float)fmin(4.0, fmax(-4.0, q1.x));
    X[4 * e + 1] = (float)fmin(4.0, fmax(-4.0, q1.y));
    X[4 * e + 2] = (float)fmin(4.0, fmax(-4.0, q2.x));
    X[4 * e + 3] = (float)fmin(4.0, fmax(-4.0, q2.y));
  }
}

__global__ void k_extrap_apply(const double2* __restrict__ h, int64_t nel, const float* __restrict__ Y,
                               const unsigned char* __restrict__ ok, double max_jump,
                               double2* __restrict__ delta) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
       e += (int64_t)gridDim.x * blockDim.x) {
    double2 d = make_double2(0, 0);
    if (ok[e]) {
      const double2 d1 = csub2(h[3 * nel + e], h[2 * nel + e]);
      const double yr = Y[2 * e], yi = Y[2 * e + 1];
      d = make_double2(d1.x * yr - d1.y * yi, d1.x * yi + d1.y * yr);
      const double lim = max_jump * hypot(d1.x, d1.y), a = hypot(d.x, d.y);
      if (a > lim) {
        d.x *= lim / a;
        d.y *= lim / a;
      }
    }
    delta[e] = d;
  }
}

void ensure_batch(Mlp& n, int64_t B) {
  if (B <= n.cap) return;
  n.cap = 0;  // an allocation that fails leaves a buffer empty
  n.x.ensure(B * n.din);
  n.t.ensure(B * n.dout);
  n.h1.ensure(B * n.width);
  n.h2.ensure(B * n.width);
  n.y.ensure(B * n.dout);
  n.dy.ensure(B * n.dout);
  n.dh2.ensure(B * n.width);
  n.dh1.ensure(B * n.width);
  n.cap = B;
}

}  // namespace

void mlp_init(Mlp& n, int64_t din, int64_t width, int64_t dout, uint64_t seed, cudaStream_t s) {
  n.din = din;
  n.width = width;
  n.dout = dout;
  n.st = s;
  n.nparam = n.ob3() + dout;
  std::vector<float> h(n.nparam, 0.f);
  std::mt19937_64 rng(seed);
  auto fill = [&](int64_t off, int64_t rows, int64_t cols) {  // uniform(-a, a), a = sqrt(6/(fan_in+fan_out))
    const double a = std::sqrt(6.0 / (double)(rows + cols));
    std::uniform_real_distribution<double> u(-a, a);
    for (int64_t i = 0; i < rows * cols; ++i) h[off + i] = (float)u(rng);
  };
  fill(n.oW1(), width, din);
  fill(n.oW2(), width, width);
  fill(n.oW3(), dout, width);
  n.w.ensure(n.nparam);
  n.wb.ensure(n.nparam);
  n.g.ensure(n.nparam);
  n.m.ensure(n.nparam);
  n.v.ensure(n.nparam);
  CQ_CHECK_CUDA(cudaMemsetAsync(n.m.p, 0, n.nparam * sizeof(float), s));
  CQ_CHECK_CUDA(cudaMemsetAsync(n.v.p, 0, n.nparam * sizeof(float), s));
  n.adam_t = 0;
  mlp_set_params(n, h.data(), s);
}

void mlp_set_params(Mlp& n, const float* host, cudaStream_t s) {
  CQ_CHECK_CUDA(cudaMemcpyAsync(n.w.p, host, n.nparam * sizeof(float), cudaMemcpyHostToDevice, s));
  k_to_bf16<<<grid_for(n.nparam, 256), 256, 0, s>>>(n.w.p, n.wb.p, n.nparam);
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
}

// networks the fused output-layer kernel takes (the learned update's is 4 -> 256 -> 256 -> 2);
// others run the output layer as separate products
static bool fused_out(const Mlp& n) { return n.width <= 256 && n.dout <= 4; }
template <bool GRAD>
static void launch_out(Mlp& n, const float* t, int64_t B, float* y, unsigned blocks,
                       cudaStream_t s) {
  const __nv_bfloat16 *W3 = n.wb.p + n.oW3(), *b3 = n.wb.p + n.ob3();
  const int H = (int)n.width;
  switch (n.dout) {
    case 1: k_mlp_out<1, GRAD><<<blocks, 512, 0, s>>>(n.h2.p, W3, b3, t, B, H, y, n.dh2.p, n.part.p); break;
    case 2: k_mlp_out<2, GRAD><<<blocks, 512, 0, s>>>(n.h2.p, W3, b3, t, B, H, y, n.dh2.p, n.part.p); break;
    case 3: k_mlp_out<3, GRAD><<<blocks, 512, 0, s>>>(n.h2.p, W3, b3, t, B, H, y, n.dh2.p, n.part.p); break;
    default: k_mlp_out<4, GRAD><<<blocks, 512, 0, s>>>(n.h2.p, W3, b3, t, B, H, y, n.dh2.p, n.part.p); break;
  }
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
}
static int64_t out_blocks(int64_t B) { return std::min<int64_t>(148, (B + 15) / 16); }
static int64_t in_blocks(int64_t B) { return std::min<int64_t>(592, (B + 15) / 16); }

// h1, h2 of a batch
static void mlp_hidden(Mlp& n, const float* x, int64_t B, cudaStream_t s) {
  const __nv_bfloat16* W = n.wb.p;
  const int64_t H = n.width;
  gemm<__nv_bfloat16, kBiasTanh, true, true>(x, n.din, W + n.oW1(), n.din, n.h1.p, H, B, H, n.din,
                                             W + n.ob1(), nullptr, n.part, s);
  gemm<__nv_bfloat16, kBiasTanh, true, true>(n.h1.p, H, W + n.oW2(), H, n.h2.p, H, B, H, H,
                                             W + n.ob2(), nullptr, n.part, s);
}

void mlp_forward(Mlp& n, const float* x, int64_t B, float* y, cudaStream_t s) {
  ensure_batch(n, B);
  const __nv_bfloat16* W = n.wb.p;
  const int64_t H = n.width;
  mlp_hidden(n, x, B, s);
  if (fused_out(n))
    launch_out<false>(n, nullptr, B, y, (unsigned)out_blocks(B), s);
  else
    gemm<__nv_bfloat16, kBias, true, true>(n.h2.p, H, W + n.oW3(), H, y, n.dout, B, n.dout, H,
                                           W + n.ob3(), nullptr, n.part, s);
}

// Forward and backward of a 65536-sample batch of the 4 -> 256 -> 256 -> 2 network: 0.99 ms, 0.87 ms
// on the device, bound by the FP32 pipe in the three 65536 x 256 x 256 products (36-42 TFLOP/s).
// The weight gradients have few output tiles and are cut along the batch: uncut they take 40.7 ms,
// and their long sums leave the gradient 2.3e-6 from FP64 where the sliced ones leave 6e-8.
float mlp_backward(Mlp& n, const float* x, const float* t, int64_t B, cudaStream_t s) {
  ensure_batch(n, B);
  const int64_t H = n.width, D = n.dout, nout = B * D;
  float* g = n.g.p;
  const __nv_bfloat16* W = n.wb.p;
  std::vector<float> part;
  // one workspace for every split reduction below (growing it step by step would free and
  // allocate between the kernels of a first call): the slices of the weight gradients, the block
  // sums of the output layer, the input layer and the biases
  auto slices = [&](int64_t M, int64_t N) { return gemm_slices(M, N, B) * M * N; };
  n.part.ensure(std::max({slices(H, H),
                          n.din <= 8 ? in_blocks(B) * (H * n.din + H) : slices(H, n.din),
                          fused_out(n) ? out_blocks(B) * (D * H + H + D + 1) : slices(D, H),
                          colsum_blocks(B) * std::max(H, D)}));
  if (fused_out(n)) {
    mlp_hidden(n, x, B, s);
    const unsigned blocks = (unsigned)out_blocks(B);
    const int64_t np = D * H + H + D + 1;
    n.part.ensure(blocks * np);
    launch_out<true>(n, t, B, nullptr, blocks, s);
    // dW3, db3 follow each other in the parameters; db2 stands before them
    sum_parts(n.part.p, blocks, np, D * H, g + n.oW3(), s);
    sum_parts(n.part.p + D * H, blocks, np, H, g + n.ob2(), s);
    sum_parts(n.part.p + D * H + H, blocks, np, D, g + n.ob3(), s);
    n.lpart.ensure(148);
    part.resize(blocks);
    CQ_CHECK_CUDA(cudaMemcpy2DAsync(n.lpart.p, sizeof(float), n.part.p + np - 1,
                                    np * sizeof(float), sizeof(float), blocks,
                                    cudaMemcpyDeviceToDevice, s));
  } else {
    mlp_forward(n, x, B, n.y.p, s);
    const int nblk = 148;
    n.lpart.ensure(nblk);
    k_mse<<<nblk, 256, 0, s>>>(n.y.p, t, n.dy.p, nout, n.lpart.p);
    count_launch();
    // output layer: dW3 = dy^T h2, db3 = colsum(dy), dz2 = (dy W3) * (1 - h2^2)
    gemm<float, kStore, false, false>(n.dy.p, D, n.h2.p, H, g + n.oW3(), H, D, H, B, nullptr,
                                      nullptr, n.part, s);
    colsum(n.dy.p, B, D, g + n.ob3(), n.part, s);
    gemm<__nv_bfloat16, kTanhGrad, true, false>(n.dy.p, D, W + n.oW3(), H, n.dh2.p, H, B, H, D,
                                                nullptr, n.h2.p, n.part, s);
    colsum(n.dh2.p, B, H, g + n.ob2(), n.part, s);
    part.resize(nblk);
  }
  // dW2 = dz2^T h1; dz1 = (dz2 W2) * (1 - h1^2)
  gemm<float, kStore, false, false>(n.dh2.p, H, n.h1.p, H, g + n.oW2(), H, H, H, B, nullptr,
                                    nullptr, n.part, s);
  gemm<__nv_bfloat16, kTanhGrad, true, false>(n.dh2.p, H, W + n.oW2(), H, n.dh1.p, H, B, H, H,
                                              nullptr, n.h1.p, n.part, s);
  // dW1 = dz1^T x, db1 = colsum(dz1)
  if (n.din <= 8) {
    const unsigned blocks = (unsigned)in_blocks(B);
    const int64_t np = H * n.din + H;  // W1 and b1 follow each other
    n.part.ensure(blocks * np);
    k_mlp_in_grad<<<blocks, 256, 0, s>>>(n.dh1.p, x, B, (int)H, (int)n.din, n.part.p);
    count_launch();
    sum_parts(n.part.p, blocks, np, np, g + n.oW1(), s);
  } else {
    gemm<float, kStore, false, false>(n.dh1.p, H, x, n.din, g + n.oW1(), n.din, H, n.din, B,
                                      nullptr, nullptr, n.part, s);
    colsum(n.dh1.p, B, H, g + n.ob1(), n.part, s);
  }
  CQ_CHECK_CUDA(cudaGetLastError());
  CQ_CHECK_CUDA(cudaMemcpyAsync(part.data(), n.lpart.p, part.size() * sizeof(float),
                                cudaMemcpyDeviceToHost, s));
  CQ_CHECK_CUDA(cudaStreamSynchronize(s));
  double sum = 0;
  for (float v : part) sum += v;
  return (float)(sum / (double)nout);
}

void mlp_extrapolate(Mlp& n, const double2* hist, int64_t nel, double max_jump, double2* delta,
                     cudaStream_t s) {
  CQ_REQUIRE(n.din == 4 && n.dout == 2, COQUI_B200_EINVAL,
             "the extrapolating network takes 4 inputs and gives 2 outputs");
  DevBuf<float> X, Y;
  DevBuf<unsigned char> ok;
  X.ensure(nel * 4);
  Y.ensure(nel * 2);
  ok.ensure(nel);
  k_extrap_features<<<grid_for(nel, 256), 256, 0, s>>>(hist, nel, X.p, ok.p);
  count_launch();
  mlp_forward(n, X.p, nel, Y.p, s);
  k_extrap_apply<<<grid_for(nel, 256), 256, 0, s>>>(hist, nel, Y.p, ok.p, max_jump, delta);
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
  CQ_CHECK_CUDA(cudaStreamSynchronize(s));  // X, Y, ok are freed on return
}

void mlp_adam_step(Mlp& n, float lr, cudaStream_t s) {
  ++n.adam_t;
  const float c1 = 1.f - std::pow(0.9f, (float)n.adam_t);
  const float c2 = 1.f - std::pow(0.999f, (float)n.adam_t);
  k_adam<<<grid_for(n.nparam, 256), 256, 0, s>>>(n.w.p, n.wb.p, n.g.p, n.m.p, n.v.p, n.nparam, lr,
                                                 c1, c2);
  count_launch();
  CQ_CHECK_CUDA(cudaGetLastError());
}

}  // namespace cq

// ---------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------
struct coqui_b200_mlp {
  cq::Mlp net;
  std::string err;
};

cq::Mlp& mlp_net(coqui_b200_mlp* h) { return h->net; }

namespace {
template <typename F> int mlp_guarded(coqui_b200_mlp* h, F&& f) {
  if (!h) return COQUI_B200_EINVAL;
  try {
    CQ_CHECK_CUDA(cudaSetDevice(h->net.dev));
    f();
    CQ_CHECK_CUDA(cudaStreamSynchronize(h->net.st));
    h->err.clear();
    return COQUI_B200_OK;
  } catch (const cq::Error& e) {
    h->err = e.what();
    return e.code;
  } catch (const std::exception& e) {
    h->err = e.what();
    return COQUI_B200_EINVAL;
  }
}
}  // namespace

extern "C" {

int coqui_b200_mlp_create(coqui_b200_mlp** out, int64_t in_dim, int64_t width, int64_t out_dim,
                          uint64_t seed, int device) {
  if (!out || in_dim < 1 || width < 1 || out_dim < 1) return COQUI_B200_EINVAL;
  *out = nullptr;
  auto* h = new (std::nothrow) coqui_b200_mlp();
  if (!h) return COQUI_B200_ENOMEM;
  h->net.dev = device;
  int rc = mlp_guarded(h, [&] {
    CQ_CHECK_CUDA(cudaStreamCreateWithFlags(&h->net.st, cudaStreamNonBlocking));
    cq::mlp_init(h->net, in_dim, width, out_dim, seed, h->net.st);
  });
  if (rc != COQUI_B200_OK) {
    coqui_b200_mlp_destroy(h);
    return rc;
  }
  *out = h;
  return COQUI_B200_OK;
}

void coqui_b200_mlp_destroy(coqui_b200_mlp* h) {
  if (!h) return;
  cudaSetDevice(h->net.dev);
  if (h->net.st) cudaStreamSynchronize(h->net.st);
  cudaStream_t st = h->net.st;
  delete h;  // device buffers are freed by their destructors
  if (st) cudaStreamDestroy(st);
}

const char* coqui_b200_mlp_last_error(const coqui_b200_mlp* h) { return h ? h->err.c_str() : ""; }

int64_t coqui_b200_mlp_num_params(const coqui_b200_mlp* h) { return h ? h->net.nparam : 0; }

int coqui_b200_mlp_set_params(coqui_b200_mlp* h, const float* params) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(params, COQUI_B200_EINVAL, "null parameters");
    cq::mlp_set_params(h->net, params, h->net.st);
  });
}

int coqui_b200_mlp_get_params(coqui_b200_mlp* h, float* params) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(params, COQUI_B200_EINVAL, "null parameters");
    CQ_CHECK_CUDA(cudaMemcpyAsync(params, h->net.w.p, h->net.nparam * sizeof(float),
                                  cudaMemcpyDeviceToHost, h->net.st));
  });
}

int coqui_b200_mlp_forward(coqui_b200_mlp* h, const float* X, int64_t B, float* Y) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(X && Y && B >= 1, COQUI_B200_EINVAL, "bad arguments");
    cq::Mlp& n = h->net;
    cq::DevBuf<float> x, y;
    x.ensure(B * n.din);
    y.ensure(B * n.dout);
    CQ_CHECK_CUDA(cudaMemcpyAsync(x.p, X, B * n.din * sizeof(float), cudaMemcpyHostToDevice, n.st));
    cq::mlp_forward(n, x.p, B, y.p, n.st);
    CQ_CHECK_CUDA(cudaMemcpyAsync(Y, y.p, B * n.dout * sizeof(float), cudaMemcpyDeviceToHost, n.st));
    CQ_CHECK_CUDA(cudaStreamSynchronize(n.st));
  });
}

int coqui_b200_mlp_gradient(coqui_b200_mlp* h, const float* X, const float* T, int64_t B,
                            float* loss, float* grad) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(X && T && B >= 1 && loss && grad, COQUI_B200_EINVAL, "bad arguments");
    cq::Mlp& n = h->net;
    cq::ensure_batch(n, B);  // the network's own input buffers
    CQ_CHECK_CUDA(cudaMemcpyAsync(n.x.p, X, B * n.din * sizeof(float), cudaMemcpyHostToDevice, n.st));
    CQ_CHECK_CUDA(cudaMemcpyAsync(n.t.p, T, B * n.dout * sizeof(float), cudaMemcpyHostToDevice, n.st));
    *loss = cq::mlp_backward(n, n.x.p, n.t.p, B, n.st);
    CQ_CHECK_CUDA(cudaMemcpyAsync(grad, n.g.p, n.nparam * sizeof(float), cudaMemcpyDeviceToHost, n.st));
    CQ_CHECK_CUDA(cudaStreamSynchronize(n.st));
  });
}

int coqui_b200_mlp_extrapolate(coqui_b200_mlp* h, const double* hist, int64_t n, double max_jump,
                               double* delta) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(hist && delta && n >= 1 && max_jump > 0, COQUI_B200_EINVAL, "bad arguments");
    cq::Mlp& net = h->net;
    cq::DevBuf<double2> dh, dd;
    dh.ensure(4 * n);
    dd.ensure(n);
    CQ_CHECK_CUDA(cudaMemcpyAsync(dh.p, hist, 4 * n * sizeof(double2), cudaMemcpyHostToDevice, net.st));
    cq::mlp_extrapolate(net, dh.p, n, max_jump, dd.p, net.st);
    CQ_CHECK_CUDA(cudaMemcpyAsync(delta, dd.p, n * sizeof(double2), cudaMemcpyDeviceToHost, net.st));
    CQ_CHECK_CUDA(cudaStreamSynchronize(net.st));
  });
}

int coqui_b200_mlp_train(coqui_b200_mlp* h, const float* X, const float* T, int64_t n_samples,
                         int64_t batch, int64_t epochs, double lr, uint64_t seed,
                         float* loss_history) {
  return mlp_guarded(h, [&] {
    CQ_REQUIRE(X && T && n_samples >= 1 && batch >= 1 && epochs >= 1, COQUI_B200_EINVAL,
               "bad arguments");
    cq::Mlp& n = h->net;
    n.xall.ensure(n_samples * n.din);
    n.tall.ensure(n_samples * n.dout);
    CQ_CHECK_CUDA(cudaMemcpyAsync(n.xall.p, X, n_samples * n.din * sizeof(float),
                                  cudaMemcpyHostToDevice, n.st));
    CQ_CHECK_CUDA(cudaMemcpyAsync(n.tall.p, T, n_samples * n.dout * sizeof(float),
                                  cudaMemcpyHostToDevice, n.st));
    const int64_t B = std::min(batch, n_samples);
    n.idx.ensure(n_samples);
    cq::DevBuf<float> xb, tb;
    xb.ensure(B * n.din);
    tb.ensure(B * n.dout);
    std::vector<int64_t> perm(n_samples);
    std::iota(perm.begin(), perm.end(), 0);
    std::mt19937_64 rng(seed);
    for (int64_t ep = 0; ep < epochs; ++ep) {
      std::shuffle(perm.begin(), perm.end(), rng);
      CQ_CHECK_CUDA(cudaMemcpyAsync(n.idx.p, perm.data(), n_samples * sizeof(int64_t),
                                    cudaMemcpyHostToDevice, n.st));
      double sum = 0;
      int64_t nb = 0;
      for (int64_t b0 = 0; b0 + B <= n_samples; b0 += B) {
        cq::k_gather_rows<<<cq::grid_for(B * n.din, 256), 256, 0, n.st>>>(n.xall.p, n.idx.p + b0,
                                                                           xb.p, B, n.din);
        cq::k_gather_rows<<<cq::grid_for(B * n.dout, 256), 256, 0, n.st>>>(n.tall.p, n.idx.p + b0,
                                                                            tb.p, B, n.dout);
        cq::count_launch(2);
        sum += cq::mlp_backward(n, xb.p, tb.p, B, n.st);
        cq::mlp_adam_step(n, (float)lr, n.st);
        ++nb;
      }
      if (loss_history) loss_history[ep] = (float)(sum / std::max<int64_t>(nb, 1));
    }
  });
}

}  // extern "C"
