// mlp.cu -- hand-written forward / backward / Adam kernels of the warm-start MLP.
#include <cmath>
#include <random>
#include <vector>

#include "mlp.cuh"

namespace uvlm {
namespace {

constexpr float kInvSqrt2 = 0.70710678118654752f;
constexpr float kInvSqrt2Pi = 0.39894228040143268f;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * kInvSqrt2)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * kInvSqrt2)) + z * kInvSqrt2Pi * __expf(-0.5f * z * z);
}

// FP32 product C[r][c] = sum_i A'(i, r) B'(i, c) on the FMA pipe, in one form per
// operand layout:
// MODE 0 (forward):       A' = X[r][i] (ld K),  B' = W[i][c] (bf16, ld N)
// MODE 1 (backward-data): A' = dZ[r][i] (ld N), B' = W[c][i] (bf16, ld N)
// MODE 2 (weight grad):   A' = Aprev[i][r] (ld K), B' = dZ[i][c] (ld N)
// EPI 1: Z = acc + bias, A = GELU(Z); EPI 2: C = acc * GELU'(Zp[r][c]); EPI 0:
// the partial sums [blockIdx.z][r][c] of the inner range inner_per_z of the
// weight gradient, whose inner dimension is the batch (256 x 256 outputs are 16
// tiles only: on its own each of them summed 4096 rows in 310 us).
// 64 x 64 output tiles of 128 threads, 8 x 4 values each from 16-byte
// shared-memory reads (three per 32 FMAs), 32 inner steps at a time; the next
// step's 16-byte global loads are in registers while the FMAs run (32-row tiles
// and 16 inner steps: 1-8 % slower per call).  Every leading dimension is a
// multiple of 8 (8 features, 256 hidden units).  Forward and backward of 4096
// rows, the call with its copies: 1250 -> 410 us.
constexpr int kMmTR = 8, kMmRows = 8 * kMmTR, kMmTile = 64, kMmK = 32, kMmThreads = 128;

// Most splits of a weight gradient over the batch, and the fewest rows of one:
// 16 tiles x 32 splits of a 4096-row batch are 3.5 CTAs per SM.
constexpr int kMlpSplits = 32, kMlpSplitRows = 64;
constexpr int kMlpSumRows = 128;  // rows of one partial column sum

__device__ __forceinline__ void bf16x8(const uint4& u, float (&o)[8]) {
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    o[2 * k] = __uint_as_float(w[k] << 16);
    o[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
}

template <int MODE, int EPI>
__global__ void __launch_bounds__(kMmThreads) mlp_gemm(const float* __restrict__ A, const __nv_bfloat16* __restrict__ Wb,
                                                       const float* __restrict__ Bf, int rows, int cols, int inner,
                                                       int inner_per_z, int lda, int ldb,
                                                       const float* __restrict__ bias, const float* __restrict__ Zp,
                                                       float* __restrict__ C, float* __restrict__ Cact, int ldc) {
  constexpr int kA = kMmRows * kMmK / 4 / kMmThreads;  // 16-byte loads of one thread
  constexpr int kB = kMmTile * kMmK / 4 / kMmThreads, kW = kB / 2;
  __shared__ __align__(16) float As[kMmK][kMmRows + 4];
  __shared__ __align__(16) float Bs[kMmK][kMmTile + 4];
  const int row0 = blockIdx.x * kMmRows, col0 = blockIdx.y * kMmTile;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int begin = blockIdx.z * inner_per_z, end = min(inner, begin + inner_per_z);
  float4 av[kA], bv[kB];
  uint4 wv[kW];
  auto load = [&](int i0) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kA; ++t) {
      const int q = tid + kMmThreads * t;
      if (MODE == 2) {
        const int i = i0 + q / (kMmRows / 4), r = row0 + q % (kMmRows / 4) * 4;
        av[t] = i < end && r < rows ? *reinterpret_cast<const float4*>(A + (long long)i * lda + r) : zero;
      } else {
        const int r = row0 + q / (kMmK / 4), i = i0 + q % (kMmK / 4) * 4;
        av[t] = i < end && r < rows ? *reinterpret_cast<const float4*>(A + (long long)r * lda + i) : zero;
      }
    }
    if (MODE == 2) {
#pragma unroll
      for (int t = 0; t < kB; ++t) {
        const int q = tid + kMmThreads * t, i = i0 + q / (kMmTile / 4), c = col0 + q % (kMmTile / 4) * 4;
        bv[t] = i < end && c < cols ? *reinterpret_cast<const float4*>(Bf + (long long)i * ldb + c) : zero;
      }
    } else {
#pragma unroll
      for (int t = 0; t < kW; ++t) {
        const int q = tid + kMmThreads * t;
        const int i = MODE == 0 ? i0 + q / (kMmTile / 8) : i0 + q % (kMmK / 8) * 8;
        const int c = MODE == 0 ? col0 + q % (kMmTile / 8) * 8 : col0 + q / (kMmK / 8);
        wv[t] = i < end && c < cols
                    ? *reinterpret_cast<const uint4*>(Wb + (MODE == 0 ? (long long)i * ldb + c : (long long)c * ldb + i))
                    : make_uint4(0, 0, 0, 0);
      }
    }
  };
  auto store = [&]() {
#pragma unroll
    for (int t = 0; t < kA; ++t) {
      const int q = tid + kMmThreads * t;
      if (MODE == 2) {
        *reinterpret_cast<float4*>(&As[q / (kMmRows / 4)][q % (kMmRows / 4) * 4]) = av[t];
      } else {
        const int r = q / (kMmK / 4), k = q % (kMmK / 4) * 4;
        As[k][r] = av[t].x;
        As[k + 1][r] = av[t].y;
        As[k + 2][r] = av[t].z;
        As[k + 3][r] = av[t].w;
      }
    }
    if (MODE == 2) {
#pragma unroll
      for (int t = 0; t < kB; ++t) {
        const int q = tid + kMmThreads * t;
        *reinterpret_cast<float4*>(&Bs[q / (kMmTile / 4)][q % (kMmTile / 4) * 4]) = bv[t];
      }
    } else {
#pragma unroll
      for (int t = 0; t < kW; ++t) {
        const int q = tid + kMmThreads * t;
        float w[8];
        bf16x8(wv[t], w);
        if (MODE == 0) {
          float* p = &Bs[q / (kMmTile / 8)][q % (kMmTile / 8) * 8];
          *reinterpret_cast<float4*>(p) = make_float4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<float4*>(p + 4) = make_float4(w[4], w[5], w[6], w[7]);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) Bs[q % (kMmK / 8) * 8 + k][q / (kMmK / 8)] = w[k];
        }
      }
    }
  };
  float acc[kMmTR][4] = {};
  load(begin);
  for (int i0 = begin; i0 < end; i0 += kMmK) {
    __syncthreads();
    store();
    __syncthreads();
    if (i0 + kMmK < end) load(i0 + kMmK);
#pragma unroll
    for (int k = 0; k < kMmK; ++k) {
      float a[kMmTR];
#pragma unroll
      for (int u = 0; u < kMmTR; u += 4)
        *reinterpret_cast<float4*>(a + u) = *reinterpret_cast<const float4*>(&As[k][ty * kMmTR + u]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
#pragma unroll
      for (int u = 0; u < kMmTR; ++u) {
        acc[u][0] += a[u] * b.x;
        acc[u][1] += a[u] * b.y;
        acc[u][2] += a[u] * b.z;
        acc[u][3] += a[u] * b.w;
      }
    }
  }
  const int c = col0 + tx * 4;
  if (c >= cols) return;
  if (EPI == 0) C += (long long)blockIdx.z * rows * ldc;
#pragma unroll
  for (int u = 0; u < kMmTR; ++u) {
    const int R = row0 + ty * kMmTR + u;
    if (R >= rows) continue;
    const long long o = (long long)R * ldc + c;
    float4 v = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    if (EPI == 1) {
      const float4 bb = *reinterpret_cast<const float4*>(bias + c);
      v.x += bb.x, v.y += bb.y, v.z += bb.z, v.w += bb.w;
      *reinterpret_cast<float4*>(Cact + o) = make_float4(gelu(v.x), gelu(v.y), gelu(v.z), gelu(v.w));
    }
    if (EPI == 2) {
      const float4 z = *reinterpret_cast<const float4*>(Zp + o);
      v.x *= gelu_grad(z.x), v.y *= gelu_grad(z.y), v.z *= gelu_grad(z.z), v.w *= gelu_grad(z.w);
    }
    *reinterpret_cast<float4*>(C + o) = v;
  }
}

// out[q] = sum of the splits' partial sums, in order, in FP64
template <typename P>
__global__ void sum_splits(const P* __restrict__ part, int splits, int n, float* __restrict__ out) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    double s = 0;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) s += (double)part[(long long)z * n + q];
    out[q] = (float)s;
  }
}

// last layer (out = 1): y[b] = out_scale * (A[b] . w + b0), warp per row
__global__ void head_forward(const float* __restrict__ A, int B, int K, const __nv_bfloat16* __restrict__ w,
                             const float* __restrict__ b0, const float* __restrict__ norm, float* y) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (row >= B) return;
  float s = 0;
  for (int k = lane; k < K; k += 32) s += A[row * K + k] * __bfloat162float(w[k]);
  for (int off = 16; off; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (lane == 0) y[row] = (s + b0[0]) * norm[2 * kMlpIn];
}

// x' = (x - mean) / std into act[0] (ld kMlpIn)
__global__ void normalise_inputs(const float* __restrict__ x, long long B, const float* __restrict__ norm, float* a0) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < B * kMlpIn; q += (long long)gridDim.x * blockDim.x) {
    const int f = (int)(q % kMlpIn);
    a0[q] = (x[q] - norm[f]) / norm[kMlpIn + f];
  }
}

// dy = 2 (y - t) / (B s^2) on the network output scale; loss partial sums
__global__ void loss_grad(const float* __restrict__ y, const float* __restrict__ t, long long B,
                          const float* __restrict__ norm, float* dy, double* loss) {
  __shared__ double sh[8];
  const float s = norm[2 * kMlpIn];
  double acc = 0;
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < B; b += (long long)gridDim.x * blockDim.x) {
    const float e = (y[b] - t[b]) / s;  // error in network units
    acc += (double)e * e;
    dy[b] = 2.f * e / (float)B;
  }
  for (int off = 16; off; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0;
    for (int i = 0; i < (int)(blockDim.x / 32); ++i) v += sh[i];
    atomicAdd(loss, v / (double)B);
  }
}

// head backward: dW4[k] = sum_b A[b][k] dy[b]; db4 = sum_b dy[b];
// dZ3[b][k] = dy[b] * w[k] * GELU'(Z3[b][k])
__global__ void head_backward_data(const float* __restrict__ dy, long long B, int K, const __nv_bfloat16* __restrict__ w,
                                   const float* __restrict__ Z, float* dZ) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < B * K; q += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(q % K);
    const long long b = q / K;
    dZ[q] = dy[b] * __bfloat162float(w[k]) * gelu_grad(Z[q]);
  }
}

// Column sums of one range of rows: part[blockIdx.y][c] = sum_b M[b][c] *
// (wvec ? wvec[b] : 1) in FP64, 32 columns and kMlpSumRows rows per CTA with the
// rows along the warps (one CTA per column read a sector for every value).
__global__ void __launch_bounds__(256) column_sums(const float* __restrict__ M, long long B, int cols,
                                                   const float* __restrict__ wvec, double* __restrict__ part) {
  __shared__ double sh[8][33];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  const long long b0 = (long long)blockIdx.y * kMlpSumRows, b1 = min(B, b0 + kMlpSumRows);
  double s = 0;
  if (c < cols) {
#pragma unroll 4
    for (long long b = b0 + wid; b < b1; b += 8) s += (double)M[b * cols + c] * (wvec ? wvec[b] : 1.f);
  }
  sh[wid][lane] = s;
  __syncthreads();
  if (wid == 0 && c < cols) {
#pragma unroll
    for (int w = 1; w < 8; ++w) s += sh[w][lane];
    part[(long long)blockIdx.y * cols + c] = s;
  }
}

__global__ void __launch_bounds__(256) vector_sum(const float* __restrict__ v, long long n, float* out) {
  __shared__ double sh[8];
  double s = 0;
  for (long long b = threadIdx.x; b < n; b += 256) s += (double)v[b];
  for (int off = 16; off; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    s = 0;
    for (int i = 0; i < 8; ++i) s += sh[i];
    out[0] = (float)s;
  }
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, size_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2, __nv_bfloat16* pb) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float upd = lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    const float pi = p[i] - upd;
    p[i] = pi;
    pb[i] = __float2bfloat16(pi);
  }
}

__global__ void to_bf16(const float* p, size_t n, __nv_bfloat16* pb) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    pb[i] = __float2bfloat16(p[i]);
}

__global__ void features_kernel(int num, int R, int C, const double* g_n, const double* g_nm1, const double* b_np1,
                                const double* b_n, const double* phase, float* feat) {
  const int per = R * C;
  const int N = per * num;
  for (int K = blockIdx.x * blockDim.x + threadIdx.x; K < N; K += gridDim.x * blockDim.x) {
    const int n = K / per, i = (K % per) / C, j = K % C;
    float* f = feat + (long long)K * kMlpIn;
    f[0] = (float)g_n[K];
    f[1] = (float)(g_n[K] - g_nm1[K]);
    f[2] = (float)b_np1[K];
    f[3] = (float)(b_np1[K] - b_n[K]);
    f[4] = (float)sin(phase[n]);
    f[5] = (float)cos(phase[n]);
    f[6] = 2.f * (i + 0.5f) / R - 1.f;
    f[7] = 2.f * (j + 0.5f) / C - 1.f;
  }
}

__global__ void guess_kernel(int N, const double* g_n, const double* g_nm1, const float* y, double* x0) {
  for (int K = blockIdx.x * blockDim.x + threadIdx.x; K < N; K += gridDim.x * blockDim.x)
    x0[K] = 2.0 * g_n[K] - g_nm1[K] + (double)y[K];
}

__global__ void targets_kernel(int N, const double* g_np1, const double* g_n, const double* g_nm1, float* t) {
  for (int K = blockIdx.x * blockDim.x + threadIdx.x; K < N; K += gridDim.x * blockDim.x)
    t[K] = (float)(g_np1[K] - (2.0 * g_n[K] - g_nm1[K]));
}

inline int g1(long long n) { return (int)std::min<long long>(std::max<long long>((n + 255) / 256, 1), 8192); }

}  // namespace

Error mlp_create(Mlp* m, unsigned long long seed) {
  mlp_free(m);
  const int dims[kMlpDepth + 2] = {kMlpIn, kMlpHidden, kMlpHidden, kMlpHidden, 1};
  size_t off = 0;
  for (int l = 0; l <= kMlpDepth; ++l) {
    m->layer[l].in = dims[l];
    m->layer[l].out = dims[l + 1];
    m->layer[l].w_off = off;
    off += (size_t)dims[l] * dims[l + 1];
    m->layer[l].b_off = off;
    off += dims[l + 1];
  }
  m->n_params = off;
  std::vector<float> p(off, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l <= kMlpDepth; ++l) {
    const float lim = std::sqrt(3.0f / (float)m->layer[l].in) * (l == kMlpDepth ? 0.1f : 1.0f);
    std::uniform_real_distribution<float> U(-lim, lim);
    for (size_t q = 0; q < (size_t)m->layer[l].in * m->layer[l].out; ++q) p[m->layer[l].w_off + q] = U(rng);
  }
  UVLM_CUDA_TRY(cudaMalloc(&m->master, sizeof(float) * off));
  UVLM_CUDA_TRY(cudaMalloc(&m->wbf, sizeof(__nv_bfloat16) * off));
  UVLM_CUDA_TRY(cudaMalloc(&m->grad, sizeof(float) * off));
  UVLM_CUDA_TRY(cudaMalloc(&m->adam_m, sizeof(float) * off));
  UVLM_CUDA_TRY(cudaMalloc(&m->adam_v, sizeof(float) * off));
  UVLM_CUDA_TRY(cudaMalloc(&m->norm, sizeof(float) * (2 * kMlpIn + 1)));
  UVLM_CUDA_TRY(cudaMalloc(&m->loss, sizeof(double)));
  UVLM_CUDA_TRY(cudaMemcpy(m->master, p.data(), sizeof(float) * off, cudaMemcpyHostToDevice));
  UVLM_CUDA_TRY(cudaMemset(m->adam_m, 0, sizeof(float) * off));
  UVLM_CUDA_TRY(cudaMemset(m->adam_v, 0, sizeof(float) * off));
  for (int f = 0; f < kMlpIn; ++f) {
    m->h_norm[f] = 0.f;
    m->h_norm[kMlpIn + f] = 1.f;
  }
  m->h_norm[2 * kMlpIn] = 1.f;
  UVLM_CUDA_TRY(cudaMemcpy(m->norm, m->h_norm, sizeof(m->h_norm), cudaMemcpyHostToDevice));
  m->adam_t = 0;
  return mlp_sync_bf16(m, 0);
}

void mlp_free(Mlp* m) {
  cudaFree(m->master);
  cudaFree(m->wbf);
  cudaFree(m->grad);
  cudaFree(m->adam_m);
  cudaFree(m->adam_v);
  cudaFree(m->norm);
  cudaFree(m->loss);
  cudaFree(m->act);
  cudaFree(m->pre);
  cudaFree(m->dact);
  cudaFree(m->part);
  cudaFree(m->colpart);
  cudaFree(m->y);
  cudaFree(m->dy);
  cudaFree(m->wT);
  cudaFree(m->tc_err);
  *m = Mlp{};
}

Error mlp_reserve(Mlp* m, long long B) {
  if (B <= m->cap) return ok();
  cudaFree(m->act);
  cudaFree(m->pre);
  cudaFree(m->dact);
  cudaFree(m->y);
  cudaFree(m->dy);
  cudaFree(m->colpart);
  m->colpart = nullptr;
  m->act = m->pre = m->dact = m->y = m->dy = nullptr;
  const size_t H = kMlpHidden;
  UVLM_CUDA_TRY(cudaMalloc(&m->act, sizeof(float) * (kMlpDepth + 1) * B * H));
  UVLM_CUDA_TRY(cudaMalloc(&m->pre, sizeof(float) * kMlpDepth * B * H));
  UVLM_CUDA_TRY(cudaMalloc(&m->dact, sizeof(float) * 2 * B * H));
  UVLM_CUDA_TRY(cudaMalloc(&m->y, sizeof(float) * B));
  UVLM_CUDA_TRY(cudaMalloc(&m->dy, sizeof(float) * B));
  m->cap = B;
  return ok();
}

Error mlp_sync_bf16(Mlp* m, cudaStream_t st) {
  m->version += 1;
  to_bf16<<<g1((long long)m->n_params), 256, 0, st>>>(m->master, m->n_params, m->wbf);
  UVLM_LAUNCH_CHECK();
  return ok();
}

Error mlp_forward(Mlp* m, const float* x, long long B, float* y, cudaStream_t st) {
  if (B <= 0) return ok();
  UVLM_TRY(mlp_reserve(m, B));
  const long long H = kMlpHidden;
  normalise_inputs<<<g1(B * kMlpIn), 256, 0, st>>>(x, B, m->norm, m->act);
  UVLM_LAUNCH_CHECK();
  for (int l = 0; l < kMlpDepth; ++l) {
    const MlpLayer& L = m->layer[l];
    const float* Ain = m->act + (long long)l * B * H;
    float* Z = m->pre + (long long)l * B * H;
    float* Aout = m->act + (long long)(l + 1) * B * H;
    dim3 grid(ceil_div(B, kMmRows), ceil_div(L.out, kMmTile));
    mlp_gemm<0, 1><<<grid, kMmThreads, 0, st>>>(Ain, m->wbf + L.w_off, nullptr, (int)B, L.out, L.in, L.in, L.in, L.out,
                                                m->master + L.b_off, nullptr, Z, Aout, L.out);
    UVLM_LAUNCH_CHECK();
  }
  const MlpLayer& Lh = m->layer[kMlpDepth];
  head_forward<<<ceil_div(B, 8), 256, 0, st>>>(m->act + (long long)kMlpDepth * B * H, (int)B, Lh.in,
                                               m->wbf + Lh.w_off, m->master + Lh.b_off, m->norm, y ? y : m->y);
  UVLM_LAUNCH_CHECK();
  return ok();
}

Error mlp_loss_backward(Mlp* m, const float* x, const float* target, long long B, double* loss_host,
                        cudaStream_t st) {
  UVLM_TRY(mlp_forward(m, x, B, m->y, st));
  if (!m->part) UVLM_CUDA_TRY(cudaMalloc(&m->part, sizeof(float) * (size_t)kMlpSplits * kMlpHidden * kMlpHidden));
  if (!m->colpart)
    UVLM_CUDA_TRY(cudaMalloc(&m->colpart, sizeof(double) * (size_t)ceil_div(m->cap, kMlpSumRows) * kMlpHidden));
  const long long H = kMlpHidden;
  UVLM_CUDA_TRY(cudaMemsetAsync(m->loss, 0, sizeof(double), st));
  loss_grad<<<std::min(g1(B), 1024), 256, 0, st>>>(m->y, target, B, m->norm, m->dy, m->loss);
  UVLM_LAUNCH_CHECK();
  // head: dW4 = A3^T dy, db4 = sum dy, dZ3 = dy w4 GELU'(Z3)
  const MlpLayer& Lh = m->layer[kMlpDepth];
  const float* A3 = m->act + (long long)kMlpDepth * B * H;
  const int sums = ceil_div(B, kMlpSumRows);
  column_sums<<<dim3(ceil_div(Lh.in, 32), sums), 256, 0, st>>>(A3, B, Lh.in, m->dy, m->colpart);
  UVLM_LAUNCH_CHECK();
  sum_splits<<<ceil_div(Lh.in, 32), 32, 0, st>>>(m->colpart, sums, Lh.in, m->grad + Lh.w_off);
  UVLM_LAUNCH_CHECK();
  vector_sum<<<1, 256, 0, st>>>(m->dy, B, m->grad + Lh.b_off);
  UVLM_LAUNCH_CHECK();
  float* dZ = m->dact;            // dZ of the current layer
  float* dZnext = m->dact + B * H;
  head_backward_data<<<g1(B * Lh.in), 256, 0, st>>>(m->dy, B, Lh.in, m->wbf + Lh.w_off,
                                                    m->pre + (long long)(kMlpDepth - 1) * B * H, dZ);
  UVLM_LAUNCH_CHECK();
  for (int l = kMlpDepth - 1; l >= 0; --l) {
    const MlpLayer& L = m->layer[l];
    const float* Ain = m->act + (long long)l * B * H;
    // dW = Ain^T dZ  [in x out], db = column sums of dZ
    // split over the batch in pieces of at least kMlpSplitRows rows
    const int per = std::max<int>(kMlpSplitRows, ceil_div(ceil_div(B, kMlpSplits), kMmK) * kMmK);
    const int splits = ceil_div(B, per);
    dim3 gw(ceil_div(L.in, kMmRows), ceil_div(L.out, kMmTile), splits);
    mlp_gemm<2, 0><<<gw, kMmThreads, 0, st>>>(Ain, nullptr, dZ, L.in, L.out, (int)B, per, L.in, L.out, nullptr, nullptr,
                                              m->part, nullptr, L.out);
    UVLM_LAUNCH_CHECK();
    sum_splits<<<g1((long long)L.in * L.out), 256, 0, st>>>(m->part, splits, L.in * L.out, m->grad + L.w_off);
    UVLM_LAUNCH_CHECK();
    column_sums<<<dim3(ceil_div(L.out, 32), sums), 256, 0, st>>>(dZ, B, L.out, nullptr, m->colpart);
    UVLM_LAUNCH_CHECK();
    sum_splits<<<ceil_div(L.out, 32), 32, 0, st>>>(m->colpart, sums, L.out, m->grad + L.b_off);
    UVLM_LAUNCH_CHECK();
    if (l > 0) {
      // dZ_{l-1} = (dZ W^T) * GELU'(Z_{l-1})
      dim3 gd(ceil_div(B, kMmRows), ceil_div(L.in, kMmTile));
      mlp_gemm<1, 2><<<gd, kMmThreads, 0, st>>>(dZ, m->wbf + L.w_off, nullptr, (int)B, L.in, L.out, L.out, L.out, L.out,
                                                nullptr, m->pre + (long long)(l - 1) * B * H, dZnext, nullptr, L.in);
      UVLM_LAUNCH_CHECK();
      std::swap(dZ, dZnext);
    }
  }
  if (loss_host) {
    UVLM_CUDA_TRY(cudaMemcpyAsync(loss_host, m->loss, sizeof(double), cudaMemcpyDeviceToHost, st));
    UVLM_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return ok();
}

Error mlp_adam_step(Mlp* m, float lr, cudaStream_t st) {
  m->adam_t += 1;
  m->version += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - (float)std::pow(b1, (double)m->adam_t);
  const float c2 = 1.f - (float)std::pow(b2, (double)m->adam_t);
  adam_kernel<<<g1((long long)m->n_params), 256, 0, st>>>(m->master, m->grad, m->adam_m, m->adam_v, m->n_params, lr,
                                                          b1, b2, 1e-8f, c1, c2, m->wbf);
  UVLM_LAUNCH_CHECK();
  return ok();
}

Error mlp_features(int num, int R, int C, const double* g_n, const double* g_nm1, const double* b_np1,
                   const double* b_n, const double* phase, float* feat, cudaStream_t st) {
  features_kernel<<<g1((long long)num * R * C), 256, 0, st>>>(num, R, C, g_n, g_nm1, b_np1, b_n, phase, feat);
  UVLM_LAUNCH_CHECK();
  return ok();
}

Error mlp_apply_guess(int N, const double* g_n, const double* g_nm1, const float* y, double* x0, cudaStream_t st) {
  guess_kernel<<<g1(N), 256, 0, st>>>(N, g_n, g_nm1, y, x0);
  UVLM_LAUNCH_CHECK();
  return ok();
}

Error mlp_targets(int N, const double* g_np1, const double* g_n, const double* g_nm1, float* t, cudaStream_t st) {
  targets_kernel<<<g1(N), 256, 0, st>>>(N, g_np1, g_n, g_nm1, t);
  UVLM_LAUNCH_CHECK();
  return ok();
}

}  // namespace uvlm
