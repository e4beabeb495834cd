// Kernels of the Fourier-neural-operator surrogate (forward, backward, Adam).
//
// The FNO is small (width 32, 16 x 16 retained modes); its dense contractions --
// truncated DFTs written as products with DFT matrices, the pointwise channel
// maps, the projection, the weight gradients -- run on the tensor-core GEMM
// (fno_umma.cu).  The per-mode complex channel mixing of the spectral
// convolution, bias + GELU, channel reductions, the relative-L2 loss and the
// Adam update have their own element-wise kernels here.  FP32 throughout, FP64
// accumulation in the reductions.
#include <cuda_runtime.h>
#include <math.h>
#include "fno_act.cuh"
#include "fw_internal.h"

namespace fw {

// Spectral mixing.  F: [B][Cin][2][K] (real block then imaginary block of the
// K retained modes), R: [Cin][Cout][2][K], O: [B][Cout][2][K].
// forward:   O[b][o][k] = sum_i F[b][i][k] R[i][o][k]
__global__ void mix_fwd_kernel(int Bn, int Ci, int Co, int K, const float* F, const float* R, float* O) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)Bn * Co * K) return;
  const int k = idx % K;
  const int o = (idx / K) % Co;
  const int b = idx / ((long long)K * Co);
  float re = 0.f, im = 0.f;
  for (int i = 0; i < Ci; ++i) {
    const float fr = F[(((size_t)b * Ci + i) * 2) * K + k], fi = F[(((size_t)b * Ci + i) * 2 + 1) * K + k];
    const float rr = R[(((size_t)i * Co + o) * 2) * K + k], ri = R[(((size_t)i * Co + o) * 2 + 1) * K + k];
    re += fr * rr - fi * ri;
    im += fr * ri + fi * rr;
  }
  O[(((size_t)b * Co + o) * 2) * K + k] = re;
  O[(((size_t)b * Co + o) * 2 + 1) * K + k] = im;
}
// dF[b][i][k] = sum_o dO[b][o][k] conj(R[i][o][k])
__global__ void mix_bwd_in_kernel(int Bn, int Ci, int Co, int K, const float* dO, const float* R, float* dF) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)Bn * Ci * K) return;
  const int k = idx % K;
  const int i = (idx / K) % Ci;
  const int b = idx / ((long long)K * Ci);
  float re = 0.f, im = 0.f;
  for (int o = 0; o < Co; ++o) {
    const float gr = dO[(((size_t)b * Co + o) * 2) * K + k], gi = dO[(((size_t)b * Co + o) * 2 + 1) * K + k];
    const float rr = R[(((size_t)i * Co + o) * 2) * K + k], ri = R[(((size_t)i * Co + o) * 2 + 1) * K + k];
    re += gr * rr + gi * ri;
    im += gi * rr - gr * ri;
  }
  dF[(((size_t)b * Ci + i) * 2) * K + k] = re;
  dF[(((size_t)b * Ci + i) * 2 + 1) * K + k] = im;
}
// dR[i][o][k] = sum_b conj(F[b][i][k]) dO[b][o][k]
__global__ void mix_bwd_w_kernel(int Bn, int Ci, int Co, int K, const float* F, const float* dO, float* dR) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)Ci * Co * K) return;
  const int k = idx % K;
  const int o = (idx / K) % Co;
  const int i = idx / ((long long)K * Co);
  double re = 0.0, im = 0.0;
  for (int b = 0; b < Bn; ++b) {
    const float fr = F[(((size_t)b * Ci + i) * 2) * K + k], fi = F[(((size_t)b * Ci + i) * 2 + 1) * K + k];
    const float gr = dO[(((size_t)b * Co + o) * 2) * K + k], gi = dO[(((size_t)b * Co + o) * 2 + 1) * K + k];
    re += (double)fr * gr + (double)fi * gi;
    im += (double)fr * gi - (double)fi * gr;
  }
  dR[(((size_t)i * Co + o) * 2) * K + k] = (float)re;
  dR[(((size_t)i * Co + o) * 2 + 1) * K + k] = (float)im;
}

// pre = X + bias[c]; Y = act ? gelu(pre) : pre.  X, pre, Y: [B][C][L]
__global__ void bias_act_kernel(long long n, int C, long long L, const float* X, const float* bias, float* pre,
                                float* Y, int act) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int c = (i / L) % C;
    const float p = X[i] + bias[c];
    if (pre) pre[i] = p;
    Y[i] = act ? gelu(p) : p;
  }
}
// dpre = act ? dY * gelu'(pre) : dY
__global__ void act_bwd_kernel(long long n, const float* dY, const float* pre, float* dpre, int act) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dpre[i] = act ? dY[i] * gelu_d(pre[i]) : dY[i];
}
// out[c] (+)= sum_{b, l} X[b][c][l]; one 1024-thread block per channel, FP64
// accumulation, float4 loads (four in flight per thread) when L % 4 == 0 and X
// is 16-byte aligned
constexpr int kCsumThreads = 1024;
__global__ void __launch_bounds__(kCsumThreads) channel_sum_kernel(int Bn, int C, long long L, const float* X,
                                                                   float* out, int accumulate, int vec) {
  const int c = blockIdx.x;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  for (int b = 0; b < Bn; ++b) {
    const float* x = X + ((size_t)b * C + c) * L;
    if (vec) {
      const float4* x4 = reinterpret_cast<const float4*>(x);
      const long long n4 = L / 4;
      long long l = threadIdx.x;
      for (; l + 3 * kCsumThreads < n4; l += 4 * kCsumThreads) {
        const float4 a = __ldg(x4 + l), b1 = __ldg(x4 + l + kCsumThreads), c1 = __ldg(x4 + l + 2 * kCsumThreads),
                     d = __ldg(x4 + l + 3 * kCsumThreads);
        s0 += (double)a.x + a.y + (double)a.z + a.w;
        s1 += (double)b1.x + b1.y + (double)b1.z + b1.w;
        s2 += (double)c1.x + c1.y + (double)c1.z + c1.w;
        s3 += (double)d.x + d.y + (double)d.z + d.w;
      }
      for (; l < n4; l += kCsumThreads) {
        const float4 a = __ldg(x4 + l);
        s0 += (double)a.x + a.y + (double)a.z + a.w;
      }
    } else {
      for (long long l = threadIdx.x; l < L; l += kCsumThreads) s0 += x[l];
    }
  }
  double s = (s0 + s1) + (s2 + s3);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double red[kCsumThreads / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) out[c] = (float)(t + (accumulate ? (double)out[c] : 0.0));
  }
}
// loss_b = ||Y_b - T_b||^2 / ||T_b||^2; dY = 2 (Y - T) / ||T_b||^2 / B.  One block per sample.
__global__ void rel_l2_kernel(long long L, const float* Y, const float* T, float* dY, double* loss, int Bn) {
  const int b = blockIdx.x;
  const float* y = Y + (size_t)b * L;
  const float* t = T + (size_t)b * L;
  double e = 0.0, n = 0.0;
  for (long long l = threadIdx.x; l < L; l += blockDim.x) {
    const double d = (double)y[l] - t[l];
    e += d * d;
    n += (double)t[l] * t[l];
  }
  __shared__ double r1[256], r2[256];
  r1[threadIdx.x] = e;
  r2[threadIdx.x] = n;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      r1[threadIdx.x] += r1[threadIdx.x + o];
      r2[threadIdx.x] += r2[threadIdx.x + o];
    }
    __syncthreads();
  }
  const double nn = r2[0] > 0 ? r2[0] : 1.0;
  if (threadIdx.x == 0) loss[b] = r1[0] / nn;
  if (dY) {
    const float s = (float)(2.0 / nn / Bn);
    for (long long l = threadIdx.x; l < L; l += blockDim.x) dY[(size_t)b * L + l] = s * (y[l] - t[l]);
  }
}
__global__ void adam_kernel(long long n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                            float eps, float bc1, float bc2, float wd) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * p[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  }
}
// lift input: feats[b][f][p][x], f = 0..(NP-1): sample parameters, NP, NP+1: x, p coordinates (normalised)
__global__ void features_kernel(int Bn, int NP, int G0, int G1, const float* params, const float* xs, const float* ps,
                                float* out) {
  const long long L = (long long)G0 * G1;
  const long long n = (long long)Bn * (NP + 2) * L;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long l = i % L;
    const int f = (i / L) % (NP + 2);
    const int b = i / (L * (NP + 2));
    float v;
    if (f < NP) v = params[(size_t)b * NP + f];
    else if (f == NP) v = xs[l % G1];
    else v = ps[l / G1];
    out[i] = v;
  }
}

}  // namespace fw

using namespace fw;

static int grid1(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b > 8192 ? 8192 : (b < 1 ? 1 : b));
}

extern "C" int fw_fno_mix(int mode, int Bn, int Ci, int Co, int K, const float* X, const float* Y, float* out,
                          void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (mode == 0) mix_fwd_kernel<<<grid1((long long)Bn * Co * K), 256, 0, st>>>(Bn, Ci, Co, K, X, Y, out);
  else if (mode == 1) mix_bwd_in_kernel<<<grid1((long long)Bn * Ci * K), 256, 0, st>>>(Bn, Ci, Co, K, X, Y, out);
  else if (mode == 2) mix_bwd_w_kernel<<<grid1((long long)Ci * Co * K), 256, 0, st>>>(Bn, Ci, Co, K, X, Y, out);
  else return fail(FW_EINVAL, "fw_fno_mix: mode must be 0 (forward), 1 (input grad) or 2 (weight grad)");
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_mix");
}

extern "C" int fw_fno_bias_act(long long n, int C, long long L, const float* X, const float* bias, float* pre, float* Y,
                               int act, void* stream) {
  bias_act_kernel<<<grid1(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, C, L, X, bias, pre, Y, act);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_bias_act");
}

extern "C" int fw_fno_act_bwd(long long n, const float* dY, const float* pre, float* dpre, int act, void* stream) {
  act_bwd_kernel<<<grid1(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, dY, pre, dpre, act);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_act_bwd");
}

extern "C" int fw_fno_channel_sum(int Bn, int C, long long L, const float* X, float* out, int accumulate,
                                  void* stream) {
  const int vec = (L % 4 == 0) && ((reinterpret_cast<uintptr_t>(X) & 15u) == 0);
  channel_sum_kernel<<<C, kCsumThreads, 0, static_cast<cudaStream_t>(stream)>>>(Bn, C, L, X, out, accumulate, vec);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_channel_sum");
}

// ---------------------------------------------------------------------------
// Weight gradients out[r][c] = sum_b sum_l dY[b][r][l] X[b][c][l] (and the bias
// gradients sum dY[b][r][l]) over channel-major activations, in FP32 FMAs.  The
// contraction runs over every pixel and gives 32 x 32 outputs a tile, so the
// tensor core has nothing to reuse: its operands had to be split and stored to
// shared memory for 12 MMAs a chunk (0.32 ms a layer at 16 x 256^2; this kernel
// 0.07, near the time of reading both operands once).  A CTA stages 32 + 32 rows of
// 128 pixels; each of its eight warps contracts 16 of them for the whole tile,
// lane (rg, cg) owning rows rg + 8 i and columns cg + 4 j (128 FMAs per 12 vector
// loads without bank conflicts).  A weight's chain adds at most 256 products in FP32
// (kFlush stages); warps, flushes and CTAs are summed in FP64.  The bias sums are FP64
// from the first addition, and stay so between CTAs as a high and a low float.
namespace wgrad {
constexpr int TP = 128, PITCH = TP + 4;
constexpr int kFlush = 16;  // stages of 16 products a thread
constexpr size_t SMEM = (size_t)2 * 32 * PITCH * 4;
}  // namespace wgrad

__global__ void __launch_bounds__(256, 2) wgrad_kernel(int rows, int cols, long long L, long long range, int nr,
                                                       const float* __restrict__ dY, long long sY,
                                                       const float* __restrict__ X, long long sX, float* __restrict__ work,
                                                       float* __restrict__ bwork) {
  using namespace wgrad;
  extern __shared__ __align__(16) float sm[];
  float* Ys = sm;
  float* Xs = sm + 32 * PITCH;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = lane >> 2, cg = lane & 3;
  const int r0 = (blockIdx.x % nr) * 32, c0 = (blockIdx.x / nr) * 32;
  const int split = blockIdx.z * gridDim.y + blockIdx.y;  // (sample, range)
  const long long l0 = (long long)blockIdx.y * range, l1 = l0 + range < L ? l0 + range : L;
  const float* y = dY + (long long)blockIdx.z * sY;
  const float* x = X + (long long)blockIdx.z * sX;
  const bool wb = bwork != nullptr && c0 == 0;
  float acc[4][8];
  double bs[4] = {0, 0, 0, 0}, ws[4] = {0, 0, 0, 0};  // bias sums of rows rg + 8 i; weights tid + 256 i of the tile
  auto clear = [&] {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  };
  // the warps' chains through shared memory (8 x 1024 floats) into ws
  auto flush = [&] {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sm[warp * 1024 + (rg + 8 * i) * 32 + cg + 4 * j] = acc[i][j];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double s = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += (double)sm[w * 1024 + tid + 256 * i];
      ws[i] += s;
    }
  };
  clear();
  float4 ry[4], rx[4];
  auto fetch = [&](long long l) {  // warp w: rows w, w + 8, ...; lane: four pixels
    const bool in = l + 4 * lane < l1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + warp + 8 * i, c = c0 + warp + 8 * i;
      ry[i] = in && r < rows ? __ldg(reinterpret_cast<const float4*>(y + r * L + l + 4 * lane)) : make_float4(0, 0, 0, 0);
      rx[i] = in && c < cols ? __ldg(reinterpret_cast<const float4*>(x + c * L + l + 4 * lane)) : make_float4(0, 0, 0, 0);
    }
  };
  fetch(l0);
  int stage = 0;
  for (long long l = l0; l < l1; l += TP) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *reinterpret_cast<float4*>(Ys + (warp + 8 * i) * PITCH + 4 * lane) = ry[i];
      *reinterpret_cast<float4*>(Xs + (warp + 8 * i) * PITCH + 4 * lane) = rx[i];
    }
    __syncthreads();
    if (l + TP < l1) fetch(l + TP);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int p = warp * 16 + 4 * q;
      float4 b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(Xs + (cg + 4 * j) * PITCH + p);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(Ys + (rg + 8 * i) * PITCH + p);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
        }
      }
    }
    if (wb)  // lane cg: a quarter of the warp's pixels
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(Ys + (rg + 8 * i) * PITCH + warp * 16 + 4 * cg);
        bs[i] += ((double)a.x + (double)a.y) + ((double)a.z + (double)a.w);
      }
    if (++stage == kFlush && l + TP < l1) {
      flush();
      clear();
      stage = 0;
    }
  }
  flush();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = tid + 256 * i, r = r0 + (e >> 5), c = c0 + (e & 31);
    if (r < rows && c < cols) work[(long long)split * rows * cols + (long long)r * cols + c] = (float)ws[i];
  }
  if (wb) {
    double* bd = reinterpret_cast<double*>(sm);  // [warp][row]
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bs[i] += __shfl_xor_sync(0xffffffffu, bs[i], 1);
      bs[i] += __shfl_xor_sync(0xffffffffu, bs[i], 2);
      if (cg == 0) bd[warp * 32 + rg + 8 * i] = bs[i];
    }
    __syncthreads();
    if (tid < 32 && r0 + tid < rows) {
      double s = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += bd[w * 32 + tid];
      float* o = bwork + 2 * ((long long)split * rows + r0 + tid);
      o[0] = (float)s;
      o[1] = (float)(s - (double)o[0]);
    }
  }
}

// out[e] = sum over Z slices (FP64) for the E weights, then the R bias sums
__global__ void wgrad_sum_kernel(int Z, int E, int R, const float* __restrict__ work, const float* __restrict__ bwork,
                                 float* out, float* bias) {
  const int e = blockIdx.x * 32 + threadIdx.x;
  const bool w = e < E;
  double s = 0.0;
  if (e < E + R)
    for (int z = threadIdx.y; z < Z; z += 8) {
      if (w) {
        s += (double)work[(long long)z * E + e];
      } else {
        const float* b = bwork + 2 * ((long long)z * R + e - E);
        s += (double)b[0] + (double)b[1];
      }
    }
  __shared__ double red[8][33];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && e < E + R) {
    double t = 0.0;
#pragma unroll
    for (int y = 0; y < 8; ++y) t += red[y][threadIdx.x];
    if (w) out[e] = (float)t;
    else bias[e - E] = (float)t;
  }
}

// Pixel ranges per sample: two CTAs per SM over the launch, at least 512 pixels
// a range (a multiple of the 128-pixel stage).
static void wgrad_ranges(int rows, int cols, long long L, int batch, int* ns, long long* range) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long tiles = (long long)((rows + 31) / 32) * ((cols + 31) / 32) * batch;
  long long want = (4LL * sms + tiles - 1) / tiles;
  if (want > (L + 511) / 512) want = (L + 511) / 512;
  if (want < 1) want = 1;
  *range = ((L + want - 1) / want + wgrad::TP - 1) / wgrad::TP * wgrad::TP;
  *ns = (int)((L + *range - 1) / *range);
}

static int wgrad_check(int rows, int cols, long long L, int batch) {
  if (rows < 1 || cols < 1 || L < 4 || L % 4 != 0 || L > (1LL << 30) || batch < 1 || batch > 65535 || rows > 4096 || cols > 4096)
    return fail(FW_EINVAL, "fw_fno_wgrad_bias: sizes must be positive, L a multiple of 4");
  return FW_OK;
}

extern "C" int fw_fno_wgrad_bias_work(int rows, int cols, long long L, int batch, long long* floats_out) {
  if (floats_out == nullptr) return fail(FW_EINVAL, "fw_fno_wgrad_bias_work: NULL argument");
  if (int rc = wgrad_check(rows, cols, L, batch)) return rc;
  int ns;
  long long range;
  wgrad_ranges(rows, cols, L, batch, &ns, &range);
  *floats_out = (long long)batch * ns * rows * (cols + 2);
  return FW_OK;
}

extern "C" int fw_fno_wgrad_bias(int rows, int cols, long long L, const float* dY, long long strideY, const float* X,
                                 long long strideX, int batch, float* work, long long work_floats, float* out, float* bias,
                                 void* stream) {
  if (int rc = wgrad_check(rows, cols, L, batch)) return rc;
  if (dY == nullptr || X == nullptr || work == nullptr || out == nullptr) return fail(FW_EINVAL, "fw_fno_wgrad_bias: NULL argument");
  if ((((uintptr_t)dY | (uintptr_t)X) & 15u) != 0 || strideY % 4 != 0 || strideX % 4 != 0)
    return fail(FW_EINVAL, "fw_fno_wgrad_bias: operands must start on 16 bytes");
  int ns;
  long long range;
  wgrad_ranges(rows, cols, L, batch, &ns, &range);
  const long long z = (long long)batch * ns;
  if (work_floats < z * rows * (cols + 2)) return fail(FW_EINVAL, "fw_fno_wgrad_bias: work buffer too small");
  float* bwork = bias != nullptr ? work + z * rows * cols : nullptr;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int nr = (rows + 31) / 32, nc = (cols + 31) / 32;
  wgrad_kernel<<<dim3(nr * nc, ns, batch), 256, wgrad::SMEM, st>>>(rows, cols, L, range, nr, dY, strideY, X, strideX, work, bwork);
  const int E = rows * cols, R = bias != nullptr ? rows : 0;
  wgrad_sum_kernel<<<(E + R + 31) / 32, dim3(32, 8), 0, st>>>((int)z, E, R, work, bwork, out, bias);
  count_launch(2);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_wgrad_bias");
}

// ---------------------------------------------------------------------------
// Backward pass of the projection out = Q2 GELU(Q1 v + c1) + c2 (128 hidden, 32
// channels) for d = d(loss)/d(out): the hidden layer is evaluated again tile by
// tile, so neither it nor its gradient touches memory (128 channels of 4 bytes a
// pixel, written twice and read five times as separate products: 2.9 ms at
// 16 x 256^2; this kernel reads v and d and writes dv).  Per tile of 64 pixels:
//   h = Q1 v + c1;  dh = Q2 d GELU'(h);  dc1 += dh;  dQ2 += GELU(h) d     4 x 8 (j, x) a thread
//   dv = Q1^T dh                                   4 x 8 (c, x) a thread, a quarter of j each
//   dQ1 += dh v^T                                  4 x 4 (j, c) a thread
// Every product reads two or three 16-byte vectors per 32 FMAs.  Tile sums add up
// in FP64.
namespace projb {
constexpr int H = 128, C = 32, TX = 64, PX = TX + 4;
constexpr int F_Q1T = 0, F_Q1N = C * H, F_V = 2 * C * H, F_D = F_V + C * PX, F_DH = F_D + TX, F_RED = F_DH + H * PX,
              FLOATS = F_RED + 4 * C * PX;
constexpr int REC = H * C + 2 * H + 1;  // dQ1, dc1, dQ2, dc2 of a block
}  // namespace projb

__global__ void __launch_bounds__(256, 2) project_bwd_kernel(long long L, int batch, const float* __restrict__ V, long long sV,
                                                             const float* __restrict__ Q1, const float* __restrict__ c1,
                                                             const float* __restrict__ Q2, const float* __restrict__ dout,
                                                             float* __restrict__ dV, double* __restrict__ work) {
  using namespace projb;
  extern __shared__ __align__(16) float sm[];
  float *q1t = sm + F_Q1T, *q1n = sm + F_Q1N, *vs = sm + F_V, *ds = sm + F_D, *dh = sm + F_DH, *red = sm + F_RED;
  const int tid = threadIdx.x;
  for (int i = tid; i < H * C; i += 256) {
    const float q = __ldg(Q1 + i);
    q1n[i] = q;
    q1t[(i % C) * H + i / C] = q;
  }
  const int tj = tid >> 3, t8 = tid & 7;  // hidden rows 4 tj .. + 3 (h), tj + 32 i (dQ1); pixels 4 t8, 32 + 4 t8; channels t8 + 8 i
  float b1[4], w2[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    b1[i] = __ldg(c1 + 4 * tj + i);
    w2[i] = __ldg(Q2 + 4 * tj + i);
  }
  double gq[4][4], gc[4], g2[4], gd = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    gc[i] = g2[i] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) gq[i][j] = 0;
  }
  const long long per = (L + TX - 1) / TX, total = per * batch;
  const long long first = blockIdx.x * total / gridDim.x, last = (blockIdx.x + 1) * total / gridDim.x;
  float4 rv[2], rd;
  auto fetch = [&](long long t) {
    const long long b = t / per, l = (t - b * per) * TX;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (tid >> 4) + 16 * i;
      const long long p = l + 4 * (tid & 15);
      rv[i] = p < L ? __ldg(reinterpret_cast<const float4*>(V + b * sV + c * L + p)) : make_float4(0, 0, 0, 0);
    }
    if (tid < TX / 4) {
      const long long p = l + 4 * tid;
      rd = p < L ? __ldg(reinterpret_cast<const float4*>(dout + b * L + p)) : make_float4(0, 0, 0, 0);
    }
  };
  if (first < last) fetch(first);
  for (long long t = first; t < last; ++t) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(vs + ((tid >> 4) + 16 * i) * PX + 4 * (tid & 15)) = rv[i];
    if (tid < TX / 4) {
      *reinterpret_cast<float4*>(ds + 4 * tid) = rd;
      gd += ((double)rd.x + (double)rd.y) + ((double)rd.z + (double)rd.w);
    }
    __syncthreads();
    if (t + 1 < last) fetch(t + 1);
    auto put = [](float (&f)[8], const float4 a, const float4 b) {
      f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    };
    auto row8 = [&](float (&f)[8], const float* r) {
      put(f, *reinterpret_cast<const float4*>(r + 4 * t8), *reinterpret_cast<const float4*>(r + 32 + 4 * t8));
    };
    {  // hidden layer and its gradient
      float h[4][8], x[8];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) h[i][k] = 0.f;
#pragma unroll 8
      for (int c = 0; c < C; ++c) {
        const float4 q = *reinterpret_cast<const float4*>(q1t + c * H + 4 * tj);
        row8(x, vs + c * PX);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          h[0][k] = fmaf(q.x, x[k], h[0][k]);
          h[1][k] = fmaf(q.y, x[k], h[1][k]);
          h[2][k] = fmaf(q.z, x[k], h[2][k]);
          h[3][k] = fmaf(q.w, x[k], h[3][k]);
        }
      }
      row8(x, ds);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        double sc = 0;
        float s2 = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float u = h[i][k] + b1[i];
          s2 = fmaf(gelu_tail(u), x[k], s2);
          h[i][k] = w2[i] * x[k] * gelu_d_tail(u);
          sc += (double)h[i][k];
        }
        gc[i] += sc;
        g2[i] += (double)s2;
        float* r = dh + (4 * tj + i) * PX;
        *reinterpret_cast<float4*>(r + 4 * t8) = make_float4(h[i][0], h[i][1], h[i][2], h[i][3]);
        *reinterpret_cast<float4*>(r + 32 + 4 * t8) = make_float4(h[i][4], h[i][5], h[i][6], h[i][7]);
      }
    }
    __syncthreads();
    {  // input gradient, hidden rows 32 jg .. + 31
      const int jg = tid >> 6, tc = (tid >> 3) & 7;
      float g[4][8], x[8];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) g[i][k] = 0.f;
#pragma unroll 8
      for (int jj = 0; jj < 32; ++jj) {
        const int j = 32 * jg + jj;
        const float4 q = *reinterpret_cast<const float4*>(q1n + j * C + 4 * tc);
        row8(x, dh + j * PX);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          g[0][k] = fmaf(q.x, x[k], g[0][k]);
          g[1][k] = fmaf(q.y, x[k], g[1][k]);
          g[2][k] = fmaf(q.z, x[k], g[2][k]);
          g[3][k] = fmaf(q.w, x[k], g[3][k]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* r = red + (jg * C + 4 * tc + i) * PX;
        *reinterpret_cast<float4*>(r + 4 * t8) = make_float4(g[i][0], g[i][1], g[i][2], g[i][3]);
        *reinterpret_cast<float4*>(r + 32 + 4 * t8) = make_float4(g[i][4], g[i][5], g[i][6], g[i][7]);
      }
    }
    {  // weight gradient
      float w[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) w[i][j] = 0.f;
#pragma unroll 4
      for (int p = 0; p < TX; p += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(vs + (t8 + 8 * j) * PX + p);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 q = *reinterpret_cast<const float4*>(dh + (tj + 32 * i) * PX + p);
#pragma unroll
          for (int j = 0; j < 4; ++j) w[i][j] = fmaf(q.w, b[j].w, fmaf(q.z, b[j].z, fmaf(q.y, b[j].y, fmaf(q.x, b[j].x, w[i][j]))));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) gq[i][j] += (double)w[i][j];
    }
    __syncthreads();
    const long long b = t / per, l = (t - b * per) * TX;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (tid >> 4) + 16 * i, x = 4 * (tid & 15);
      float4 s = *reinterpret_cast<const float4*>(red + c * PX + x);
#pragma unroll
      for (int k = 1; k < 4; ++k) {
        const float4 u = *reinterpret_cast<const float4*>(red + (k * C + c) * PX + x);
        s.x += u.x, s.y += u.y, s.z += u.z, s.w += u.w;
      }
      if (l + x < L) *reinterpret_cast<float4*>(dV + (b * C + c) * L + l + x) = s;
    }
  }
  // the block's sums; gc, g2 over the eight threads that share hidden rows, gd over the loaders
  double* rec = work + (long long)blockIdx.x * REC;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) rec[(tj + 32 * i) * C + t8 + 8 * j] = gq[i][j];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      gc[i] += __shfl_xor_sync(0xffffffffu, gc[i], o);
      g2[i] += __shfl_xor_sync(0xffffffffu, g2[i], o);
    }
    if (t8 == 0) {
      rec[H * C + 4 * tj + i] = gc[i];
      rec[H * C + H + 4 * tj + i] = g2[i];
    }
  }
  if (tid < 32) {
    for (int o = 16; o > 0; o >>= 1) gd += __shfl_xor_sync(0xffffffffu, gd, o);
    if (tid == 0) rec[REC - 1] = gd;
  }
}

__global__ void project_bwd_sum_kernel(int blocks, const double* __restrict__ work, float* gQ1, float* gc1, float* gQ2, float* gc2) {
  using namespace projb;
  const int e = blockIdx.x * 32 + threadIdx.x;
  double s = 0.0;
  if (e < REC)
    for (int z = threadIdx.y; z < blocks; z += 8) s += work[(long long)z * REC + e];
  __shared__ double red[8][33];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || e >= REC) return;
  double t = 0.0;
#pragma unroll
  for (int y = 0; y < 8; ++y) t += red[y][threadIdx.x];
  if (e < H * C) gQ1[e] = (float)t;
  else if (e < H * C + H) gc1[e - H * C] = (float)t;
  else if (e < REC - 1) gQ2[e - H * C - H] = (float)t;
  else gc2[0] = (float)t;
}

static int project_bwd_blocks(long long L, int batch) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long tiles = (L + projb::TX - 1) / projb::TX * batch;
  return (int)(tiles < 2LL * sms ? tiles : 2LL * sms);
}

extern "C" int fw_fno_project_bwd_work(long long L, int batch, long long* doubles_out) {
  if (doubles_out == nullptr || L < 4 || L % 4 != 0 || L > (1LL << 30) || batch < 1 || batch > 65535)
    return fail(FW_EINVAL, "fw_fno_project_bwd_work: bad argument");
  *doubles_out = (long long)project_bwd_blocks(L, batch) * projb::REC;
  return FW_OK;
}

extern "C" int fw_fno_project_bwd(long long L, int batch, const float* V, long long strideV, const float* Q1, const float* c1,
                                  const float* Q2, const float* dout, float* dV, double* work, long long work_doubles,
                                  float* gQ1, float* gc1, float* gQ2, float* gc2, void* stream) {
  long long need = 0;
  if (int rc = fw_fno_project_bwd_work(L, batch, &need)) return rc;
  if (V == nullptr || Q1 == nullptr || c1 == nullptr || Q2 == nullptr || dout == nullptr || dV == nullptr || work == nullptr ||
      gQ1 == nullptr || gc1 == nullptr || gQ2 == nullptr || gc2 == nullptr)
    return fail(FW_EINVAL, "fw_fno_project_bwd: NULL argument");
  if ((((uintptr_t)V | (uintptr_t)dout | (uintptr_t)dV) & 15u) != 0 || strideV % 4 != 0)
    return fail(FW_EINVAL, "fw_fno_project_bwd: activations must start on 16 bytes");
  if (work_doubles < need) return fail(FW_EINVAL, "fw_fno_project_bwd: work buffer too small");
  constexpr size_t smem = (size_t)projb::FLOATS * 4;
  static PerDeviceOnce attr;
  cudaError_t e = set_smem_once(attr, project_bwd_kernel, smem);
  if (e != cudaSuccess) return cuda_fail(e, "fw_fno_project_bwd");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int blocks = project_bwd_blocks(L, batch);
  project_bwd_kernel<<<blocks, 256, smem, st>>>(L, batch, V, strideV, Q1, c1, Q2, dout, dV, work);
  project_bwd_sum_kernel<<<(projb::REC + 31) / 32, dim3(32, 8), 0, st>>>(blocks, work, gQ1, gc1, gQ2, gc2);
  count_launch(2);
  e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_project_bwd");
}

extern "C" int fw_fno_rel_l2(int Bn, long long L, const float* Y, const float* T, float* dY, double* loss,
                             void* stream) {
  rel_l2_kernel<<<Bn, 256, 0, static_cast<cudaStream_t>(stream)>>>(L, Y, T, dY, loss, Bn);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_rel_l2");
}

extern "C" int fw_fno_adam(long long n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                           float eps, int step, float weight_decay, void* stream) {
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  adam_kernel<<<grid1(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, p, g, m, v, lr, b1, b2, eps, bc1, bc2,
                                                                        weight_decay);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_adam");
}

extern "C" int fw_fno_features(int Bn, int NP, int G0, int G1, const float* params, const float* xs, const float* ps,
                               float* out, void* stream) {
  features_kernel<<<grid1((long long)Bn * (NP + 2) * G0 * G1), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      Bn, NP, G0, G1, params, xs, ps, out);
  count_launch(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FW_OK : cuda_fail(e, "fw_fno_features");
}

extern "C" int fw_fno_status(int* status_out, int clear) {
  if (status_out == nullptr) return fail(FW_EINVAL, "fw_fno_status: NULL argument");
  return fno_status_read(status_out, clear);
}
