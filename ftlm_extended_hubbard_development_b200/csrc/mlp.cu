// Twist-surrogate MLP: FP32 forward, backward and Adam kernels on the GPU.
//
// Network: x[n_in] -> depth hidden layers of `width` units with tanh -> linear
// y[n_out]. Parameters are one flat FP32 buffer, per layer W[out][in] then
// b[out]. Loss: masked mean squared error, sum(mask*(y-t)^2)/sum(mask).
// Every product is summed in index order (no atomics, no split sums), so
// training is deterministic for a given seed, and the two routes below give the
// same bits. A training step runs as two launches where the parameters fit in
// shared memory (k_train_rows, k_train_params), else as one tiled GEMM per
// layer and direction; both stay in FP32.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

#include "ftlm_internal.h"

struct ftlm_mlp {
  int device = 0;
  int n_in = 0, width = 0, depth = 0, n_out = 0;
  cudaStream_t stream = nullptr;
  std::vector<int> fan_in, fan_out;   // per layer
  std::vector<int64_t> w_off, b_off;  // offsets into the flat parameter buffer
  int64_t n_params = 0;
  ftlm::DBuf params, grads, adam_m, adam_v;
  ftlm::DBuf act;      // activations of the current batch, per layer [n][fan_out]
  ftlm::DBuf dact;     // gradients w.r.t. activations
  ftlm::DBuf data_x, data_t, data_m, batch_idx, batch_x, batch_t, batch_m, red, io;
  ftlm::DBuf perm, history;  // training order of one epoch; per-epoch loss sums
  ftlm::DBuf row_sum;        // sum of every training row's mask
  ftlm::Arena arena;
  std::vector<ftlm::DBuf*> bufs() {
    return {&params, &grads, &adam_m, &adam_v, &act, &dact, &data_x, &data_t, &data_m, &batch_idx, &batch_x,
            &batch_t, &batch_m, &red, &io, &perm, &history, &row_sum};
  }
  int64_t data_n = 0;
  int64_t batch_cap = 0;
  int64_t adam_t = 0;
  bool fused_step = true;  // FTLM_TRAIN_STEP=layers: the per-layer kernels at every size
  std::string last_error;
};

namespace ftlm {
namespace {

constexpr int kTile = 32;

// C[m][n] = sum_k A(m,k) B(k,n), A(m,k) = A[m*as + k*ak], B(k,n) = B[k*bs + n*bn].
// mode 0: store; 1: + bias[n], tanh; 2: + bias[n]; 3: multiply by (1 - aux[m][n]^2).
__global__ void k_gemm(int M, int N, int K, const float* __restrict__ A, int64_t as, int64_t ak,
                       const float* __restrict__ B, int64_t bs, int64_t bn, float* __restrict__ C,
                       const float* __restrict__ bias, const float* __restrict__ aux, int mode) {
  __shared__ float As[kTile][kTile + 1];
  __shared__ float Bs[kTile][kTile + 1];
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < K; k0 += kTile) {
    for (int r = ty; r < kTile; r += 8) {
      const int m = m0 + r, k = k0 + tx;
      As[r][tx] = (m < M && k < K) ? A[m * as + k * ak] : 0.f;
      const int kk = k0 + r, n = n0 + tx;
      Bs[r][tx] = (kk < K && n < N) ? B[kk * bs + n * bn] : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kTile; ++k) {
      const float b = Bs[k][tx];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = fmaf(As[ty + 8 * i][k], b, acc[i]);
    }
    __syncthreads();
  }
  const int n = n0 + tx;
  if (n >= N) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty + 8 * i;
    if (m >= M) continue;
    float v = acc[i];
    if (mode == 1) v = tanhf(v + bias[n]);
    else if (mode == 2) v = v + bias[n];
    else if (mode == 3) {
      const float h = aux[static_cast<int64_t>(m) * N + n];
      v = v * (1.f - h * h);
    }
    C[static_cast<int64_t>(m) * N + n] = v;
  }
}

// Column sums db[n] = sum_m dz[m][n] (fixed order).
__global__ void k_colsum(int M, int N, const float* __restrict__ dz, float* __restrict__ db) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float s = 0.f;
  for (int m = 0; m < M; ++m) s += dz[static_cast<int64_t>(m) * N + n];
  db[n] = s;
}

// Output gradient of the masked MSE and per-row loss partials.
__global__ void k_mse(int M, int N, const float* __restrict__ y, const float* __restrict__ t,
                      const float* __restrict__ mask, float inv_count, float* __restrict__ dy,
                      float* __restrict__ row_loss) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  float l = 0.f;
  for (int n = 0; n < N; ++n) {
    const int64_t i = static_cast<int64_t>(m) * N + n;
    const float d = y[i] - t[i];
    dy[i] = 2.f * mask[i] * d * inv_count;
    l += mask[i] * d * d;
  }
  row_loss[m] = l;
}

// out = sum(v) * scale, or out += sum(v) * scale when accumulating.
__global__ void k_sum(int M, const float* __restrict__ v, float* __restrict__ out, float scale, int accumulate) {
  __shared__ double s[256];
  double a = 0.0;
  for (int i = threadIdx.x; i < M; i += 256) a += v[i];
  s[threadIdx.x] = a;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = static_cast<float>(s[0] * scale) + (accumulate ? *out : 0.f);
}

__global__ void k_gather_rows(int M, int W, const int32_t* __restrict__ idx, const float* __restrict__ src,
                              float* __restrict__ dst) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<int64_t>(M) * W) return;
  const int m = static_cast<int>(t / W), w = static_cast<int>(t % W);
  dst[t] = src[static_cast<int64_t>(idx[m]) * W + w];
}

struct Adam {
  float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void adam_update(const Adam& A, float gi, float* __restrict__ p, float* __restrict__ m,
                                            float* __restrict__ v) {
  const float mi = A.b1 * *m + (1.f - A.b1) * gi;
  const float vi = A.b2 * *v + (1.f - A.b2) * gi * gi;
  *m = mi;
  *v = vi;
  *p -= A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
}

__global__ void k_adam(int64_t n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, const __grid_constant__ Adam A) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i < n) adam_update(A, g[i], p + i, m + i, v + i);
}

// ---- a training step in two launches
//
// The layers of a mini-batch are a chain of small products (512 x 128 x 128), so
// a launch per product and direction (21 per step, 11 of them GEMMs on 16-64
// CTAs) took 285 us a step at 32-128-128-128-32 with 512 rows, 0.1% of the FP32
// rate. k_train_rows gives a CTA a few rows of the batch and all parameters in
// shared memory (164 KB), through which its rows go forward and back without
// leaving the SM; k_train_params forms every weight's gradient as one sum over
// the batch and applies Adam to it in registers. Bound now: the chains of
// dependent multiply-adds (K per layer, the batch per weight) and the shared
// loads that feed them: 16 + 15 us a step there; 86 steps with copies and
// allocations 35 -> 5.3 ms.

constexpr int kTrMaxLayers = 17;
constexpr int kTrThreads = 256;
constexpr size_t kTrSmem = 200 * 1024;

struct TrainNet {
  int nl;                     // layers
  int fi[kTrMaxLayers], fo[kTrMaxLayers];
  int ld[kTrMaxLayers];       // row stride of W in shared memory: an odd number of 16-byte units
  int sw[kTrMaxLayers];       // its offset there (floats)
  int64_t w[kTrMaxLayers], b[kTrMaxLayers];  // offsets into the parameters
  int64_t act[kTrMaxLayers];  // offsets of the layer's [n][fo] outputs and their gradients
  int n, lda;                 // batch rows; row stride of the activations in shared memory
  int par_end;                // floats of shared memory the parameters take
};

__device__ __forceinline__ void cp_async4(float* s, const float* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(s))), "l"(g));
}
__device__ __forceinline__ void cp_async16(float* s, const float* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(s))), "l"(g));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
__device__ __forceinline__ void cp_wait(int left) {  // at most `left` groups pending
  switch (left) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
  }
}

// acc[j] = sum_k in[r0 + j step][k] w[k], k ascending.
template <int RP>
__device__ __forceinline__ void tr_forward(const float* in, int lda, int r0, int step, int R, const float* w, int k4,
                                           float (&acc)[RP]) {
  const float4* a[RP];
#pragma unroll
  for (int j = 0; j < RP; ++j) {
    acc[j] = 0.f;
    a[j] = reinterpret_cast<const float4*>(in + min(r0 + j * step, R - 1) * lda);
  }
  const float4* w4 = reinterpret_cast<const float4*>(w);
#pragma unroll 8
  for (int k = 0; k < k4; ++k) {
    const float4 b = w4[k];
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const float4 x = a[j][k];
      acc[j] = fmaf(x.x, b.x, acc[j]);
      acc[j] = fmaf(x.y, b.y, acc[j]);
      acc[j] = fmaf(x.z, b.z, acc[j]);
      acc[j] = fmaf(x.w, b.w, acc[j]);
    }
  }
}

// acc[j] = sum_o dz[r0 + j step][o] W[o][k], o ascending; w = W + k.
template <int RP>
__device__ __forceinline__ void tr_backward(const float* dz, int lda, int r0, int step, int R, const float* w, int ld,
                                            int o4, float (&acc)[RP]) {
  const float4* a[RP];
#pragma unroll
  for (int j = 0; j < RP; ++j) {
    acc[j] = 0.f;
    a[j] = reinterpret_cast<const float4*>(dz + min(r0 + j * step, R - 1) * lda);
  }
#pragma unroll 4
  for (int o = 0; o < o4; ++o) {
    const float b0 = w[0], b1 = w[ld], b2 = w[2 * ld], b3 = w[3 * ld];
    w += 4 * ld;
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const float4 x = a[j][o];
      acc[j] = fmaf(x.x, b0, acc[j]);
      acc[j] = fmaf(x.y, b1, acc[j]);
      acc[j] = fmaf(x.z, b2, acc[j]);
      acc[j] = fmaf(x.w, b3, acc[j]);
    }
  }
}

// Calls f(output, first row, row step) for every (output, row group) of a layer
// of `fo` outputs, RP rows each.
template <int R, typename F>
__device__ __forceinline__ void tr_layer(int fo, F&& f) {
  const int w32 = (fo + 31) / 32 * 32;
  int grp = 1;
  while (grp < R && 2 * grp * w32 <= kTrThreads) grp *= 2;
  for (int t = threadIdx.x; t < grp * w32; t += kTrThreads) {
    const int o = t % w32, g = t / w32;
    if (o < fo) f(o, g, grp);
  }
}

// Forward, loss and backward of R rows of the batch per CTA: gather of the rows,
// activations and pre-activation gradients of every layer to global memory for
// k_train_params. Shared memory: the parameters (rows and columns padded with
// zeros to multiples of 4), two activation buffers per layer.
template <int R>
__global__ void __launch_bounds__(kTrThreads) k_train_rows(const __grid_constant__ TrainNet N,
                                                           const float* __restrict__ par, const int32_t* __restrict__ idx,
                                                           const float* __restrict__ x, const float* __restrict__ t,
                                                           const float* __restrict__ mask, float inv_count,
                                                           float* __restrict__ act, float* __restrict__ dact,
                                                           float* __restrict__ row_loss) {
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lda = N.lda, nl = N.nl;
  const int m0 = blockIdx.x * R, rows = min(R, N.n - m0);
  float* sa = sm + N.par_end;           // layer l's input: sa + l R lda
  float* sd = sa + (nl + 1) * R * lda;  // gradients: two buffers, then targets' terms
  // parameters, one group per layer so that layer 0 starts when its own are in
  for (int l = 0; l < nl; ++l) {
    const int fi = N.fi[l], fo = N.fo[l], ld = N.ld[l], fo4 = (fo + 3) / 4 * 4, fi4 = (fi + 3) / 4 * 4;
    float* w = sm + N.sw[l];
    const float* g = par + N.w[l];
    // a row per 8 lanes; no division by the row length
    const bool wide = fi % 4 == 0 && N.w[l] % 4 == 0;
    for (int o = tid / 8; o < fo; o += kTrThreads / 8) {
      float* d = w + o * ld;
      const float* q = g + static_cast<int64_t>(o) * fi;
      if (wide) {
#pragma unroll 4
        for (int k = 4 * (tid % 8); k < fi; k += 32) cp_async16(d + k, q + k);
      } else {
        for (int k = tid % 8; k < fi; k += 8) cp_async4(d + k, q + k);
        if (fi + tid % 8 < fi4) d[fi + tid % 8] = 0.f;
      }
    }
    for (int i = tid; i < (fo4 - fo) * fi4; i += kTrThreads) w[(fo + i / fi4) * ld + i % fi4] = 0.f;
    cp_commit();
  }
  // the rows' inputs; everything else zero (pads, rows past the batch)
  for (int i = tid; i < (nl + 3) * R * lda; i += kTrThreads) sa[i] = 0.f;
  __syncthreads();
  for (int i = tid; i < rows * N.fi[0]; i += kTrThreads) {
    const int r = i / N.fi[0], k = i - r * N.fi[0];
    sa[r * lda + k] = x[static_cast<int64_t>(idx[m0 + r]) * N.fi[0] + k];
  }
  for (int l = 0; l < nl; ++l) {
    cp_wait(min(3, nl - 1 - l));
    __syncthreads();
    const float* in = sa + l * R * lda;
    float* out = sa + (l + 1) * R * lda;
    const float* w = sm + N.sw[l];
    const int fo = N.fo[l], ld = N.ld[l], k4 = (N.fi[l] + 3) / 4;
    const bool last = l + 1 == nl;
    tr_layer<R>(fo, [&](int o, int g, int grp) {
      const float bias = par[N.b[l] + o];
      auto run = [&](auto rp) {
        constexpr int RP = decltype(rp)::value;
        float acc[RP];
        tr_forward<RP>(in, lda, g, grp, R, w + o * ld, k4, acc);
#pragma unroll
        for (int j = 0; j < RP; ++j) {
          const int r = g + j * grp;
          if (r >= rows) continue;
          const float v = last ? acc[j] + bias : tanhf(acc[j] + bias);
          out[r * lda + o] = v;
          if (!last) act[N.act[l] + static_cast<int64_t>(m0 + r) * fo + o] = v;
        }
      };
      if (R / grp >= 8) run(std::integral_constant<int, (R >= 8 ? 8 : R)>());
      else if (R / grp == 4) run(std::integral_constant<int, (R >= 4 ? 4 : R)>());
      else if (R / grp == 2) run(std::integral_constant<int, (R >= 2 ? 2 : R)>());
      else run(std::integral_constant<int, 1>());
    });
  }
  __syncthreads();
  // masked squared error: gradient of the output, and the rows' loss
  {
    const int fo = N.fo[nl - 1];
    float* y = sa + nl * R * lda;
    float* dz = sd;
    float* md = sd + R * lda;
    for (int i = tid; i < rows * fo; i += kTrThreads) {
      const int r = i / fo, n = i - r * fo;
      const int64_t src = static_cast<int64_t>(idx[m0 + r]) * fo + n;
      const float mk = mask[src], d = y[r * lda + n] - t[src];
      const float dy = 2.f * mk * d * inv_count;
      dz[r * lda + n] = dy;
      dact[N.act[nl - 1] + static_cast<int64_t>(m0 + r) * fo + n] = dy;
      md[r * lda + n] = mk * d;
      y[r * lda + n] = d;
    }
    __syncthreads();
    if (tid < rows) {
      float ls = 0.f;
      for (int n = 0; n < fo; ++n) ls += md[tid * lda + n] * y[tid * lda + n];
      row_loss[m0 + tid] = ls;
    }
    __syncthreads();
  }
  for (int l = nl - 1; l > 0; --l) {
    const float* dz = sd + ((nl - 1 - l) & 1) * R * lda;
    float* dp = sd + ((nl - l) & 1) * R * lda;
    const float* h = sa + l * R * lda;
    const float* w = sm + N.sw[l];
    const int fi = N.fi[l], ld = N.ld[l], o4 = (N.fo[l] + 3) / 4;
    // what an earlier, wider gradient left past this one's end
    for (int i = tid; i < R * 4; i += kTrThreads)
      if (fi + i % 4 < (fi + 3) / 4 * 4) dp[i / 4 * lda + fi + i % 4] = 0.f;
    tr_layer<R>(fi, [&](int k, int g, int grp) {
      auto run = [&](auto rp) {
        constexpr int RP = decltype(rp)::value;
        float acc[RP];
        tr_backward<RP>(dz, lda, g, grp, R, w + k, ld, o4, acc);
#pragma unroll
        for (int j = 0; j < RP; ++j) {
          const int r = g + j * grp;
          if (r >= rows) continue;
          const float hv = h[r * lda + k];
          const float v = acc[j] * (1.f - hv * hv);
          dp[r * lda + k] = v;
          dact[N.act[l - 1] + static_cast<int64_t>(m0 + r) * fi + k] = v;
        }
      };
      if (R / grp >= 8) run(std::integral_constant<int, (R >= 8 ? 8 : R)>());
      else if (R / grp == 4) run(std::integral_constant<int, (R >= 4 ? 4 : R)>());
      else if (R / grp == 2) run(std::integral_constant<int, (R >= 2 ? 2 : R)>());
      else run(std::integral_constant<int, 1>());
    });
    __syncthreads();
  }
}

constexpr int kTpTile = 16;      // outputs x inputs of a CTA
constexpr int kTpThreads = 256;  // one weight per thread
constexpr int kTpRows = 128;     // batch rows per stage
constexpr int kTpStages = 4;

// dW[o][i] = sum_m dz[m][o] in[m][i] and db[o] = sum_m dz[m][o], m ascending, and
// their Adam update; the last CTA adds the batch's loss to `loss`.
__global__ void __launch_bounds__(kTpThreads) k_train_params(const __grid_constant__ TrainNet N,
                                                             const __grid_constant__ Adam A,
                                                             const int32_t* __restrict__ idx,
                                                             const float* __restrict__ x, const float* __restrict__ act,
                                                             const float* __restrict__ dact, float* __restrict__ par,
                                                             float* __restrict__ am, float* __restrict__ av,
                                                             const float* __restrict__ row_loss, float inv_count,
                                                             float* __restrict__ loss) {
  extern __shared__ __align__(16) float sm[];  // [stage][row][16 dz, 16 in]
  const int tid = threadIdx.x;
  if (blockIdx.x + 1 == gridDim.x) {  // as k_sum: 256 strided sums, added by halves
    double* s = reinterpret_cast<double*>(sm);
    for (int k = tid; k < 256; k += kTpThreads) {
      double a = 0.0;
      for (int i = k; i < N.n; i += 256) a += row_loss[i];
      s[k] = a;
    }
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (tid < o) s[tid] += s[tid + o];
      __syncthreads();
    }
    if (tid == 0) *loss = static_cast<float>(s[0] * inv_count) + *loss;
    return;
  }
  int l = 0, tile = blockIdx.x;
  for (;; ++l) {
    const int c = ((N.fo[l] + kTpTile - 1) / kTpTile) * ((N.fi[l] + kTpTile - 1) / kTpTile);
    if (tile < c) break;
    tile -= c;
  }
  const int fi = N.fi[l], fo = N.fo[l], ti = (fi + kTpTile - 1) / kTpTile;
  const int o0 = tile / ti * kTpTile, i0 = tile % ti * kTpTile;
  const float* dz = dact + N.act[l];
  const float* in = l == 0 ? x : act + N.act[l - 1];
  const bool wide = fi % 4 == 0 && fo % 4 == 0 && N.act[l] % 4 == 0 && (l == 0 || N.act[l - 1] % 4 == 0);
  const int nst = (N.n + kTpRows - 1) / kTpRows;
  auto load = [&](int st) {
    if (st < nst) {
      float* s = sm + st % kTpStages * kTpRows * 2 * kTpTile;
      const int m0 = st * kTpRows, nr = min(kTpRows, N.n - m0);
      if (wide) {
#pragma unroll 4
        for (int i = tid; i < nr * 8; i += kTpThreads) {
          const int r = i / 8, q = i % 8, col = (q < 4 ? o0 + 4 * q : i0 + 4 * (q - 4));
          float* d = s + r * 2 * kTpTile + 4 * q;
          if (q < 4) {
            if (col < fo) cp_async16(d, dz + static_cast<int64_t>(m0 + r) * fo + col);
          } else if (col < fi) {
            cp_async16(d, in + static_cast<int64_t>(l == 0 ? idx[m0 + r] : m0 + r) * fi + col);
          }
        }
      } else {
        for (int i = tid; i < nr * 32; i += kTpThreads) {
          const int r = i / 32, q = i % 32, col = (q < 16 ? o0 + q : i0 + q - 16);
          float* d = s + r * 2 * kTpTile + q;
          if (q < 16) {
            if (col < fo) cp_async4(d, dz + static_cast<int64_t>(m0 + r) * fo + col);
          } else if (col < fi) {
            cp_async4(d, in + static_cast<int64_t>(l == 0 ? idx[m0 + r] : m0 + r) * fi + col);
          }
        }
      }
    }
    cp_commit();
  };
  for (int st = 0; st < kTpStages - 1; ++st) load(st);
  const int to = tid / kTpTile, tj = tid % kTpTile;
  float g0 = 0.f, gb = 0.f;
  for (int st = 0; st < nst; ++st) {
    cp_wait(kTpStages - 2);
    __syncthreads();
    load(st + kTpStages - 1);
    const float* s = sm + st % kTpStages * kTpRows * 2 * kTpTile;
    const int nr = min(kTpRows, N.n - st * kTpRows);
    // two warps per scheduler: the loads of 16 rows together, else each waits for its own
    int r = 0;
    for (; r + 16 <= nr; r += 16) {
      float a[16], b[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        a[u] = s[(r + u) * 2 * kTpTile + to];
        b[u] = s[(r + u) * 2 * kTpTile + kTpTile + tj];
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        g0 = fmaf(a[u], b[u], g0);
        gb += a[u];
      }
    }
    for (; r < nr; ++r) {
      const float a = s[r * 2 * kTpTile + to];
      g0 = fmaf(a, s[r * 2 * kTpTile + kTpTile + tj], g0);
      gb += a;
    }
  }
  const int o = o0 + to, i = i0 + tj;
  if (o >= fo) return;
  const int64_t w = N.w[l] + static_cast<int64_t>(o) * fi + i;
  if (i < fi) adam_update(A, g0, par + w, am + w, av + w);
  if (i0 == 0 && tj == 0) adam_update(A, gb, par + N.b[l] + o, am + N.b[l] + o, av + N.b[l] + o);
}

// Sum of every row of the mask, in FP64.
__global__ void k_row_sums(int64_t n, int W, const float* __restrict__ mask, double* __restrict__ out) {
  const int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (r >= n) return;
  double s = 0.0;
  for (int w = 0; w < W; ++w) s += mask[r * W + w];
  out[r] = s;
}

void gemm(ftlm_mlp* net, int M, int N, int K, const float* A, int64_t as, int64_t ak, const float* B, int64_t bs,
          int64_t bn, float* Cc, const float* bias, const float* aux, int mode) {
  dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
  k_gemm<<<grid, dim3(32, 8), 0, net->stream>>>(M, N, K, A, as, ak, B, bs, bn, Cc, bias, aux, mode);
  FTLM_LAUNCH_CHECK();
}

int64_t act_offset(const ftlm_mlp* net, int layer, int64_t n) {
  int64_t o = 0;
  for (int l = 0; l < layer; ++l) o += n * net->fan_out[l];
  return o;
}

void ensure_batch(ftlm_mlp* net, int64_t n) {
  if (n <= net->batch_cap) return;
  int64_t per_row = 0;
  for (int f : net->fan_out) per_row += f;
  net->act.ensure(sizeof(float) * n * per_row);
  net->dact.ensure(sizeof(float) * n * per_row);
  net->batch_x.ensure(sizeof(float) * n * net->n_in);
  net->batch_t.ensure(sizeof(float) * n * net->n_out);
  net->batch_m.ensure(sizeof(float) * n * net->n_out);
  net->batch_idx.ensure(sizeof(int32_t) * n);
  net->red.ensure(sizeof(float) * (n + 8));
  net->batch_cap = n;
}

// Forward of n rows of x (device): activations in net->act; returns output.
float* forward(ftlm_mlp* net, const float* x, int64_t n) {
  ensure_batch(net, n);
  const int L = static_cast<int>(net->fan_in.size());
  const float* in = x;
  float* p = net->params.as<float>();
  for (int l = 0; l < L; ++l) {
    float* out = net->act.as<float>() + act_offset(net, l, n);
    const int fi = net->fan_in[l], fo = net->fan_out[l];
    // out[n][fo] = in[n][fi] * W^T, W[fo][fi]
    gemm(net, static_cast<int>(n), fo, fi, in, fi, 1, p + net->w_off[l], 1, fi, out, p + net->b_off[l], nullptr,
         l + 1 < L ? 1 : 2);
    in = out;
  }
  return net->act.as<float>() + act_offset(net, L - 1, n);
}

// Backward from dy = dL/dy (in net->dact, last layer) into net->grads.
void backward(ftlm_mlp* net, const float* x, int64_t n) {
  const int L = static_cast<int>(net->fan_in.size());
  float* p = net->params.as<float>();
  float* g = net->grads.as<float>();
  for (int l = L - 1; l >= 0; --l) {
    const int fi = net->fan_in[l], fo = net->fan_out[l];
    const float* dz = net->dact.as<float>() + act_offset(net, l, n);  // dL/d(pre-activation) of layer l
    const float* xin = l == 0 ? x : net->act.as<float>() + act_offset(net, l - 1, n);
    // dW[fo][fi] = dz^T xin
    gemm(net, fo, fi, static_cast<int>(n), dz, 1, fo, xin, fi, 1, g + net->w_off[l], nullptr, nullptr, 0);
    k_colsum<<<(fo + 127) / 128, 128, 0, net->stream>>>(static_cast<int>(n), fo, dz, g + net->b_off[l]);
    FTLM_LAUNCH_CHECK();
    if (l > 0) {
      // dz_prev[n][fi] = (dz W) * (1 - h_prev^2)
      float* dprev = net->dact.as<float>() + act_offset(net, l - 1, n);
      gemm(net, static_cast<int>(n), fi, fo, dz, fo, 1, p + net->w_off[l], fi, 1, dprev, nullptr,
           net->act.as<float>() + act_offset(net, l - 1, n), 3);
    }
  }
}

// Rows per CTA of k_train_rows: one wave of CTAs where the batch allows.
int train_rows(int64_t n) { return n <= 148 ? 1 : n <= 296 ? 2 : n <= 592 ? 4 : 8; }

size_t train_smem(const TrainNet& N, int R) {
  return sizeof(float) * (static_cast<size_t>(N.par_end) + static_cast<size_t>(N.nl + 3) * R * N.lda);
}

// The two-launch step for batches of n rows; false when the parameters do not
// fit in shared memory beside the rows.
bool train_net(const ftlm_mlp* net, int64_t n, TrainNet& N) {
  N.nl = static_cast<int>(net->fan_in.size());
  N.n = static_cast<int>(n);
  int64_t at = 0, widest = 0;
  for (int l = 0; l < N.nl; ++l) {
    const int fi = net->fan_in[l], fo = net->fan_out[l];
    if (fi > 4096 || fo > 4096) return false;  // far too wide, and the sums below stay small
    N.fi[l] = fi;
    N.fo[l] = fo;
    N.ld[l] = 4 * ((fi + 3) / 4 | 1);
    N.sw[l] = static_cast<int>(at);
    N.w[l] = net->w_off[l];
    N.b[l] = net->b_off[l];
    N.act[l] = act_offset(net, l, n);
    at += static_cast<int64_t>(N.ld[l]) * ((fo + 3) / 4 * 4);
    widest = std::max<int64_t>(widest, std::max(fi, fo));
    if (at * static_cast<int64_t>(sizeof(float)) > static_cast<int64_t>(kTrSmem)) return false;
  }
  N.par_end = static_cast<int>(at);
  N.lda = static_cast<int>((widest + 3) / 4 * 4);
  return train_smem(N, train_rows(n)) <= kTrSmem;
}

template <int R>
void launch_train_rows(ftlm_mlp* m, const TrainNet& N, const int32_t* idx, float inv_count) {
  const size_t smem = train_smem(N, R);
  smem_limit(k_train_rows<R>, kTrSmem);
  FTLM_CUDA(cudaFuncSetAttribute(k_train_rows<R>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  k_train_rows<R><<<(N.n + R - 1) / R, kTrThreads, smem, m->stream>>>(
      N, m->params.as<float>(), idx, m->data_x.as<float>(), m->data_t.as<float>(), m->data_m.as<float>(), inv_count,
      m->act.as<float>(), m->dact.as<float>(), m->red.as<float>());
  FTLM_LAUNCH_CHECK();  // before the next attribute call, which clears a refused launch's error
}

void train_step(ftlm_mlp* m, const TrainNet& N, const int32_t* idx, float count, const Adam& A, float* loss) {
  switch (train_rows(N.n)) {
    case 1: launch_train_rows<1>(m, N, idx, 1.f / count); break;
    case 2: launch_train_rows<2>(m, N, idx, 1.f / count); break;
    case 4: launch_train_rows<4>(m, N, idx, 1.f / count); break;
    default: launch_train_rows<8>(m, N, idx, 1.f / count); break;
  }
  int tiles = 0;
  for (int l = 0; l < N.nl; ++l)
    tiles += ((N.fo[l] + kTpTile - 1) / kTpTile) * ((N.fi[l] + kTpTile - 1) / kTpTile);
  constexpr size_t smem = sizeof(float) * kTpStages * kTpRows * 2 * kTpTile;
  smem_limit(k_train_params, smem);
  FTLM_CUDA(cudaFuncSetAttribute(k_train_params, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  k_train_params<<<tiles + 1, kTpThreads, smem, m->stream>>>(
      N, A, idx, m->data_x.as<float>(), m->act.as<float>(), m->dact.as<float>(), m->params.as<float>(),
      m->adam_m.as<float>(), m->adam_v.as<float>(), m->red.as<float>(), 1.f / count, loss);
  FTLM_LAUNCH_CHECK();
}

// Loss and gradient on n rows already on the device. The loss (sum over the
// mask / count) is written to `loss_slot` on the device, or added to it when
// `accumulate` is set; nothing waits for the host.
void loss_grad(ftlm_mlp* net, const float* x, const float* t, const float* mask, int64_t n, float count,
               float* loss_slot, int accumulate) {
  float* y = forward(net, x, n);
  const int L = static_cast<int>(net->fan_in.size());
  float* dy = net->dact.as<float>() + act_offset(net, L - 1, n);
  k_mse<<<static_cast<int>((n + 127) / 128), 128, 0, net->stream>>>(static_cast<int>(n), net->n_out, y, t, mask,
                                                                    1.f / count, dy, net->red.as<float>());
  k_sum<<<1, 256, 0, net->stream>>>(static_cast<int>(n), net->red.as<float>(), loss_slot, 1.f / count, accumulate);
  FTLM_LAUNCH_CHECK();
  backward(net, x, n);
}

template <typename F>
int guarded(ftlm_mlp* net, F&& f) {
  if (!net) return FTLM_ERR_ARG;
  try {
    FTLM_CUDA(cudaSetDevice(net->device));
    f(net);
    return FTLM_OK;
  } catch (const Error& e) {
    net->last_error = e.what();
    return e.code;
  } catch (const std::exception& e) {
    net->last_error = e.what();
    return FTLM_ERR_INTERNAL;
  }
}

}  // namespace
}  // namespace ftlm

using ftlm::Error;

extern "C" {

int ftlm_mlp_create(int32_t n_in, int32_t width, int32_t depth, int32_t n_out, uint64_t seed, int32_t device,
                    ftlm_mlp** out) {
  if (!out || n_in <= 0 || width <= 0 || depth <= 0 || n_out <= 0 || depth > 16) return FTLM_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    cudaGetLastError();
    return FTLM_ERR_CUDA;
  }
  ftlm_mlp* net = new (std::nothrow) ftlm_mlp();
  if (!net) return FTLM_ERR_INTERNAL;
  net->device = device;
  net->n_in = n_in;
  net->width = width;
  net->depth = depth;
  net->n_out = n_out;
  if (const char* ts = std::getenv("FTLM_TRAIN_STEP")) net->fused_step = std::string(ts) != "layers";
  for (int l = 0; l <= depth; ++l) {
    net->fan_in.push_back(l == 0 ? n_in : width);
    net->fan_out.push_back(l == depth ? n_out : width);
  }
  int64_t off = 0;
  for (size_t l = 0; l < net->fan_in.size(); ++l) {
    net->w_off.push_back(off);
    off += static_cast<int64_t>(net->fan_in[l]) * net->fan_out[l];
    net->b_off.push_back(off);
    off += net->fan_out[l];
  }
  net->n_params = off;
  // Glorot-uniform weights, zero biases, from a seeded generator
  std::vector<float> h(static_cast<size_t>(off), 0.f);
  std::mt19937_64 rng(seed);
  for (size_t l = 0; l < net->fan_in.size(); ++l) {
    const double a = std::sqrt(6.0 / (net->fan_in[l] + net->fan_out[l]));
    std::uniform_real_distribution<double> u(-a, a);
    for (int64_t i = 0; i < static_cast<int64_t>(net->fan_in[l]) * net->fan_out[l]; ++i)
      h[static_cast<size_t>(net->w_off[l] + i)] = static_cast<float>(u(rng));
  }
  try {
    FTLM_CUDA(cudaSetDevice(device));
    FTLM_CUDA(cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking));
    net->arena.first = size_t(16) << 20;  // a training set and its batches
    for (auto* b : net->bufs()) b->arena = &net->arena;
    net->params.ensure(sizeof(float) * off);
    net->grads.ensure(sizeof(float) * off);
    net->adam_m.ensure(sizeof(float) * off);
    net->adam_v.ensure(sizeof(float) * off);
    FTLM_CUDA(cudaMemcpy(net->params.p, h.data(), sizeof(float) * off, cudaMemcpyHostToDevice));
    FTLM_CUDA(cudaMemset(net->adam_m.p, 0, sizeof(float) * off));
    FTLM_CUDA(cudaMemset(net->adam_v.p, 0, sizeof(float) * off));
  } catch (const Error&) {
    delete net;
    return FTLM_ERR_CUDA;
  }
  *out = net;
  return FTLM_OK;
}

void ftlm_mlp_destroy(ftlm_mlp* net) {
  if (!net) return;
  cudaSetDevice(net->device);
  if (net->stream) cudaStreamSynchronize(net->stream);
  for (auto* x : net->bufs()) x->release();
  net->arena.release();
  if (net->stream) cudaStreamDestroy(net->stream);
  delete net;
}

int ftlm_mlp_last_error(const ftlm_mlp* net, char* buf, size_t len) {
  if (!buf || len == 0) return FTLM_ERR_ARG;
  const std::string msg = net ? net->last_error : std::string("null network");
  const size_t n = std::min(len - 1, msg.size());
  std::memcpy(buf, msg.data(), n);
  buf[n] = '\0';
  return FTLM_OK;
}

int ftlm_mlp_num_params(const ftlm_mlp* net, int64_t* count) {
  if (!net || !count) return FTLM_ERR_ARG;
  *count = net->n_params;
  return FTLM_OK;
}

int ftlm_mlp_get_params(ftlm_mlp* net, float* host, int64_t count) {
  return ftlm::guarded(net, [&](ftlm_mlp* m) {
    if (!host || count != m->n_params) throw Error(FTLM_ERR_ARG, "parameter count mismatch");
    FTLM_CUDA(cudaMemcpy(host, m->params.p, sizeof(float) * count, cudaMemcpyDeviceToHost));
  });
}

int ftlm_mlp_set_params(ftlm_mlp* net, const float* host, int64_t count) {
  return ftlm::guarded(net, [&](ftlm_mlp* m) {
    if (!host || count != m->n_params) throw Error(FTLM_ERR_ARG, "parameter count mismatch");
    FTLM_CUDA(cudaMemcpy(m->params.p, host, sizeof(float) * count, cudaMemcpyHostToDevice));
  });
}

int ftlm_mlp_forward(ftlm_mlp* net, const float* x, int64_t n, float* y) {
  return ftlm::guarded(net, [&](ftlm_mlp* m) {
    if (!x || !y || n <= 0) throw Error(FTLM_ERR_ARG, "bad forward arguments");
    m->io.ensure(sizeof(float) * n * m->n_in);
    FTLM_CUDA(cudaMemcpyAsync(m->io.p, x, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream));
    const float* out = ftlm::forward(m, m->io.as<float>(), n);
    FTLM_CUDA(cudaMemcpyAsync(y, out, sizeof(float) * n * m->n_out, cudaMemcpyDeviceToHost, m->stream));
    FTLM_CUDA(cudaStreamSynchronize(m->stream));
  });
}

int ftlm_mlp_loss_grad(ftlm_mlp* net, const float* x, const float* t, const float* mask, int64_t n, float* loss,
                       float* grad) {
  return ftlm::guarded(net, [&](ftlm_mlp* m) {
    if (!x || !t || !mask || !loss || n <= 0) throw Error(FTLM_ERR_ARG, "bad loss_grad arguments");
    ftlm::ensure_batch(m, n);
    FTLM_CUDA(cudaMemcpyAsync(m->batch_x.p, x, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream));
    FTLM_CUDA(cudaMemcpyAsync(m->batch_t.p, t, sizeof(float) * n * m->n_out, cudaMemcpyHostToDevice, m->stream));
    FTLM_CUDA(cudaMemcpyAsync(m->batch_m.p, mask, sizeof(float) * n * m->n_out, cudaMemcpyHostToDevice, m->stream));
    double cnt = 0.0;
    for (int64_t i = 0; i < n * m->n_out; ++i) cnt += mask[i];
    if (cnt <= 0.0) throw Error(FTLM_ERR_ARG, "empty mask");
    float* slot = m->red.as<float>() + n;
    ftlm::loss_grad(m, m->batch_x.as<float>(), m->batch_t.as<float>(), m->batch_m.as<float>(), n,
                    static_cast<float>(cnt), slot, 0);
    FTLM_CUDA(cudaMemcpyAsync(loss, slot, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    FTLM_CUDA(cudaStreamSynchronize(m->stream));
    if (grad)
      FTLM_CUDA(cudaMemcpy(grad, m->grads.p, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost));
  });
}

int ftlm_mlp_train(ftlm_mlp* net, const float* x, const float* t, const float* mask, int64_t n, int32_t epochs,
                   int32_t batch, float lr, uint64_t seed, float* loss_history) {
  return ftlm::guarded(net, [&](ftlm_mlp* m) {
    if (!x || !t || !mask || n <= 0 || epochs <= 0 || batch <= 0) throw Error(FTLM_ERR_ARG, "bad train arguments");
    m->data_x.ensure(sizeof(float) * n * m->n_in);
    m->data_t.ensure(sizeof(float) * n * m->n_out);
    m->data_m.ensure(sizeof(float) * n * m->n_out);
    FTLM_CUDA(cudaMemcpyAsync(m->data_x.p, x, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream));
    FTLM_CUDA(cudaMemcpyAsync(m->data_t.p, t, sizeof(float) * n * m->n_out, cudaMemcpyHostToDevice, m->stream));
    FTLM_CUDA(cudaMemcpyAsync(m->data_m.p, mask, sizeof(float) * n * m->n_out, cudaMemcpyHostToDevice, m->stream));
    const int64_t B = std::min<int64_t>(batch, n);
    ftlm::ensure_batch(m, B);
    m->perm.ensure(sizeof(int32_t) * n);
    m->history.ensure(sizeof(float) * epochs);
    FTLM_CUDA(cudaMemsetAsync(m->history.p, 0, sizeof(float) * epochs, m->stream));
    // The mask's row sums: a batch's count is the sum of its rows'.
    m->row_sum.ensure(sizeof(double) * n);
    ftlm::k_row_sums<<<static_cast<int>((n + 127) / 128), 128, 0, m->stream>>>(n, m->n_out, m->data_m.as<float>(),
                                                                              m->row_sum.as<double>());
    FTLM_LAUNCH_CHECK();
    std::vector<double> row_sum(static_cast<size_t>(n));
    FTLM_CUDA(cudaMemcpyAsync(row_sum.data(), m->row_sum.p, sizeof(double) * n, cudaMemcpyDeviceToHost, m->stream));
    FTLM_CUDA(cudaStreamSynchronize(m->stream));
    std::vector<int32_t> perm(static_cast<size_t>(n));
    for (int64_t i = 0; i < n; ++i) perm[static_cast<size_t>(i)] = static_cast<int32_t>(i);
    std::mt19937_64 rng(seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    std::vector<int> batches(static_cast<size_t>(epochs), 0);
    ftlm::TrainNet N;
    const bool fused = m->fused_step && ftlm::train_net(m, B, N);
    for (int e = 0; e < epochs; ++e) {
      std::shuffle(perm.begin(), perm.end(), rng);
      FTLM_CUDA(cudaStreamSynchronize(m->stream));  // the previous epoch's order is no longer read
      FTLM_CUDA(cudaMemcpyAsync(m->perm.p, perm.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, m->stream));
      FTLM_CUDA(cudaStreamSynchronize(m->stream));  // before the host shuffles again
      float* slot = m->history.as<float>() + e;
      for (int64_t s = 0; s + B <= n; s += B) {  // full batches only
        double cnt = 0.0;
        for (int64_t i = 0; i < B; ++i) cnt += row_sum[static_cast<size_t>(perm[static_cast<size_t>(s + i)])];
        if (cnt <= 0.0) continue;
        const int32_t* idx = m->perm.as<int32_t>() + s;
        ++batches[static_cast<size_t>(e)];
        ++m->adam_t;
        const ftlm::Adam A{lr, b1, b2, eps, 1.f - std::pow(b1, static_cast<float>(m->adam_t)),
                           1.f - std::pow(b2, static_cast<float>(m->adam_t))};
        if (fused) {
          ftlm::train_step(m, N, idx, static_cast<float>(cnt), A, slot);
          continue;
        }
        const int th = 256;
        ftlm::k_gather_rows<<<static_cast<int>((B * m->n_in + th - 1) / th), th, 0, m->stream>>>(
            static_cast<int>(B), m->n_in, idx, m->data_x.as<float>(), m->batch_x.as<float>());
        ftlm::k_gather_rows<<<static_cast<int>((B * m->n_out + th - 1) / th), th, 0, m->stream>>>(
            static_cast<int>(B), m->n_out, idx, m->data_t.as<float>(), m->batch_t.as<float>());
        ftlm::k_gather_rows<<<static_cast<int>((B * m->n_out + th - 1) / th), th, 0, m->stream>>>(
            static_cast<int>(B), m->n_out, idx, m->data_m.as<float>(), m->batch_m.as<float>());
        FTLM_LAUNCH_CHECK();
        ftlm::loss_grad(m, m->batch_x.as<float>(), m->batch_t.as<float>(), m->batch_m.as<float>(), B,
                        static_cast<float>(cnt), slot, 1);
        ftlm::k_adam<<<static_cast<int>((m->n_params + 255) / 256), 256, 0, m->stream>>>(
            m->n_params, m->params.as<float>(), m->grads.as<float>(), m->adam_m.as<float>(), m->adam_v.as<float>(), A);
        FTLM_LAUNCH_CHECK();
      }
    }
    FTLM_CUDA(cudaStreamSynchronize(m->stream));
    if (loss_history) {
      std::vector<float> h(static_cast<size_t>(epochs));
      FTLM_CUDA(cudaMemcpy(h.data(), m->history.p, sizeof(float) * epochs, cudaMemcpyDeviceToHost));
      for (int e = 0; e < epochs; ++e)
        loss_history[e] = batches[static_cast<size_t>(e)] ? h[static_cast<size_t>(e)] / batches[static_cast<size_t>(e)]
                                                          : 0.f;
    }
  });
}

}  // extern "C"
