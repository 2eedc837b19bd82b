// Gaussian start vectors on the GPU (main.cpp:1015-1025): libstdc++'s
// mt19937_64 and normal_distribution, whose draws the reference takes one after
// the other. g++ evaluates Complex(normal(rng), normal(rng)) right to left, so
// an element is (second draw, first draw), and both draws of an element come
// from one accepted pair of the polar method (Marsaglia): the first is y f, the
// second x f. Elements are therefore the accepted pairs in order, and a vector
// is a stream compaction over the generator's outputs.
//
// One CTA per vector: thread t < 156 owns words t and t + 156 of the 312-word
// state (the second needs only the new value of the first), so the state takes
// one barrier per 156 pairs, shared with the compaction of the pairs before
// them. Bound: the chain state -> accepted pairs -> logarithm and square root
// of each 156 pairs, about 1 us. The host drew a vector per thread (small blocks:
// all on one) and copied them over: 5 vectors of 207 k rows 1.7 ms against about
// 10; the small blocks of a 3x3 curve, 2.6 M draws, 103 -> 60 ms for the curve.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ftlm_internal.h"

namespace ftlm {

namespace {

constexpr int kMtWords = 312, kMtPairs = 156;
constexpr int kGaussThreads = 160;  // 5 warps, the last four lanes idle
constexpr int kGaussWarps = kGaussThreads / 32;

__device__ __forceinline__ uint64_t mt_twist(uint64_t up, uint64_t low) {
  const uint64_t y = (up & 0xFFFFFFFF80000000ull) | (low & 0x7FFFFFFFull);
  return (y >> 1) ^ ((y & 1) ? 0xB5026F5AA96619E9ull : 0ull);
}

// generate_canonical<double, 53>, mapped to (-1, 1).
__device__ __forceinline__ double mt_uniform(uint64_t y) {
  y ^= (y >> 29) & 0x5555555555555555ull;
  y ^= (y << 17) & 0x71D67FFFEDA60000ull;
  y ^= (y << 37) & 0xFFF7EEE000000000ull;
  y ^= y >> 43;
  double u = __dmul_rn(__ull2double_rn(y), 0x1p-64);
  if (u >= 1.0) u = 1.0 - 0x1p-53;
  return __dadd_rn(__dmul_rn(2.0, u), -1.0);
}

__global__ void __launch_bounds__(kGaussThreads) k_start_gauss(const GaussJob* __restrict__ jobs,
                                                               double2* __restrict__ out) {
  __shared__ uint64_t mt[2][kMtWords];
  __shared__ int cnt[2][kGaussWarps];
  __shared__ double red[kGaussWarps];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const GaussJob J = jobs[blockIdx.x];
  double2* dst = out + J.off;
  if (tid == 0) {
    uint64_t s = J.seed;
    mt[0][0] = s;
    for (int i = 1; i < kMtWords; ++i) {
      s = 6364136223846793005ull * (s ^ (s >> 62)) + static_cast<uint64_t>(i);
      mt[0][i] = s;
    }
  }
  __syncthreads();
  int64_t base = 0;  // elements before the pending pairs
  double x = 0.0, y = 0.0, r2 = 0.0, n2 = 0.0;
  unsigned int ballot = 0;  // the warp's accepted ones of the pending pairs
  for (int k = 0;; ++k) {
    const uint64_t* o = mt[k & 1];
    uint64_t* w = mt[(k & 1) ^ 1];
    if (tid < kMtPairs) {
      const uint64_t a = o[tid + kMtPairs], n1 = a ^ mt_twist(o[tid], o[tid + 1]);
      const uint64_t nx = tid + 1 < kMtPairs ? o[tid + kMtPairs + 1] : o[kMtPairs] ^ mt_twist(o[0], o[1]);
      w[tid] = n1;
      w[tid + kMtPairs] = n1 ^ mt_twist(a, nx);
    }
    __syncthreads();
    if (k > 0) {  // the pairs of the previous state
      int64_t at = base;
      int all = 0;
#pragma unroll
      for (int v = 0; v < kGaussWarps; ++v) {
        const int c = cnt[(k & 1) ^ 1][v];
        if (v < wid) at += c;
        all += c;
      }
      if ((ballot >> lane) & 1) {
        at += __popc(ballot & ((1u << lane) - 1));
        if (at < J.dim) {
          const double f = sqrt(-2.0 * log(r2) / r2);
          const double re = __dmul_rn(x, f), im = __dmul_rn(y, f);
          dst[at] = make_double2(re, im);
          n2 += re * re + im * im;
        }
      }
      base += all;
      if (base >= J.dim) break;
    }
    bool ok = false;
    if (tid < kMtPairs) {
      x = mt_uniform(w[2 * tid]);
      y = mt_uniform(w[2 * tid + 1]);
      r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
      ok = r2 <= 1.0 && r2 != 0.0;
    }
    ballot = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) cnt[k & 1][wid] = __popc(ballot);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, s);
  if (lane == 0) red[wid] = n2;
  __syncthreads();  // also: every element is written
  double t = 0.0;
  for (int v = 0; v < kGaussWarps; ++v) t += red[v];
  const double nrm = sqrt(t);
  for (int64_t i = tid; i < J.dim; i += kGaussThreads) {
    const double2 z = dst[i];
    dst[i] = make_double2(z.x / nrm, z.y / nrm);
  }
}

}  // namespace

void gaussian_starts(Ctx& c, const std::vector<GaussJob>& jobs, double2* out) {
  if (jobs.empty()) return;
  c.gauss_jobs.ensure(sizeof(GaussJob) * jobs.size());
  FTLM_CUDA(cudaMemcpyAsync(c.gauss_jobs.p, jobs.data(), sizeof(GaussJob) * jobs.size(), cudaMemcpyHostToDevice,
                            c.stream));
  k_start_gauss<<<static_cast<int>(jobs.size()), kGaussThreads, 0, c.stream>>>(c.gauss_jobs.as<GaussJob>(), out);
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
}

}  // namespace ftlm
