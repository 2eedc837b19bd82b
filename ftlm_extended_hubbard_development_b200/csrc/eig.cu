// Exact block spectra on the GPU (diagonalize_block_exact, main.cpp:847-911).
//
// Every block of the list is assembled as a dense column-major Hermitian
// matrix straight from its hop enumeration (pack.cu: the CSR's entries,
// summed in the CSR's order, with no CSR stored), symmetrised as (M + M^H)/2
// like the reference, then all matrices are diagonalised by ONE launch:
// complex Householder reduction to real symmetric tridiagonal form, then every
// eigenvalue independently by Sturm-sequence multisection, four lanes per
// eigenvalue, which yields them sorted ascending. Eigenvalues only (jobz =
// 'N').
//
// The launch is a grid of clusters. The largest matrices are reduced by a whole
// cluster each, the others by one CTA each (eig_plan chooses the cluster size
// and where the line lies); both kinds are taken largest first from counters.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <numeric>

#include "ftlm_internal.h"

namespace ftlm {

namespace {

constexpr int kEigThreads = 512;
constexpr int kEigWarps = kEigThreads / 32;
constexpr int kEigUnroll = 4;
constexpr int kMaxDense = 7000;
constexpr size_t kEigMaxSmem = 200 * 1024;  // three complex work vectors per CTA, else in global memory

// Fixed-order sum over the CTA, the same in every thread. Consecutive calls
// alternate between the two halves of red.
__device__ __forceinline__ double block_sum(double v, double (*red)[kEigWarps], int& flip) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  double* r = red[flip];
  flip ^= 1;
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < kEigWarps; ++w) s += r[w];
  return s;
}

__device__ __forceinline__ double block_minmax(double v, double (*red)[kEigWarps], int& flip, bool is_max) {
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, t) : fmin(v, t);
  }
  double* r = red[flip];
  flip ^= 1;
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = r[0];
  for (int w = 1; w < kEigWarps; ++w) s = is_max ? fmax(s, r[w]) : fmin(s, r[w]);
  return s;
}

// Number of eigenvalues of the tridiagonal (d, e2 = e^2) below x.
__device__ int sturm_count(int n, const double* d, const double* e2, double x, double pivmin) {
  double q = d[0] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  int cnt = q < 0.0;
  for (int i = 1; i < n; ++i) {
    q = d[i] - x - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    cnt += q < 0.0;
  }
  return cnt;
}

__device__ __forceinline__ void group_sync(bool cluster) {
  if (cluster) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

__device__ __forceinline__ double2 ld_cg(const double2* p) { return __ldcg(p); }

// One matrix, by the nr CTAs of a group (a cluster, or one CTA with nr = 1).
// work: d[n], e2[n], then two complex vectors p[2][n] through which the CTAs
// exchange B v; v, w, u: this CTA's own complex work vectors.
//
// Step k reflects column k of the trailing matrix. The rank-2 update of step
// k - 1 is applied while step k's product B v is formed, so the matrix is read
// and written once per step: the update of column k alone gives the next
// reflector u (every CTA computes it, from the same numbers in the same
// order), then each warp takes its columns j, applies - v w^H - w v^H, stores
// them, and adds up (B u)_j = sum_i conj(B_ij) u_i, which needs no other column.
// One barrier per step, after which every CTA forms w from the whole product.
// Columns stay with the same warp throughout. Bound: L2 traffic, 32 bytes per
// trailing element and step, and 4-6 us of barriers and dependent sums per
// step. Against one 256-thread CTA per matrix with B v and the update in
// separate passes: 620 matrices up to 622 rows (4x2 ED curve) 325 -> 27 ms,
// nine of 1764 rows 7625 -> 299 ms, nine of 336 rows 49 -> 3.3 ms.
__device__ void dense_eig(int n, double2* __restrict__ A, double* __restrict__ work, double* __restrict__ ev,
                          double2* v, double2* w, double2* u, int rank, int nr, double (*red)[kEigWarps], int& flip) {
  double* d = work;
  double* e2 = work + n;
  double2* pbuf = reinterpret_cast<double2*>(work + 2 * n);
  const int tid = threadIdx.x, lane = tid & 31;
  const int gwarp = rank * kEigWarps + (tid >> 5), nwarps = nr * kEigWarps;
  const bool cluster = nr > 1;
  for (int i = tid; i < n; i += kEigThreads) v[i] = w[i] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int k = 0; k + 2 < n; ++k) {
    const int m = n - k - 1;
    const double2* col = A + k + static_cast<int64_t>(k) * n;  // A[k][k]
    const double2 v0 = v[0], w0 = w[0];
    // column k with the pending update, its norm
    double s2 = 0.0;
    for (int i = tid; i < m; i += kEigThreads) {
      double2 x = ld_cg(col + 1 + i);
      const double2 vi = v[i + 1], wi = w[i + 1];
      x.x -= (vi.x * w0.x + vi.y * w0.y) + (wi.x * v0.x + wi.y * v0.y);
      x.y -= (vi.y * w0.x - vi.x * w0.y) + (wi.y * v0.x - wi.x * v0.y);
      u[i] = x;
      s2 += x.x * x.x + x.y * x.y;
    }
    const double alpha = sqrt(block_sum(s2, red, flip));
    if (rank == 0 && tid == 0) {
      d[k] = ld_cg(col).x - 2.0 * (v0.x * w0.x + v0.y * w0.y);
      e2[k] = alpha * alpha;
    }
    const double2 x0 = u[0];
    const double ax0 = hypot(x0.x, x0.y);
    const double tau = alpha > 0.0 ? 1.0 / (alpha * (alpha + ax0)) : 0.0;  // 2 / |u|^2; 0: nothing to reflect
    __syncthreads();  // every thread has read u[0]
    if (tid == 0) {
      const double phr = ax0 > 0.0 ? x0.x / ax0 : 1.0;
      const double phi = ax0 > 0.0 ? x0.y / ax0 : 0.0;
      u[0] = make_double2(x0.x + phr * alpha, x0.y + phi * alpha);
    }
    __syncthreads();
    // pending update of the columns behind, and their products with u
    double2* p = pbuf + static_cast<int64_t>(k & 1) * n;
    const int c0 = k + 1;
    int j = c0 / nwarps * nwarps + gwarp;  // this warp's columns: j = gwarp (mod nwarps)
    if (j < c0) j += nwarps;
    for (; j < n; j += nwarps) {
      double2* a = A + c0 + static_cast<int64_t>(j) * n;
      const double2 wj = w[j - c0 + 1], vj = v[j - c0 + 1];
      double2 s = make_double2(0.0, 0.0);
#pragma unroll kEigUnroll
      for (int i = lane; i < m; i += 32) {
        const double2 vi = v[i + 1], wi = w[i + 1], ui = u[i];
        double2 b = a[i];
        b.x -= (vi.x * wj.x + vi.y * wj.y) + (wi.x * vj.x + wi.y * vj.y);
        b.y -= (vi.y * wj.x - vi.x * wj.y) + (wi.y * vj.x - wi.x * vj.y);
        a[i] = b;
        s.x += b.x * ui.x + b.y * ui.y;
        s.y += b.x * ui.y - b.y * ui.x;
      }
      for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      }
      if (lane == 0) __stcg(p + (j - c0), make_double2(tau * s.x, tau * s.y));
    }
    group_sync(cluster);
    // w = p - (tau/2)(u^H p) u; v <- u
    double kr = 0.0;
    for (int i = tid; i < m; i += kEigThreads) {
      const double2 pi = ld_cg(p + i), ui = u[i];
      w[i] = pi;
      kr += ui.x * pi.x + ui.y * pi.y;
    }
    const double K = 0.5 * tau * block_sum(kr, red, flip);
    for (int i = tid; i < m; i += kEigThreads) {
      const double2 ui = u[i];
      w[i] = make_double2(w[i].x - K * ui.x, w[i].y - K * ui.y);
    }
    double2* t = v;
    v = u;
    u = t;
    __syncthreads();
  }
  if (rank == 0 && tid == 0) {  // the last 2x2 (or 1x1) with the pending update
    const double2 v0 = v[0], w0 = w[0];
    if (n >= 2) {
      const double2* c = A + (n - 2) + static_cast<int64_t>(n - 2) * n;
      const double2 v1 = v[1], w1 = w[1];
      const double2 t = ld_cg(c + 1);
      const double tr = t.x - ((v1.x * w0.x + v1.y * w0.y) + (w1.x * v0.x + w1.y * v0.y));
      const double ti = t.y - ((v1.y * w0.x - v1.x * w0.y) + (w1.y * v0.x - w1.x * v0.y));
      d[n - 2] = ld_cg(c).x - 2.0 * (v0.x * w0.x + v0.y * w0.y);
      d[n - 1] = ld_cg(c + n + 1).x - 2.0 * (v1.x * w1.x + v1.y * w1.y);
      e2[n - 2] = tr * tr + ti * ti;
    } else {
      d[0] = ld_cg(A).x;
    }
    e2[n - 1] = 0.0;
  }
  group_sync(cluster);
  // tridiagonal matrix beside the CTA: d in v, e2 in w (as doubles)
  double* ds = reinterpret_cast<double*>(v);
  double* es = reinterpret_cast<double*>(w);
  for (int i = tid; i < n; i += kEigThreads) {
    ds[i] = __ldcg(d + i);
    es[i] = __ldcg(e2 + i);
  }
  __syncthreads();
  // Gershgorin interval and multisection
  double lo = DBL_MAX, hi = -DBL_MAX, emax = 0.0;
  for (int i = tid; i < n; i += kEigThreads) {
    const double el = i > 0 ? sqrt(es[i - 1]) : 0.0;
    const double er = i + 1 < n ? sqrt(es[i]) : 0.0;
    lo = fmin(lo, ds[i] - el - er);
    hi = fmax(hi, ds[i] + el + er);
    emax = fmax(emax, es[i]);
  }
  lo = block_minmax(lo, red, flip, false);
  hi = block_minmax(hi, red, flip, true);
  emax = block_minmax(emax, red, flip, true);
  const double pivmin = DBL_MIN * fmax(1.0, emax);
  const double span = fmax(fabs(lo), fabs(hi));
  lo -= 4.0 * DBL_EPSILON * span + pivmin;
  hi += 4.0 * DBL_EPSILON * span + pivmin;
  // four lanes per eigenvalue j count at the inner points of a fifth each: the
  // j-th eigenvalue lies below the first point with more than j below it
  const int sub = lane & 3;
  const int quads = nr * kEigThreads / 4;
  for (int j0 = 0; j0 < n; j0 += quads) {
    const int j = j0 + (rank * kEigThreads + tid) / 4;
    const bool real = j < n;
    double a = lo, b = hi;
    bool run = real;
    for (int it = 0; it < 64; ++it) {
      run = run && b - a > 2.0 * DBL_EPSILON * fmax(fabs(a), fabs(b));
      const double x = a + (b - a) * (0.2 * (sub + 1));
      const bool inside = x > a && x < b;
      int above = 0;
      if (run && inside) above = sturm_count(n, ds, es, x, pivmin) > j;
      const unsigned ok = __ballot_sync(0xffffffffu, inside) >> (lane & ~3) & 15u;
      const unsigned m = __ballot_sync(0xffffffffu, above) >> (lane & ~3) & 15u;
      if (run && ok != 15u) {
        // the interval no longer holds four inner points: finish by halves
        const double mid = 0.5 * (a + b);
        if (mid <= a || mid >= b) run = false;
        else if (sturm_count(n, ds, es, mid, pivmin) > j) b = mid;
        else a = mid;
      } else if (run) {
        const int f = m ? __ffs(m) - 1 : 4;  // counts grow with x: first point with more than j below
        const double w5 = b - a;
        const double na = f > 0 ? a + w5 * (0.2 * f) : a;
        if (f < 4) b = a + w5 * (0.2 * (f + 1));
        a = na;
      }
      if (!__any_sync(0xffffffffu, run)) break;
    }
    if (real && sub == 0) ev[j] = 0.5 * (a + b);
  }
  group_sync(cluster);  // the work vectors are free for the next matrix
}

struct EigArgs {
  int nmat, nlarge;        // matrices, those taken by clusters (the first of `order`)
  const int32_t* order;    // largest first
  const int32_t* dims;
  const int64_t* aoff;
  const int64_t* eoff;
  const int64_t* woff;
  double2* arena;
  double* evout;
  double* work;
  double2* vecs;           // per CTA three vectors of nmax, null: shared memory
  int64_t nmax;
  int* counters;           // [2], zeroed: next large, next small matrix
  int* slots;              // [clusters][2]
  int cluster;             // CTAs per cluster
};

__global__ void __launch_bounds__(kEigThreads) k_dense_eig(const __grid_constant__ EigArgs P) {
  extern __shared__ double2 sh[];
  __shared__ double red[2][kEigWarps];
  __shared__ int s_next;
  int flip = 0;
  const int rank = blockIdx.x % P.cluster, tid = threadIdx.x;
  double2* v = P.vecs ? P.vecs + static_cast<int64_t>(blockIdx.x) * 3 * P.nmax : sh;
  double2* w = v + P.nmax;
  double2* u = w + P.nmax;
  // matrices of whole clusters: rank 0 takes the next one for all
  int* slot = P.slots + 2 * (blockIdx.x / P.cluster);
  for (int it = 0; P.nlarge > 0; ++it) {
    if (rank == 0 && tid == 0) __stcg(slot + (it & 1), atomicAdd(P.counters, 1));
    group_sync(true);
    const int t = __ldcg(slot + (it & 1));
    if (t >= P.nlarge) break;
    const int mi = P.order[t];
    dense_eig(P.dims[mi], P.arena + P.aoff[mi], P.work + P.woff[mi], P.evout + P.eoff[mi], v, w, u, rank, P.cluster,
              red, flip);
  }
  // the rest, one CTA each
  while (true) {
    __syncthreads();
    if (tid == 0) s_next = P.nlarge + atomicAdd(P.counters + 1, 1);
    __syncthreads();
    const int t = s_next;
    if (t >= P.nmat) break;
    const int mi = P.order[t];
    dense_eig(P.dims[mi], P.arena + P.aoff[mi], P.work + P.woff[mi], P.evout + P.eoff[mi], v, w, u, 0, 1, red, flip);
  }
}

constexpr int64_t kWorkPerRow = 6;  // doubles of dense_eig work space per row: d, e2, p[2] complex

struct DenseItem {
  int mx, my;
  int64_t n, aoff, woff;
};

// Dimensions of the listed blocks (empty ones dropped); aoff/woff relative.
std::vector<DenseItem> dense_items(Ctx& c, const std::vector<std::pair<int, int>>& blocks, int64_t& asz,
                                   int64_t& wsz) {
  std::vector<DenseItem> items;
  asz = wsz = 0;
  for (const auto& b : blocks) {
    const int64_t n = c.block_dims.at(static_cast<size_t>(b.second * c.geom.lx + b.first));
    if (n <= 0) continue;
    if (n > kMaxDense) throw Error(FTLM_ERR_CAPACITY, "block too large for the dense exact solver: " + std::to_string(n));
    items.push_back({b.first, b.second, n, asz, wsz});
    asz += n * n;
    wsz += kWorkPerRow * n;
  }
  return items;
}

// Dense Hermitian matrix of every item at arena + aoff (zeroed by the caller).
void dense_fill(Ctx& c, const std::vector<DenseItem>& items, double2* arena, int64_t abase) {
  std::vector<PackItem> rows;
  for (const DenseItem& it : items) {
    PackItem p{};
    p.mx = it.mx;
    p.my = it.my;
    p.n = it.n;
    p.off = abase + it.aoff;
    rows.push_back(p);
  }
  pack_dense(c, rows, arena);
}

struct EigPlan {
  int cluster, nlarge;
};

// Cluster size and number of matrices (the first of `order`) given to whole
// clusters: those with the smallest modelled time. A column costs a CTA 4 us
// of dependent sums, a cluster 6 us, and n^2 / cluster * 2.5e-4 us of memory
// traffic (fitted to 336-row matrices: 20, 13 and 10 us a column on 2, 4 and 8
// CTAs). One cluster size does not fit all: the exact blocks of a 4x2 curve up
// to 256 rows take 4.4 ms on clusters of 2 and 10.9 on 8, nine matrices of
// 1764 rows 986 ms on 2 and 299 on 8, the whole 4x2 ED curve 44, 30 and 39 ms
// on 2, 4 and 8.
EigPlan eig_plan(const std::vector<int32_t>& dims, const std::vector<int32_t>& order, int sms) {
  auto cost = [](double n, int cs) { return n * ((cs > 1 ? 6.0 : 4.0) + n * n * 2.5e-4 / cs); };
  std::vector<double> single(order.size() + 1, 0.0);  // [i]: the matrices from i on, one CTA each
  for (size_t i = order.size(); i-- > 0;) single[i] = single[i + 1] + cost(dims[order[i]], 1);
  auto phase = [](double sum, int slots, double most) { return std::max(sum / slots, most); };
  EigPlan best{1, 0};
  double t = phase(single[0], sms, cost(dims[order[0]], 1));
  for (int cs = 2; cs <= 8; cs *= 2) {
    double sum = 0.0;
    for (size_t i = 0; i < order.size(); ++i) {
      sum += cost(dims[order[i]], cs);
      const bool rest = i + 1 < order.size();
      const double tt = phase(sum, sms / cs, cost(dims[order[0]], cs)) +
                        (rest ? phase(single[i + 1], sms, cost(dims[order[i + 1]], 1)) : 0.0);
      if (tt < t) {
        t = tt;
        best = {cs, static_cast<int>(i + 1)};
      }
    }
  }
  return best;
}

// One k_dense_eig launch over matrices (dims, aoff into arena) writing the
// eigenvalues at evout + eoff; work: kWorkPerRow doubles per row.
void dense_solve(Ctx& c, const std::vector<int32_t>& dims, const std::vector<int64_t>& aoff,
                 const std::vector<int64_t>& eoff, double2* arena, double* evout, double* work) {
  const size_t nb = dims.size();
  if (nb == 0) return;
  std::vector<int32_t> order(nb);
  std::vector<int64_t> woff(nb);
  int64_t nmax = 0, wtot = 0;
  EigArgs P{};
  for (size_t i = 0; i < nb; ++i) {
    woff[i] = wtot;
    wtot += kWorkPerRow * static_cast<int64_t>(dims[i]);
    nmax = std::max<int64_t>(nmax, dims[i]);
  }
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return dims[a] > dims[b]; });
  const EigPlan plan = eig_plan(dims, order, c.sm_count);
  P.cluster = plan.cluster;
  P.nlarge = plan.nlarge;
  // clusters: enough for the large matrices or one small one per CTA, at most one CTA per SM
  const int want = std::max<int>(P.nlarge, static_cast<int>((nb - P.nlarge + P.cluster - 1) / P.cluster));
  const int clusters = std::max(1, std::min(want, c.sm_count / P.cluster));
  const size_t i32bytes = ((sizeof(int32_t) * (2 * nb + 2 + 2 * clusters) + 7) / 8) * 8;  // int64 arrays stay aligned
  c.dense_meta.ensure(i32bytes + sizeof(int64_t) * 3 * nb);
  int32_t* d_ctr = c.dense_meta.as<int32_t>();
  int32_t* d_order = d_ctr + 2 + 2 * clusters;
  int32_t* d_dims = d_order + nb;
  int64_t* d_aoff = reinterpret_cast<int64_t*>(c.dense_meta.as<char>() + i32bytes);
  int64_t* d_eoff = d_aoff + nb;
  int64_t* d_woff = d_eoff + nb;
  FTLM_CUDA(cudaMemsetAsync(d_ctr, 0, sizeof(int32_t) * (2 + 2 * clusters), c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_order, order.data(), sizeof(int32_t) * nb, cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_dims, dims.data(), sizeof(int32_t) * nb, cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_aoff, aoff.data(), sizeof(int64_t) * nb, cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_eoff, eoff.data(), sizeof(int64_t) * nb, cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_woff, woff.data(), sizeof(int64_t) * nb, cudaMemcpyHostToDevice, c.stream));
  c.prof.h2d_bytes += static_cast<int64_t>(nb) * 32;
  P.nmat = static_cast<int>(nb);
  P.order = d_order;
  P.dims = d_dims;
  P.aoff = d_aoff;
  P.eoff = d_eoff;
  P.woff = d_woff;
  P.arena = arena;
  P.evout = evout;
  P.work = work;
  P.nmax = std::max<int64_t>(nmax, 2);  // the reduction reads v[0], v[1] of any matrix
  P.counters = d_ctr;
  P.slots = d_ctr + 2;
  size_t smem = sizeof(double2) * 3 * static_cast<size_t>(P.nmax);
  if (smem > kEigMaxSmem) {
    c.dense_vecs.ensure(smem * clusters * P.cluster);
    P.vecs = c.dense_vecs.as<double2>();
    smem = 0;
  }
  smem_limit(k_dense_eig, kEigMaxSmem);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * P.cluster);
  cfg.blockDim = dim3(kEigThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = P.cluster;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  FTLM_CUDA(cudaLaunchKernelEx(&cfg, k_dense_eig, P));
  c.prof.kernel_launches += 1;
}

struct EventTimer {
  Ctx& c;
  double& acc;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  EventTimer(Ctx& c_, double& acc_) : c(c_), acc(acc_) {
    if (!c.timing) return;
    FTLM_CUDA(cudaEventCreate(&e0));
    FTLM_CUDA(cudaEventCreate(&e1));
    FTLM_CUDA(cudaEventRecord(e0, c.stream));
  }
  void stop() {
    if (!e0) return;
    FTLM_CUDA(cudaEventRecord(e1, c.stream));
    FTLM_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    FTLM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    acc += ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    e0 = e1 = nullptr;
  }
  ~EventTimer() {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  }
};

Spectrum exact_spectrum(const Ctx& c, int64_t n, int64_t ev_off) {
  Spectrum s;
  s.ev_off = ev_off;
  s.w_off = -1;
  s.count = n;
  s.exact = true;
  s.prefactor = 1.0;
  s.particles = c.sec.n_up + c.sec.n_dn;
  s.dim = n;
  return s;
}

}  // namespace

void run_exact_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks) {
  int64_t asz = 0, wsz = 0;
  const std::vector<DenseItem> items = dense_items(c, blocks, asz, wsz);
  if (items.empty()) return;
  c.dense_arena.ensure(sizeof(double2) * asz);
  c.dense_out.ensure(sizeof(double) * wsz);
  FTLM_CUDA(cudaMemsetAsync(c.dense_arena.p, 0, sizeof(double2) * asz, c.stream));
  std::vector<int32_t> dims;
  std::vector<int64_t> aoff, eoff;
  for (const DenseItem& it : items) {
    dims.push_back(static_cast<int32_t>(it.n));
    aoff.push_back(it.aoff);
    eoff.push_back(spectra_alloc(c, it.n));
  }
  {
    EventTimer t(c, c.prof.dense_ms);
    dense_fill(c, items, c.dense_arena.as<double2>(), 0);
    t.stop();
  }
  {
    EventTimer t(c, c.prof.eig_ms);
    dense_solve(c, dims, aoff, eoff, c.dense_arena.as<double2>(), c.spectra.as<double>(), c.dense_out.as<double>());
    t.stop();
  }
  FTLM_CUDA(cudaStreamSynchronize(c.stream));
  for (size_t i = 0; i < items.size(); ++i) c.spec[{items[i].mx, items[i].my}] = exact_spectrum(c, items[i].n, eoff[i]);
}

void queue_exact_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks) {
  int64_t asz = 0, wsz = 0;
  std::vector<DenseItem> items = dense_items(c, blocks, asz, wsz);
  if (items.empty()) return;
  if (defer_pool_bytes(c) > 0 && defer_pool_bytes(c) + static_cast<int64_t>(sizeof(double2)) * asz > kDeferPoolBytes)
    flush_deferred(c);
  const int64_t base = c.defer_asz;
  c.defer_arena.ensure_keep(sizeof(double2) * (base + asz), c.stream);
  FTLM_CUDA(cudaMemsetAsync(c.defer_arena.as<double2>() + base, 0, sizeof(double2) * asz, c.stream));
  {
    EventTimer t(c, c.prof.dense_ms);
    dense_fill(c, items, c.defer_arena.as<double2>(), base);
    t.stop();
  }
  c.defer_asz = base + asz;
  for (const DenseItem& it : items) {
    Spectrum s = exact_spectrum(c, it.n, -1);
    s.pending = static_cast<int>(c.defer_items.size());
    c.spec[{it.mx, it.my}] = s;
    c.defer_items.push_back({c.sec.n_up, c.sec.n_dn, it.mx, it.my, it.n, base + it.aoff, c.sec_gen});
  }
}

int64_t defer_pool_bytes(const Ctx& c) {
  return static_cast<int64_t>(sizeof(double2)) * (c.defer_asz + c.sb_start_used) +
         static_cast<int64_t>(sizeof(uint32_t)) * c.sb_ent_used +
         static_cast<int64_t>(sizeof(int32_t) + sizeof(double)) * c.sb_row_used +
         static_cast<int64_t>(2 * sizeof(double)) * c.sb_ab_used;
}

void flush_deferred(Ctx& c) {
  const size_t nb = c.defer_items.size();
  const size_t nr = c.defer_small.size();
  if (nb == 0 && nr == 0) {
    c.defer_acc.clear();
    return;
  }
  // exact blocks: one dense solve
  std::vector<int64_t> eoff(nb);
  if (nb > 0) {
    std::vector<int32_t> dims(nb);
    std::vector<int64_t> aoff(nb);
    int64_t etot = 0;
    for (size_t i = 0; i < nb; ++i) {
      dims[i] = static_cast<int32_t>(c.defer_items[i].n);
      aoff[i] = c.defer_items[i].aoff;
      eoff[i] = etot;
      etot += c.defer_items[i].n;
    }
    c.defer_ev.ensure(sizeof(double) * etot);
    c.defer_work.ensure(sizeof(double) * kWorkPerRow * etot);
    EventTimer t(c, c.prof.eig_ms);
    dense_solve(c, dims, aoff, eoff, c.defer_arena.as<double2>(), c.defer_ev.as<double>(), c.defer_work.as<double>());
    t.stop();
  }
  // small FTLM blocks: their Lanczos is running; one Ritz-stage launch; the spectra land
  // in this sector's arena (those of earlier sectors are dropped with it later)
  std::vector<Spectrum> rs(nr);
  if (nr > 0) {
    small_join(c);
    std::vector<RitzJob> jobs;
    for (size_t i = 0; i < nr; ++i) jobs.push_back(small_ritz_job(c, c.defer_small[i].d, &rs[i]));
    ritz_stage_many(c, jobs);
    for (size_t i = 0; i < nr; ++i) {
      rs[i].prefactor = static_cast<double>(c.defer_small[i].d.dim);
      rs[i].particles = c.defer_small[i].n_up + c.defer_small[i].n_dn;
      rs[i].dim = c.defer_small[i].d.dim;
    }
  }
  for (const DeferAcc& a : c.defer_acc) {
    const size_t i = static_cast<size_t>(a.idx);
    if (a.small) {
      thermo_accumulate(c, rs[i]);
    } else {
      const DeferItem& d = c.defer_items[i];
      thermo_accumulate_dev(c, c.defer_ev.as<double>() + eoff[i], nullptr, d.n, 1.0, d.n_up + d.n_dn);
    }
  }
  // pending spectra of the current sector become ordinary ones
  for (size_t i = 0; i < nb; ++i) {
    const DeferItem& d = c.defer_items[i];
    if (d.sec_gen != c.sec_gen) continue;
    auto it = c.spec.find({d.mx, d.my});
    if (it == c.spec.end() || it->second.pending != static_cast<int>(i)) continue;
    const int64_t off = spectra_alloc(c, d.n);
    FTLM_CUDA(cudaMemcpyAsync(c.spectra.as<double>() + off, c.defer_ev.as<double>() + eoff[i], sizeof(double) * d.n,
                              cudaMemcpyDeviceToDevice, c.stream));
    it->second.ev_off = off;
    it->second.pending = -1;
  }
  for (size_t i = 0; i < nr; ++i) {
    const DeferSmall& d = c.defer_small[i];
    if (d.sec_gen != c.sec_gen) continue;
    auto it = c.spec.find({d.mx, d.my});
    if (it == c.spec.end() || it->second.pending_small != static_cast<int>(i)) continue;
    it->second = rs[i];
  }
  c.defer_items.clear();
  c.defer_small.clear();
  small_rows_reset(c);
  c.defer_acc.clear();
  c.defer_asz = 0;
}

}  // namespace ftlm
