// Small FTLM blocks (run_ftlm_block, main.cpp:996-1113, for every block of a
// sector up to kSmallMaxDim rows).
//
// A block of a few thousand rows gives one H*V far too little work to fill
// the GPU, so stepping it with the sweep kernels spends its time in launch
// latency (four launches per Lanczos step). Here one CTA runs the whole
// Lanczos recurrence of one (block, random vector) pair: the two working
// vectors live in shared memory, H's rows are 4-byte entries read from L2
// (column, direction, sign, shift, orbit-size ratio; the coefficient is a
// table entry times a ratio), and alpha/beta go to the same [K][ld] layout the
// sweep path writes, so the Ritz stage (k_tridiag) and everything after it are
// shared. With pooled spectra a sector's launches go to a side stream, so the
// small blocks of several sectors run beside each other and beside the table
// builds of the next ones.
//
// A thread owns whole rows (i, i + threads, ...): entry k of consecutive rows
// is consecutive in memory, H v stays in registers until alpha is known, and
// the next vector overwrites the previous one in place, so a step has three
// barriers. Size classes pick the threads: 256 up to 512 rows, 512 up to 1024,
// 1024 above, one launch each, so a small block does not wait behind the
// shared memory and barriers of a large one. Bound: reads of x and of the
// coefficients in shared memory (32 bytes per FP64 hop). 3x3 curve, 5 FP64
// vectors x 80 steps, 288 blocks up to 1764 rows: 82 ms in 32 launches of 256
// threads on 20-byte CSR entries, one after another (45 of 148 SMs busy),
// against 27 ms of launches that overlap; 4x2 curve, 32 mixed vectors x 120
// steps: 24 ms against 8.2. With the fours the 3x3 curve's launches take 25 ms: the two
// halves of a chain no longer wait for each other.
//
// Arithmetic is the reference's: w = H v; alpha = Re<v, w>;
// w -= alpha v + beta_prev v_prev; beta = |w|; stop at beta < 1e-12 or the
// last step; v_next = w / beta. Sums are FP64 in a fixed order
// (deterministic). In mixed precision the vectors are stored as FP32 complex
// (each element rounded once per step) and every sum stays FP64.
#include <algorithm>
#include <cmath>
#include <numeric>

#include "ftlm_internal.h"

namespace ftlm {

namespace {

template <typename T>
struct CT;
template <>
struct CT<double> {
  using C = double2;
  __device__ static C make(double re, double im) { return make_double2(re, im); }
};
template <>
struct CT<float> {
  using C = float2;
  __device__ static C make(double re, double im) {
    return make_float2(static_cast<float>(re), static_cast<float>(im));
  }
};

// Fixed-order CTA sum of one double per thread, the same in every thread; red
// must not be the one of the previous call (one barrier per call).
template <int NW>
__device__ __forceinline__ double cta_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = (threadIdx.x & 31) < NW ? red[threadIdx.x & 31] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

struct SmallArgs {
  int ntasks, cap, nsite;
  const int2* tasks;  // (block, vector)
  const SmallBlockDesc* blocks;
  const uint32_t* ent;
  const int32_t* cnt;
  const double* diag;
  const double* phase;  // [n_k][64] complex
  const double2* start;
  double* alpha;
  double* beta;
  int32_t* steps;
  double amp_re[8], amp_im[8];
  double sqrt_deg[65];
  SmallRatios ratios;
};

template <typename T, int NT, int RPT>
__global__ void __launch_bounds__(NT) k_lanczos_small(const __grid_constant__ SmallArgs A) {
  using C = typename CT<T>::C;
  constexpr int NW = NT / 32;
  // An FP64 row's hops are added four at a time, the fours then to the row: the sums that
  // round are as short as those of 8 lanes sharing a row. FP32 rows are added in FP64 too and
  // rounded to FP32 at the end, where one chain does as well.
  constexpr bool kFours = sizeof(T) == 8;
  extern __shared__ __align__(16) unsigned char small_smem[];
  __shared__ double red[2][32];
  __shared__ double s_ratio[kSmallRatios];
  double2* coef = reinterpret_cast<double2*>(small_smem);  // [shift][dir * 2 + parity]
  C* b0 = reinterpret_cast<C*>(coef + A.nsite * 16);
  const int tid = threadIdx.x;
  for (int i = tid; i < A.ratios.n; i += NT)
    s_ratio[i] = __ddiv_rn(A.sqrt_deg[A.ratios.num[i]], A.sqrt_deg[A.ratios.den[i]]);
  for (int t = blockIdx.x; t < A.ntasks; t += gridDim.x) {
    const int2 task = A.tasks[t];
    const SmallBlockDesc B = A.blocks[task.x];
    const int r = task.y, D = B.dim;
    C* v = b0;
    C* vp = b0 + A.cap;
    __syncthreads();  // the previous task's vectors and table are no longer read
    for (int i = tid; i < A.nsite * 16; i += NT) {
      // (amp * sign) * phase, the operation order of main.cpp:794-797
      const int dir = (i >> 1) & 7;
      const double ar = i & 1 ? -A.amp_re[dir] : A.amp_re[dir];
      const double ai = i & 1 ? -A.amp_im[dir] : A.amp_im[dir];
      const double pr = A.phase[128 * B.k + 2 * (i >> 4)], pi = A.phase[128 * B.k + 2 * (i >> 4) + 1];
      coef[i] = make_double2(__dsub_rn(__dmul_rn(ar, pr), __dmul_rn(ai, pi)),
                             __dadd_rn(__dmul_rn(ar, pi), __dmul_rn(ai, pr)));
    }
    const double amp = 1.0 / sqrt(static_cast<double>(D));
    int len[RPT];
    double dg[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int i = tid + q * NT;
      len[q] = 0;
      dg[q] = 0.0;
      if (i >= D) continue;
      len[q] = A.cnt[B.row_off + i];
      dg[q] = A.diag[B.row_off + i];
      double re, im;
      if (B.start_off >= 0) {
        const double2 z = A.start[B.start_off + static_cast<int64_t>(r) * D + i];
        re = z.x;
        im = z.y;
      } else {
        philox_phase(i, r, B.seed, amp, re, im);
      }
      v[i] = CT<T>::make(re, im);
      vp[i] = CT<T>::make(0.0, 0.0);
    }
    __syncthreads();
    double beta_prev = 0.0;
    int steps = B.K;
    for (int j = 0; j < B.K; ++j) {
      // h = H v; partial Re<v, h>
      C h[RPT];
      double ap = 0.0;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int i = tid + q * NT;
        if (i >= D) continue;
        const uint32_t* e = A.ent + B.ent_off + i;
        const C xi = v[i];
        double ar = 0.0, ai = 0.0;
        int n = len[q];
        auto add = [&](uint32_t w, double& sr, double& si) {
          const double2 c = coef[(w >> 12) & 0x3FF];
          const double ratio = s_ratio[w >> 22];
          const C x = v[w & 0xFFF];
          const double cr = __dmul_rn(c.x, ratio), ci = __dmul_rn(c.y, ratio);
          sr += cr * static_cast<double>(x.x) - ci * static_cast<double>(x.y);
          si += cr * static_cast<double>(x.y) + ci * static_cast<double>(x.x);
        };
        for (; n >= 4; n -= 4, e += 4 * static_cast<int64_t>(D)) {
          const uint32_t w0 = __ldg(e), w1 = __ldg(e + D), w2 = __ldg(e + 2 * D), w3 = __ldg(e + 3 * D);
          double sr = 0.0, si = 0.0;
          double& r4 = kFours ? sr : ar;
          double& i4 = kFours ? si : ai;
          add(w0, r4, i4);
          add(w1, r4, i4);
          add(w2, r4, i4);
          add(w3, r4, i4);
          if constexpr (kFours) {
            ar += sr;
            ai += si;
          }
        }
        for (; n > 0; --n, e += D) add(__ldg(e), ar, ai);
        ar += dg[q] * static_cast<double>(xi.x);
        ai += dg[q] * static_cast<double>(xi.y);
        h[q] = CT<T>::make(ar, ai);
        ap += static_cast<double>(xi.x) * static_cast<double>(h[q].x) +
              static_cast<double>(xi.y) * static_cast<double>(h[q].y);
      }
      const double alpha = cta_sum<NW>(ap, red[0]);
      // h -= alpha v + beta_prev vp; partial |h|^2
      double np = 0.0;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int i = tid + q * NT;
        if (i >= D) continue;
        const C xi = v[i], pi = vp[i];
        h[q] = CT<T>::make(static_cast<double>(h[q].x) - alpha * static_cast<double>(xi.x) -
                               beta_prev * static_cast<double>(pi.x),
                           static_cast<double>(h[q].y) - alpha * static_cast<double>(xi.y) -
                               beta_prev * static_cast<double>(pi.y));
        np += static_cast<double>(h[q].x) * static_cast<double>(h[q].x) +
              static_cast<double>(h[q].y) * static_cast<double>(h[q].y);
      }
      const double beta = sqrt(cta_sum<NW>(np, red[1]));
      if (tid == 0) A.alpha[B.ab_off + static_cast<int64_t>(j) * B.ld + r] = alpha;
      if (beta < 1e-12 || j + 1 == B.K) {  // uniform: every thread holds the same beta
        steps = j + 1;
        break;
      }
      if (tid == 0) A.beta[B.ab_off + static_cast<int64_t>(j) * B.ld + r] = beta;
      const double inv = 1.0 / beta;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {  // v_next replaces v_prev, which only this thread reads
        const int i = tid + q * NT;
        if (i < D) vp[i] = CT<T>::make(static_cast<double>(h[q].x) * inv, static_cast<double>(h[q].y) * inv);
      }
      __syncthreads();
      C* tmp = vp;
      vp = v;
      v = tmp;
      beta_prev = beta;
    }
    if (tid == 0) A.steps[B.steps_off + r] = steps;
  }
}

template <typename T, int NT, int RPT>
void launch_small(Ctx& c, const SmallArgs& A, cudaStream_t st) {
  const size_t smem = sizeof(double2) * 16 * A.nsite + static_cast<size_t>(2) * A.cap * sizeof(typename CT<T>::C);
  auto kern = k_lanczos_small<T, NT, RPT>;
  smem_limit(kern, sizeof(double2) * 16 * 64 + static_cast<size_t>(2) * kSmallMaxDim * sizeof(typename CT<T>::C));
  int per_sm = 0;
  FTLM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem));
  if (per_sm < 1) throw Error(FTLM_ERR_CAPACITY, "small-block Lanczos does not fit on an SM");
  const int grid = static_cast<int>(std::min<int64_t>(A.ntasks, static_cast<int64_t>(c.sm_count) * per_sm));
  kern<<<grid, NT, smem, st>>>(A);
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
}

template <typename T>
void launch_class(Ctx& c, int cls, const SmallArgs& A, cudaStream_t st) {
  if (cls == 0) launch_small<T, 256, 2>(c, A, st);
  else if (cls == 1) launch_small<T, 512, 2>(c, A, st);
  else launch_small<T, 1024, 4>(c, A, st);
}

void side_sync(Ctx& c) {
  for (cudaStream_t s : c.side)
    if (s) FTLM_CUDA(cudaStreamSynchronize(s));
}

// Room for `bytes` in a pooled buffer; the side streams are idle when it moves.
void pool_room(Ctx& c, DBuf& b, size_t bytes) {
  if (bytes <= b.cap) return;
  side_sync(c);
  b.ensure_keep(std::max(bytes, 2 * b.cap), c.stream);
}

// Lanczos of the blocks (rows in the sb_* arrays), one launch per size class,
// on the next side stream when pooling, else on c.stream.
void small_lanczos(Ctx& c, const std::vector<SmallBlockDesc>& blocks) {
  const int R = c.opts.samples;
  const bool fp32 = c.opts.precision == FTLM_PREC_MIXED;
  // tasks by size class, largest block first within one
  std::vector<int> order(blocks.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return blocks[a].dim > blocks[b].dim; });
  std::vector<int2> tasks;
  tasks.reserve(blocks.size() * R);
  int first[4] = {0, 0, 0, 0}, cap[3] = {1, 1, 1};
  for (int cls = 2; cls >= 0; --cls) {
    for (int b : order) {
      const int d = blocks[b].dim;
      if ((d > 1024 ? 2 : d > 512 ? 1 : 0) != cls) continue;
      cap[cls] = std::max(cap[cls], d);
      for (int r = 0; r < R; ++r) tasks.push_back(make_int2(b, r));
    }
    first[3 - cls] = static_cast<int>(tasks.size());
  }
  const size_t tbytes = (sizeof(int2) * tasks.size() + 15) / 16 * 16, dbytes = sizeof(SmallBlockDesc) * blocks.size();
  pool_room(c, c.sb_meta, static_cast<size_t>(c.sb_meta_used) + tbytes + dbytes);
  char* meta = c.sb_meta.as<char>() + c.sb_meta_used;
  c.sb_meta_used += static_cast<int64_t>((tbytes + dbytes + 15) / 16 * 16);
  int2* d_tasks = reinterpret_cast<int2*>(meta);
  SmallBlockDesc* d_desc = reinterpret_cast<SmallBlockDesc*>(meta + tbytes);
  FTLM_CUDA(cudaMemcpyAsync(d_tasks, tasks.data(), sizeof(int2) * tasks.size(), cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(d_desc, blocks.data(), dbytes, cudaMemcpyHostToDevice, c.stream));
  SmallArgs A{};
  A.nsite = c.geom.n;
  A.blocks = d_desc;
  A.ent = c.sb_ent.as<uint32_t>();
  A.cnt = c.sb_cnt.as<int32_t>();
  A.diag = c.sb_diag.as<double>();
  A.phase = c.pack.phase.as<double>();
  A.start = c.sb_start.as<double2>();
  A.alpha = c.sb_alpha.as<double>();
  A.beta = c.sb_beta.as<double>();
  A.steps = c.sb_steps.as<int32_t>();
  std::copy(c.geom.amp_re, c.geom.amp_re + 8, A.amp_re);
  std::copy(c.geom.amp_im, c.geom.amp_im + 8, A.amp_im);
  std::copy(c.geom.sqrt_deg, c.geom.sqrt_deg + 65, A.sqrt_deg);
  A.ratios = small_ratios(c.geom.n);
  cudaStream_t st = c.stream;
  if (c.spectra_defer && !c.timing) {
    cudaStream_t& s = c.side[c.side_next];
    c.side_next = (c.side_next + 1) % Ctx::kSide;
    if (!s) FTLM_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    if (!c.side_ev) FTLM_CUDA(cudaEventCreateWithFlags(&c.side_ev, cudaEventDisableTiming));
    FTLM_CUDA(cudaEventRecord(c.side_ev, c.stream));
    FTLM_CUDA(cudaStreamWaitEvent(s, c.side_ev, 0));
    st = s;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (c.timing) {
    FTLM_CUDA(cudaEventCreate(&e0));
    FTLM_CUDA(cudaEventCreate(&e1));
    FTLM_CUDA(cudaEventRecord(e0, c.stream));
  }
  for (int cls = 2; cls >= 0; --cls) {
    A.tasks = d_tasks + first[2 - cls];
    A.ntasks = first[3 - cls] - first[2 - cls];
    A.cap = cap[cls];
    if (A.ntasks == 0) continue;
    if (fp32) launch_class<float>(c, cls, A, st);
    else launch_class<double>(c, cls, A, st);
  }
  if (c.timing) {
    FTLM_CUDA(cudaEventRecord(e1, c.stream));
    FTLM_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    FTLM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    c.prof.small_ms += ms;
    c.prof.small_tasks += static_cast<int64_t>(tasks.size());
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
}

}  // namespace

void small_join(Ctx& c) {
  for (cudaStream_t s : c.side) {
    if (!s) continue;
    FTLM_CUDA(cudaEventRecord(c.side_ev, s));
    FTLM_CUDA(cudaStreamWaitEvent(c.stream, c.side_ev, 0));
  }
}

// The next blocks overwrite the arrays in c.stream's order, which small_join
// has put behind the side streams.
void small_rows_reset(Ctx& c) {
  c.sb_ent_used = c.sb_row_used = c.sb_start_used = c.sb_ab_used = c.sb_st_used = c.sb_meta_used = 0;
}

RitzJob small_ritz_job(Ctx& c, const SmallBlockDesc& d, Spectrum* out) {
  return RitzJob{c.opts.samples, c.opts.samples, d.ld, d.K, c.sb_alpha.as<double>() + d.ab_off,
                 c.sb_beta.as<double>() + d.ab_off, c.sb_steps.as<int32_t>() + d.steps_off, out};
}

void run_small_ftlm_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks) {
  if (blocks.empty()) return;
  const int R = c.opts.samples;
  const bool ref_start = c.opts.start_vector == FTLM_START_REF_GAUSSIAN;
  int ld = 1;  // alpha/beta row stride, as the sweep path uses for one sweep of R vectors
  while (ld < std::max(R, c.opts.precision == FTLM_PREC_MIXED ? 2 : 1)) ld <<= 1;
  const int64_t most = static_cast<int64_t>(c.geom.ndir) * (c.sec.n_up + c.sec.n_dn);  // hops of a row, at most
  struct Item {
    int mx, my;
    SmallBlockDesc d;
  };
  std::vector<Item> items;
  std::vector<PackItem> rows;
  int64_t ent = 0, row = 0, start = 0, ab = 0, st = 0;
  for (const auto& b : blocks) {
    const int64_t D = c.block_dims.at(static_cast<size_t>(b.second * c.geom.lx + b.first));
    if (D <= 0) continue;
    if (D > kSmallMaxDim) throw Error(FTLM_ERR_ARG, "block too large for the small-block FTLM launch");
    SmallBlockDesc d{};
    d.dim = static_cast<int32_t>(D);
    d.K = static_cast<int32_t>(std::min<int64_t>(c.opts.lanczos_steps, D));
    d.ld = ld;
    d.k = b.second * c.geom.lx + b.first;
    d.seed = block_seed(c.opts.seed, c.sec.n_up, c.sec.n_dn, b.first, b.second);
    d.ent_off = ent;
    d.row_off = row;
    d.ab_off = ab;
    d.steps_off = st;
    d.start_off = ref_start ? start : -1;
    ent += D * most;
    row += D;
    ab += static_cast<int64_t>(d.K) * ld;
    st += R;
    if (ref_start) start += static_cast<int64_t>(R) * D;
    items.push_back({b.first, b.second, d});
  }
  if (items.empty()) return;
  const int64_t add = static_cast<int64_t>(sizeof(uint32_t)) * ent +
                      static_cast<int64_t>(sizeof(int32_t) + sizeof(double)) * row +
                      static_cast<int64_t>(sizeof(double2)) * start + static_cast<int64_t>(2 * sizeof(double)) * ab;
  if (defer_pool_bytes(c) > 0 && defer_pool_bytes(c) + add > kDeferPoolBytes) flush_deferred(c);
  for (Item& it : items) {
    it.d.ent_off += c.sb_ent_used;
    it.d.row_off += c.sb_row_used;
    it.d.ab_off += c.sb_ab_used;
    it.d.steps_off += c.sb_st_used;
    if (ref_start) it.d.start_off += c.sb_start_used;
    PackItem p{};
    p.mx = it.mx;
    p.my = it.my;
    p.n = it.d.dim;
    p.off = it.d.ent_off;
    p.off2 = it.d.row_off;
    rows.push_back(p);
  }
  pool_room(c, c.sb_ent, sizeof(uint32_t) * std::max<int64_t>(c.sb_ent_used + ent, 1));
  pool_room(c, c.sb_cnt, sizeof(int32_t) * (c.sb_row_used + row));
  pool_room(c, c.sb_diag, sizeof(double) * (c.sb_row_used + row));
  pool_room(c, c.sb_alpha, sizeof(double) * (c.sb_ab_used + ab));
  pool_room(c, c.sb_beta, sizeof(double) * (c.sb_ab_used + ab));
  pool_room(c, c.sb_steps, sizeof(int32_t) * (c.sb_st_used + st));
  FTLM_CUDA(cudaMemsetAsync(c.sb_alpha.as<double>() + c.sb_ab_used, 0, sizeof(double) * ab, c.stream));
  FTLM_CUDA(cudaMemsetAsync(c.sb_beta.as<double>() + c.sb_ab_used, 0, sizeof(double) * ab, c.stream));
  pack_entries(c, rows, c.sb_ent.as<uint32_t>(), c.sb_cnt.as<int32_t>(), c.sb_diag.as<double>());
  if (ref_start) {  // Philox start vectors are drawn by the Lanczos launch
    std::vector<GaussJob> jobs;
    for (const Item& it : items)
      for (int r = 0; r < R; ++r)
        jobs.push_back({sample_seed(it.d.seed, r), it.d.dim, it.d.start_off + static_cast<int64_t>(r) * it.d.dim});
    pool_room(c, c.sb_start, sizeof(double2) * (c.sb_start_used + start));
    gaussian_starts(c, jobs, c.sb_start.as<double2>());
  }
  c.sb_ent_used += ent;
  c.sb_row_used += row;
  c.sb_start_used += start;
  c.sb_ab_used += ab;
  c.sb_st_used += st;
  std::vector<SmallBlockDesc> desc;
  for (const Item& it : items) desc.push_back(it.d);
  if (c.spectra_defer) {  // Ritz stage with those of the other sectors, at the flush
    small_lanczos(c, desc);
    for (const Item& it : items) {
      Spectrum s;
      s.exact = false;
      s.prefactor = static_cast<double>(it.d.dim);
      s.particles = c.sec.n_up + c.sec.n_dn;
      s.dim = it.d.dim;
      s.pending_small = static_cast<int>(c.defer_small.size());
      c.spec[{it.mx, it.my}] = s;
      c.defer_small.push_back(DeferSmall{c.sec.n_up, c.sec.n_dn, it.mx, it.my, it.d, c.sec_gen});
    }
    return;
  }
  struct Reset {  // the rows are this call's own, whether it succeeds or throws
    Ctx& c;
    ~Reset() { small_rows_reset(c); }
  } reset{c};
  small_lanczos(c, desc);
  // Ritz values and weights per block, then compaction into the spectra arena
  std::vector<Spectrum> spec(items.size());
  std::vector<RitzJob> jobs;
  for (size_t i = 0; i < items.size(); ++i) jobs.push_back(small_ritz_job(c, desc[i], &spec[i]));
  ritz_stage_many(c, jobs);
  for (size_t i = 0; i < items.size(); ++i) {
    spec[i].prefactor = static_cast<double>(items[i].d.dim);
    spec[i].particles = c.sec.n_up + c.sec.n_dn;
    spec[i].dim = items[i].d.dim;
    c.spec[{items[i].mx, items[i].my}] = spec[i];
  }
}

}  // namespace ftlm
