// Split-spin H*V: the momentum-block Hamiltonian applied as two
// segment-local sweeps.
//
// Rows of a block are orbit representatives in the reference's parent order
// (main.cpp:643-675): (up representative ur, canonical down word), so the
// rows sharing an ur form one contiguous segment of at most C(N, N_down)
// rows. A down-spin hop keeps ur, so its target lies in the source row's own
// segment (13 MB of a 128-vector FP32 sweep on the 4x4 half-filled sector:
// L2-resident while the CTAs walk the rows in order). An up-spin hop lands in
// another segment and, on a large block, misses L2. The spin flip S
// (u, d) -> (d, u) maps the block onto the same momentum block of sector
// (N_down, N_up) and turns up-spin hops into down-spin hops there, so with
// the reference's matrix convention (M[src][tgt] = coefficient of |tgt,k> in
// H|src,k>, main.cpp:779-804)
//
//   M x = (diag + M_dn) x + S^T M'_dn conj(S) x,
//
// where M'_dn holds the down-spin hops of sector (N_down, N_up) and S is a
// permutation with one unit phase per row: row q of this block (state
// (u, d)) has the flipped state (d, u) = sign * T_shift(rep) of flipped row
// p(q), f_q = sign * e^{i k.shift}, and
//
//   x_D[p(q)] = conj(f_q) x[q],     (M_up x)[q] = f_q (M'_dn x_D)[p(q)].
//
// Both sweeps gather only inside the current segment. The Lanczos update
// writes w_{j+1} in both row orders, so no permutation pass runs per step.
// Alpha = Re<x, M x> = Re<x, y_U> + Re<x_D, y_D> (S is unitary). For
// N_up == N_down the flipped sector is the sector itself and its tables are
// shared.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "ftlm_internal.h"
#include "hv_common.cuh"

namespace ftlm {

namespace {

constexpr int kSegGrab = 2;  // rows a warp takes from the shared row counter at a time

int grid_rows(int64_t n, int threads) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 1 << 20)));
}

// Output rows are written once and read once by the Lanczos update: evict
// them first so the segment being gathered keeps its place in L2.
__device__ __forceinline__ void st_stream(float4* p, const float4& v) { __stcs(p, v); }
__device__ __forceinline__ void st_stream(double2* p, const double2& v) { __stcs(p, v); }

// Down-spin hops of every row of the block P.v (+ the diagonal term when
// with_diag): y = s * ((diag) x + M_dn x), per-CTA fixed-point partials of
// Re<s x, y>. One warp per row: lanes queue the row's down-spin hops, resolve
// one target each inside the segment (rank of the moved word -> class table
// of ur -> active index + segment offset), then groups of G lanes gather the
// target rows of all NV vectors. Hop order within a row: occupied source
// sites ascending, directions ascending (the reference's hop order).
template <typename W, typename R, typename T, int NV, int U, int MINB>
__global__ void __launch_bounds__(kHvThreads, MINB) k_hv_seg(const __grid_constant__ HvParams<W> P,
                                                           const typename CT<T>::V* __restrict__ in,
                                                           typename CT<T>::V* __restrict__ out,
                                                           const double* __restrict__ scale,
                                                           fx128* __restrict__ partial, const R* __restrict__ gbinom,
                                                           int with_diag, unsigned long long* __restrict__ next_row) {
  using V = typename CT<T>::V;
  constexpr int VPL = CT<T>::VPL;
  constexpr int CPR = NV / VPL;
  constexpr int G = CPR < 32 ? CPR : 32;
  constexpr int LPL = CPR / G;
  constexpr bool kSmemBinom = sizeof(W) == 4;
  constexpr int kQ = 8 * static_cast<int>(sizeof(W)) * 8;  // 8 directions x occupied sites of one spin

  __shared__ R s_binom[kSmemBinom ? 32 * 65 : 1];
  __shared__ int8_t s_nb[64][8];
  __shared__ double s_ph[2][64];
  __shared__ double s_amp[2][8];
  __shared__ double s_sq[65];
  __shared__ uint16_t s_q[kHvWarps][kQ];
  __shared__ fx128 s_acc[kHvWarps][NV];

  const Geom& g = P.g;
  const BlockView<W>& v = P.v;
  const int tid = threadIdx.x;
  if (kSmemBinom)
    for (int i = tid; i < 32 * 65; i += kHvThreads) s_binom[i] = gbinom[i];
  const R* binom = kSmemBinom ? s_binom : gbinom;
  for (int i = tid; i < 64 * 8; i += kHvThreads) s_nb[i / 8][i % 8] = g.nb[i / 8][i % 8];
  for (int i = tid; i < 64; i += kHvThreads) {
    s_ph[0][i] = v.phase_re[i];
    s_ph[1][i] = v.phase_im[i];
  }
  if (tid < 8) {
    s_amp[0][tid] = g.amp_re[tid];
    s_amp[1][tid] = g.amp_im[tid];
  }
  if (tid < 65) s_sq[tid] = g.sqrt_deg[tid];
  for (int i = tid; i < kHvWarps * NV; i += kHvThreads) s_acc[i / NV][i % NV] = 0;
  __syncthreads();

  const int lane = tid & 31;
  const int wid = tid >> 5;
  const int grp = lane / G;
  const int sub = lane % G;
  uint16_t* queue = s_q[wid];
  double sc[LPL][VPL];
#pragma unroll
  for (int l = 0; l < LPL; ++l)
#pragma unroll
    for (int e = 0; e < VPL; ++e) sc[l][e] = scale ? scale[(l * G + sub) * VPL + e] : 1.0;

  // Rows in order: from a shared counter (next_row, zeroed before the
  // launch), kSegGrab rows per grab, so all warps stay within a few thousand
  // consecutive rows and the segment they gather from stays in L2; or
  // grid-stride when next_row is null. The order does not change any result:
  // rows are independent and the dot partials are exact integer sums.
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * kHvWarps;
  int64_t grab = 0, grab_end = 0;
  int64_t row = static_cast<int64_t>(blockIdx.x) * kHvWarps + wid;
  // lane 0 keeps the next grab in flight while the current rows are processed
  unsigned long long pend = 0;
  if (next_row && lane == 0) pend = atomicAdd(next_row, static_cast<unsigned long long>(kSegGrab));
  while (true) {
    if (next_row) {
      if (grab >= grab_end) {
        grab = static_cast<int64_t>(__shfl_sync(0xffffffffu, pend, 0));
        grab_end = min(grab + kSegGrab, v.dim);
        if (lane == 0 && grab < v.dim) pend = atomicAdd(next_row, static_cast<unsigned long long>(kSegGrab));
      }
      row = grab++;
    }
    if (row >= v.dim) break;
    const uint32_t meta = __ldg(v.row_meta + row);
    const uint32_t ur = meta & 0x3FFFFFFu;
    const int deg_s = static_cast<int>(meta >> 26) + 1;
    const W d = __ldg(v.row_dn + row);
    const int cls = __ldg(v.ur_class + ur);
    const int64_t seg = __ldg(v.aoff + ur);
    const uint64_t* dt = v.dtab + static_cast<int64_t>(cls > 0 ? cls - 1 : 0) * v.c_dn;
    const double inv_s = 1.0 / s_sq[deg_s];

    // 1) hop queue: lane k takes the k-th occupied site of the down word
    int total = 0;
    for (int k0 = 0; k0 < v.n_dn; k0 += 32) {
      const int k = k0 + lane;
      uint32_t dm = 0;
      int from = 0;
      if (k < v.n_dn) {
        from = kth_bit(d, k);
        for (int j = 0; j < g.ndir; ++j) {
          const int to = s_nb[from][g.dirs[j]];
          if (!((d >> to) & 1)) dm |= 1u << j;
        }
      }
      const int cnt = __popc(dm);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      int pos = total + incl - cnt;
      for (uint32_t m = dm; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        queue[pos++] = static_cast<uint16_t>((from << 3) | g.dirs[j]);
      }
      total += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();

    // 2) resolve 32 hops at a time, gather their rows
    V acc[LPL];
#pragma unroll
    for (int l = 0; l < LPL; ++l) vzero(acc[l]);
    for (int b = 0; b < total; b += 32) {
      const int q = b + lane;
      int64_t col = -1;
      T cr = 0, ci = 0;
      if (q < total) {
        const int code = queue[q];
        const int from = code >> 3, dir = code & 7;
        const int to = s_nb[from][dir];
        const W moved = d ^ (static_cast<W>(1) << from) ^ (static_cast<W>(1) << to);
        const int64_t rd = static_cast<int64_t>(rank_of<W, R>(moved, binom));
        int64_t a = rd;
        int h = 0, s = 0, deg_t = 1;
        if (cls != 0) {
          const uint64_t e = __ldg(dt + rd);
          a = static_cast<int32_t>(static_cast<uint32_t>(e));
          h = static_cast<int>((e >> 32) & 0xFF);
          s = static_cast<int>((e >> 40) & 1);
          deg_t = static_cast<int>((e >> 48) & 0xFF);
        }
        if (a >= 0) {
          col = seg + a;
          const int p = jw_parity(d, from, to) ^ s;
          const double ar = p ? -s_amp[0][dir] : s_amp[0][dir];
          const double ai = p ? -s_amp[1][dir] : s_amp[1][dir];
          const double pr = s_ph[0][h], pi = s_ph[1][h];
          const double ratio = s_sq[deg_t] * inv_s;
          cr = static_cast<T>((ar * pr - ai * pi) * ratio);
          ci = static_cast<T>((ar * pi + ai * pr) * ratio);
        }
      }
      gather_batch<T, NV, U>(in, col, cr, ci, min(32, total - b), acc);
    }
    __syncwarp();
    // 3) fold the HPAR partial sums
#pragma unroll
    for (int o = G; o < 32; o <<= 1)
#pragma unroll
      for (int l = 0; l < LPL; ++l) vadd(acc[l], shfl_xor_v(acc[l], o));
    // 4) own-row term, scale, store, Lanczos dot
    if (grp == 0) {
      const double diag = with_diag ? diag_energy(__ldg(v.ur_bits + ur), d, g) : 0.0;
#pragma unroll
      for (int l = 0; l < LPL; ++l) {
        const V x = ld_stream(in + row * CPR + l * G + sub);
        double dt2[VPL];
        st_stream(out + row * CPR + l * G + sub, finish_row(x, acc[l], diag, sc[l], dt2));
        if (partial) {
#pragma unroll
          for (int e = 0; e < VPL; ++e) s_acc[wid][(l * G + sub) * VPL + e] += fx_of(dt2[e]);
        }
      }
    }
    if (!next_row) row += nwarps;
  }
  flush_dot<NV>(s_acc, partial);
}

// ---------------------------------------------------------------- stencils
//
// Class stencils: within one segment (fixed up representative ur) the
// down-spin operator depends only on the stabiliser class of ur, not on ur
// itself. Class 0 (trivial stabiliser) has every down word as a row in rank
// order; class c > 0 has its active canonical down words (act_list). So the
// down-spin hops of a whole block are one small CSR per class ("stencil"),
// rows = class rows, entries = the hop's target index inside the segment
// (16 bits) | dir << 16 | parity << 19 | shift << 20 | (deg - 1) << 26, in the
// on-the-fly kernel's hop order (source site ascending, direction ascending;
// hops to inactive orbits left out). The stencils of a 4x4 half-filled block
// take about 1 MB and stay in L1/L2, so a sweep reads per row only its row
// metadata and the gathered rows; the per-row rank and class-table lookups
// of k_hv_seg are gone. Needs C(N, N_down) <= 65536 (18 sites at half filling).

constexpr int64_t kStencilMaxRows = 65536;

template <typename W>
__global__ void k_stencil(int fill, const __grid_constant__ Geom g, int nclass, const int64_t* __restrict__ crb,
                          int64_t c_dn, const uint32_t* __restrict__ act_list, const uint64_t* __restrict__ dtab,
                          const W* __restrict__ dns, const uint64_t* __restrict__ binom, int64_t rows,
                          int32_t* __restrict__ counts, const int64_t* __restrict__ rp, uint32_t* __restrict__ ent) {
  for (int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; r < rows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int lo = 0, hi = nclass - 1;  // class c with crb[c] <= r < crb[c+1]
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (crb[mid] <= r) lo = mid;
      else hi = mid - 1;
    }
    const int c = lo;
    const int64_t a = r - crb[c];
    const int64_t j = c == 0 ? a : static_cast<int64_t>(act_list[static_cast<int64_t>(c - 1) * c_dn + a]);
    const W d = dns[j];
    int64_t pos = fill ? rp[r] : 0;
    int cnt = 0;
    for (W m = d; m; m &= m - 1) {
      const int from = ctz(m);
      for (int dir = 0; dir < 8; ++dir) {
        if (g.amp_re[dir] == 0.0 && g.amp_im[dir] == 0.0) continue;
        const int to = g.nb[from][dir];
        if ((d >> to) & 1) continue;
        const W moved = d ^ (static_cast<W>(1) << from) ^ (static_cast<W>(1) << to);
        const int64_t rd = static_cast<int64_t>(rank_of<W, uint64_t>(moved, binom));
        int64_t at = rd;
        int h = 0, sg = 0, deg = 1;
        if (c != 0) {
          const uint64_t e = dtab[static_cast<int64_t>(c - 1) * c_dn + rd];
          at = static_cast<int32_t>(static_cast<uint32_t>(e));
          if (at < 0) continue;
          h = static_cast<int>((e >> 32) & 0xFF);
          sg = static_cast<int>((e >> 40) & 1);
          deg = static_cast<int>((e >> 48) & 0xFF);
        }
        if (fill)
          ent[pos++] = static_cast<uint32_t>(at) | (static_cast<uint32_t>(dir) << 16) |
                       (static_cast<uint32_t>(jw_parity(d, from, to) ^ sg) << 19) | (static_cast<uint32_t>(h) << 20) |
                       (static_cast<uint32_t>(deg - 1) << 26);
        ++cnt;
      }
    }
    if (!fill) counts[r] = cnt;
  }
}

// Entries of the wide stencil sweeps, 4 bytes each: target index inside the
// segment : 16 | coefficient id : 15, id = ((ratio * 64 + shift) * 8 + dir) * 2
// + sign, ratio numbering the values of sqrt(deg_t / deg_s) (stn_ratios). Rows
// start at multiples of 4 entries, so four hops cost one 16-byte broadcast
// load. At a trivial stabiliser the id is dir * 2 + sign and the coefficient
// comes from the kernel's parameters (constant cache), else from a table in
// global memory. What this buys: a load of 16 bytes by every lane occupies the
// L1 data pipe for 4 cycles whether or not the address is the same for all
// lanes, so a 16-byte {index, re, im} entry per hop cost as much as the 16-byte
// gather it described (4x4 (4,5), 128 vectors: 73% of the L1 data pipe).
constexpr int kStnMaxRatios = 32;
constexpr int kStnCoefs = 16;  // per (ratio, shift): 8 directions x sign

struct StnRatios {
  int n;                       // number of distinct deg_t / deg_s
  uint8_t num[kStnMaxRatios];  // deg_t, deg_s of the first pair with that ratio
  uint8_t den[kStnMaxRatios];
};

template <typename T>
struct CoefT;
template <>
struct CoefT<float> {
  using C = float2;
};
template <>
struct CoefT<double> {
  using C = double2;
};

// Row order of the stencil sweeps. All segments of a class share their stencil,
// so the segments are taken in groups of S, S segments' vectors filling 64
// chunks of 16 bytes (1 KB), and a group's rows are stored with the segment as
// the fast index: position = base + g S rows + a S_g + s for row a of segment s
// of group g (S_g = S but for the last group of a class). A hop then reads one
// contiguous run of up to 1 KB for all segments of the group, whatever the
// number of vectors, which need not be a power of two, and a group's rows stay
// within a few MB, as one segment's do at 1 KB a row (interleaving a whole
// class spread the gathers of a stencil row over all of the array: 5-7% slower
// at 64 and 128 vectors). The vectors, the diagonal and the flip map of these
// sweeps are kept in this order.
//
// One class of segments (equal stabiliser, hence equal stencil): `rows` rows
// each, stencil rows crb ..., positions base ... .
struct StnClass {
  int32_t nseg, rows, c0, first;  // c0: trivial stabiliser; first: its segments in stn_seg
  int64_t crb, base;
};
constexpr int kStnRun = 64;  // chunks of a full group's row
inline int stn_group(int cpr) { return std::max(1, kStnRun / cpr); }

// One sweep: y = diag * x + M_dn x over all segments of one row order.
template <typename T>
struct StnJob {
  const typename CT<T>::V* in;
  typename CT<T>::V* out;
  const T* diag;  // per position, null: none
  const int2* srow;  // per stencil row: first entry / 4, entries
  const uint4* ent;
  const typename CoefT<T>::C* coef;
  const StnClass* cls;
  int32_t units;  // work units (below) of the job
};
// A group's stencil row, S_g cpr chunks, is cut into `parts` panels of at most
// pw <= 32 LPL chunks, one per warp. A lane's chunks belong to the same vectors
// in every panel of the same part.
struct StnPanels {
  int32_t cpr, seg, parts, pw;  // seg: S
  __host__ __device__ __forceinline__ int64_t count(int64_t nseg) const { return (nseg + seg - 1) / seg * parts; }
};
inline StnPanels stn_panels(int cpr, int lanes) {
  const int seg = stn_group(cpr), run = seg * cpr, parts = (run + lanes - 1) / lanes;
  return {cpr, seg, parts, (run + parts - 1) / parts};
}
template <typename T>
struct StnJobs {
  StnJob<T> j[2];
  int32_t njobs, nv, rows;  // rows per unit
  StnPanels pan;
  typename CoefT<T>::C c0[kStnCoefs];  // class 0: +-amplitude of each direction
};

// Row `a` of a group whose rows are rowb bytes: one 32 x 32 + 64 bit multiply-add.
template <typename V>
__device__ __forceinline__ V* stn_at(V* p, uint32_t a, uint32_t rowb) {
  using B = std::conditional_t<std::is_const_v<V>, const char, char>;
  return reinterpret_cast<V*>(reinterpret_cast<B*>(p) + static_cast<uint64_t>(a) * rowb);
}

// Pairs of FP32 numbers in one register pair.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// At most four hops, summed on their own, then added: acc += sum_u c[u] x[u].
template <int LPL>
__device__ __forceinline__ void stn_four(int n, const float2* c, const float4 (*x)[LPL], float4 (&acc)[LPL]) {
#pragma unroll
  for (int l = 0; l < LPL; ++l) {
    // Re c (x.re, x.im) and Im c (x.re, x.im) of both vectors of a chunk: two
    // multiply-adds a hop and vector, in pairs, where the complex product takes four
    uint64_t r0 = 0, i0 = 0, r1 = 0, i1 = 0;
#pragma unroll
    for (int u = 0; u < n; ++u) {
      const uint64_t cr = pack2(c[u].x, c[u].x), ci = pack2(c[u].y, c[u].y);
      const uint64_t x0 = pack2(x[u][l].x, x[u][l].y), x1 = pack2(x[u][l].z, x[u][l].w);
      r0 = fma2(cr, x0, r0);
      i0 = fma2(ci, x0, i0);
      r1 = fma2(cr, x1, r1);
      i1 = fma2(ci, x1, i1);
    }
    const float2 a0 = unpack2(r0), b0 = unpack2(i0), a1 = unpack2(r1), b1 = unpack2(i1);
    acc[l].x += a0.x - b0.y;
    acc[l].y += a0.y + b0.x;
    acc[l].z += a1.x - b1.y;
    acc[l].w += a1.y + b1.x;
  }
}
template <int LPL>
__device__ __forceinline__ void stn_four(int n, const double2* c, const double2 (*x)[LPL], double2 (&acc)[LPL]) {
#pragma unroll
  for (int l = 0; l < LPL; ++l) {
    double2 t = make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < n; ++u) cfma<double>(t, c[u].x, c[u].y, x[u][l]);
    vadd(acc[l], t);
  }
}

// N hops of a row (entries e): all gathers issued before the first FMA. FOURS: summed
// four at a time, else in a chain.
template <typename T, int LPL, int N, bool C0, bool FOURS>
__device__ __forceinline__ void stn_hops(const uint32_t* e, const StnJobs<T>& P, const typename CoefT<T>::C* coef,
                                         const typename CT<T>::V* __restrict__ xs, uint32_t rowb,
                                         typename CT<T>::V (&acc)[LPL]) {
  using V = typename CT<T>::V;
  V x[N][LPL];
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int l = 0; l < LPL; ++l) x[u][l] = __ldg(stn_at(xs, e[u] & 0xFFFFu, rowb) + l * 32);
  typename CoefT<T>::C c[N];
#pragma unroll
  for (int u = 0; u < N; ++u) {
    if constexpr (C0) c[u] = P.c0[e[u] >> 16];
    else c[u] = __ldg(coef + (e[u] >> 16));
  }
  if constexpr (FOURS) {
    stn_four<LPL>(N < 4 ? N : 4, c, x, acc);
    if constexpr (N > 4) stn_four<LPL>(N - 4, c + 4, x + 4, acc);
  } else {
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
      for (int l = 0; l < LPL; ++l) cfma<T>(acc[l], c[u].x, c[u].y, x[u][l]);
  }
}

// All hops of a row, U (4 or 8) at a time, then the remainder.
template <typename T, int LPL, int U, bool C0, bool FOURS>
__device__ __forceinline__ void stn_row(const uint4* q, int left, const StnJobs<T>& P,
                                        const typename CoefT<T>::C* coef, const typename CT<T>::V* __restrict__ xs,
                                        uint32_t rowb, typename CT<T>::V (&acc)[LPL]) {
  uint4 p = __ldg(q);
  if constexpr (U == 8) {
    while (left >= 8) {
      const uint4 p2 = __ldg(q + 1);
      const uint32_t e[8] = {p.x, p.y, p.z, p.w, p2.x, p2.y, p2.z, p2.w};
      q += 2;
      p = __ldg(q);
      stn_hops<T, LPL, 8, C0, FOURS>(e, P, coef, xs, rowb, acc);
      left -= 8;
    }
  }
  while (left >= 4) {
    const uint32_t e[4] = {p.x, p.y, p.z, p.w};
    p = __ldg(++q);
    stn_hops<T, LPL, 4, C0, FOURS>(e, P, coef, xs, rowb, acc);
    left -= 4;
  }
  const uint32_t e[3] = {p.x, p.y, p.z};
  if (left == 1) stn_hops<T, LPL, 1, C0, FOURS>(e, P, coef, xs, rowb, acc);
  else if (left == 2) stn_hops<T, LPL, 2, C0, FOURS>(e, P, coef, xs, rowb, acc);
  else if (left == 3) stn_hops<T, LPL, 3, C0, FOURS>(e, P, coef, xs, rowb, acc);
}

__device__ __forceinline__ void stn_finish(float4& y, const float4& x, float d, double* dot) {
  y.x = fmaf(d, x.x, y.x);
  y.y = fmaf(d, x.y, y.y);
  y.z = fmaf(d, x.z, y.z);
  y.w = fmaf(d, x.w, y.w);
  dot[0] += static_cast<double>(x.x) * y.x + static_cast<double>(x.y) * y.y;
  dot[1] += static_cast<double>(x.z) * y.z + static_cast<double>(x.w) * y.w;
}
__device__ __forceinline__ void stn_finish(double2& y, const double2& x, double d, double* dot) {
  y.x = fma(d, x.x, y.x);
  y.y = fma(d, x.y, y.y);
  dot[0] += x.x * y.x + x.y * y.y;
}

// The segment sweeps on the class stencils, one launch for both row orders.
//
// A warp takes a panel of a stencil row (32 lanes of LPL 16-byte chunks, 512 LPL
// contiguous bytes per hop): the row's entries are warp-uniform (one broadcast
// load per four hops, no shuffles, no divergence, no lanes' sums to fold). A
// work unit is P.rows stencil rows (stn_rows), kStnLane apart, of one panel;
// kStnLane consecutive units cover kStnLane * P.rows consecutive rows. A CTA
// takes one unit per warp, consecutive ones, from a shared counter, so at any
// moment its warps are on neighbouring rows, which share gather targets (hops
// among the low sites stay within a few hundred rows): a quarter of the
// gathered sectors hit L1. Lanes past the end of a panel load what follows it
// (the arrays end in kSweepPad spare bytes) and drop the result.
//
// A row's hops are added in fours or in a chain (stn_fours; the times below are the chain's).
//
// Bound: waits for gathered lines at 16-24 warps per SM (L1 67% busy with 30%
// hits, L2 50%; 17-20 TB/s of gathered bytes). Per H*V, both sweeps, against the
// same kernel on one short row per segment (the row order of the block):
// 6x3 (5,5) 16 FP32 vectors 1.90 -> 1.64 ms, 4x4 (4,4) 5 FP64 vectors (then
// padded to 8) 0.111 -> 0.086, 4x4 (6,6) 2 FP32 vectors 0.28 against 1.56 of the
// hop list; 4x4 (8,8) 64 vectors 11.6 -> 11.3, 4x4 (5,5) 128 vectors unchanged.
//
// y is NOT scaled (the Lanczos update applies the scale of the unnormalised
// vectors). The dot terms Re<x, y> of a unit are summed in FP64 in row order
// per segment and vector, scaled by scale^2 and added as 128-bit integers:
// neither the grid, the panels nor the assignment of units changes the sum.
constexpr int kStnLane = 8;
// Units of one group of segments of `rows` rows, `per` rows a unit.
__host__ __device__ __forceinline__ unsigned int stn_chunks(int64_t rows, int per) {
  const int64_t full = rows / (kStnLane * per), rest = rows % (kStnLane * per);
  return static_cast<unsigned int>(full * kStnLane + (rest < kStnLane ? rest : kStnLane));
}

constexpr int kStnSlots = 128;  // dot terms of a warp: parts x 32 LPL chunks x vectors per chunk, at most

template <typename T, int LPL, int U, int NT, int MINB, bool FOURS>
__global__ void __launch_bounds__(NT, MINB) k_hv_stn(const __grid_constant__ StnJobs<T> P,
                                                     const double* __restrict__ scale, fx128* __restrict__ partial,
                                                     unsigned int* __restrict__ next_item) {
  using V = typename CT<T>::V;
  constexpr int VPL = CT<T>::VPL;
  constexpr int NW = NT / 32;
  __shared__ fx128 s_acc[NW][kStnSlots];
  __shared__ unsigned int s_item[2];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int wid = tid >> 5;
  const int cpr = P.pan.cpr, parts = P.pan.parts, pw = P.pan.pw;
  const unsigned int total = static_cast<unsigned int>(P.j[0].units) + (P.njobs > 1 ? P.j[1].units : 0);
  const unsigned int nitems = (total + NW - 1) / NW;
  if (partial) {
    for (int i = tid; i < NW * kStnSlots; i += NT) s_acc[i / kStnSlots][i % kStnSlots] = 0;
    __syncthreads();
  }
  int jb = 0, cl = 0;
  unsigned int cbase = 0;  // first unit of class cl of job jb
  unsigned int item = blockIdx.x;
  if (next_item) {
    if (tid == 0) s_item[1] = atomicAdd(next_item, 1u);
    __syncthreads();
    item = s_item[1];
  }
  for (int it = 0; item < nitems; ++it) {
    unsigned int nxt = item + gridDim.x;
    if (next_item && tid == 0) nxt = atomicAdd(next_item, 1u);
    const unsigned int unit = item * NW + wid;
    if (unit < total) {
      // units grow monotonically, so job and class only move forward
      unsigned int ju = unit;
      if (ju >= static_cast<unsigned int>(P.j[0].units)) {
        ju -= P.j[0].units;
        if (jb == 0) {
          jb = 1;
          cl = 0;
          cbase = 0;
        }
      }
      const StnJob<T>& J = P.j[jb];
      StnClass C = J.cls[cl];
      unsigned int nch = stn_chunks(C.rows, P.rows);
      unsigned int cu = nch * static_cast<unsigned int>(P.pan.count(C.nseg));
      while (ju >= cbase + cu) {
        cbase += cu;
        C = J.cls[++cl];
        nch = stn_chunks(C.rows, P.rows);
        cu = nch * static_cast<unsigned int>(P.pan.count(C.nseg));
      }
      const unsigned int q = (ju - cbase) / nch;
      const int ch = static_cast<int>(ju - cbase - q * nch);
      const int a0 = (ch / kStnLane) * (kStnLane * P.rows) + ch % kStnLane;
      const int g = static_cast<int>(q) / parts, part = static_cast<int>(q) - g * parts;
      const int nsg = min(P.pan.seg, C.nseg - g * P.pan.seg);  // segments of the group
      const uint32_t rowb = static_cast<uint32_t>(nsg * cpr) * sizeof(V);  // bytes of its rows
      const int c0 = part * pw;
      const int here = min(pw, nsg * cpr - c0);  // none in the last parts of a short group
      const int64_t gbase = C.base + static_cast<int64_t>(g) * P.pan.seg * C.rows;
      const int64_t off = gbase * cpr + c0 + lane;
      const V* xs = J.in + off;
      V* ys = J.out + off;
      const T* dg[LPL];
#pragma unroll
      for (int l = 0; l < LPL; ++l)
        dg[l] = J.diag ? J.diag + gbase + min(c0 + l * 32 + lane, nsg * cpr - 1) / cpr : nullptr;
      double dot[LPL][VPL];
#pragma unroll
      for (int l = 0; l < LPL; ++l)
#pragma unroll
        for (int e = 0; e < VPL; ++e) dot[l][e] = 0.0;
      const int nr = here > 0 ? min(P.rows, (C.rows - a0 + kStnLane - 1) / kStnLane) : 0;
      const int2 hp = __ldg(J.srow + C.crb + a0 + kStnLane * min(lane, max(nr, 1) - 1));
      for (int r = 0; r < nr; ++r) {
        const int a = a0 + r * kStnLane;
        const uint4* q4 = J.ent + __shfl_sync(0xffffffffu, hp.x, r);
        const int left = __shfl_sync(0xffffffffu, hp.y, r);
        V acc[LPL];
#pragma unroll
        for (int l = 0; l < LPL; ++l) vzero(acc[l]);
        T d[LPL];
#pragma unroll
        for (int l = 0; l < LPL; ++l) d[l] = J.diag ? __ldg(dg[l] + a * nsg) : T(0);
        V xo[LPL];
#pragma unroll
        for (int l = 0; l < LPL; ++l) xo[l] = __ldg(stn_at(xs, a, rowb) + l * 32);
        if (C.c0) stn_row<T, LPL, U, true, FOURS>(q4, left, P, J.coef, xs, rowb, acc);
        else stn_row<T, LPL, U, false, FOURS>(q4, left, P, J.coef, xs, rowb, acc);
#pragma unroll
        for (int l = 0; l < LPL; ++l) {
          stn_finish(acc[l], xo[l], d[l], dot[l]);
          if (l * 32 + lane < here) st_stream(stn_at(ys, a, rowb) + l * 32, acc[l]);
        }
      }
      if (partial) {
#pragma unroll
        for (int l = 0; l < LPL; ++l)
          if (l * 32 + lane < here) {
            const int v = (c0 + l * 32 + lane) % cpr * VPL;
#pragma unroll
            for (int e = 0; e < VPL; ++e) {
              const double sc = scale ? __ldg(scale + v + e) : 1.0;
              s_acc[wid][((part * LPL + l) * VPL + e) * 32 + lane] += fx_of(sc * (sc * dot[l][e]));
            }
          }
      }
    }
    if (tid == 0) s_item[it & 1] = nxt;
    __syncthreads();
    item = s_item[it & 1];
  }
  if (!partial) return;
  __syncthreads();
  for (int i = tid; i < kStnSlots; i += NT) {
    fx128 t = s_acc[0][i];
    for (int w = 1; w < NW; ++w) t += s_acc[w][i];
    s_acc[0][i] = t;
  }
  __syncthreads();
  for (int v = tid; v < P.nv; v += NT) {
    const int e = v % VPL;
    fx128 t = 0;
    for (int c = v / VPL; c < P.pan.seg * cpr; c += cpr) {
      const int part = c / pw, k = c - part * pw;
      t += s_acc[0][((part * LPL + k / 32) * VPL + e) * 32 + k % 32];
    }
    partial[static_cast<int64_t>(blockIdx.x) * P.nv + v] = t;
  }
}

// Flip map of every row q of block Pu: the flipped state (d, u) resolved in
// the tables vd of sector (N_down, N_up): row p | shift << 32 | sign << 38,
// both sides in the sweeps' row order (pos, pos_d; null: block order).
template <typename W>
__global__ void k_flip_map(const __grid_constant__ HvParams<W> Pu, const __grid_constant__ BlockView<W> vd,
                           const uint64_t* __restrict__ binom, const uint32_t* __restrict__ pos,
                           const uint32_t* __restrict__ pos_d, uint64_t* __restrict__ fmap, int* __restrict__ bad) {
  const BlockView<W>& v = Pu.v;
  for (int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; q < v.dim;
       q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint32_t ur = v.row_meta[q] & 0x3FFFFFFu;
    const W u = v.ur_bits[ur];
    const W d = v.row_dn[q];
    int64_t col;
    int shift, sgn, deg;
    if (!resolve<W, uint64_t>(d, u, true, 0, vd, Pu.g, binom, col, shift, sgn, deg) || col < 0 || col >= vd.dim) {
      atomicAdd(bad, 1);
      fmap[pos ? pos[q] : q] = 0;
      continue;
    }
    if (pos_d) col = pos_d[col];
    fmap[pos ? pos[q] : q] = static_cast<uint64_t>(col) | (static_cast<uint64_t>(shift) << 32) | (static_cast<uint64_t>(sgn) << 38);
  }
}

// x_D[p(q)] = conj(f_q) x[q] for every 16-byte chunk.
template <typename T>
__global__ void k_flip_scatter(int64_t dim, int CPR, const typename CT<T>::V* __restrict__ x,
                               typename CT<T>::V* __restrict__ xd, const uint64_t* __restrict__ fmap,
                               const __grid_constant__ FlipPhase ph) {
  const int64_t n = dim * CPR;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / CPR;
    int64_t p;
    double fr, fi;
    flip_coef(__ldg(fmap + row), ph, p, fr, fi);
    xd[p * CPR + (i - row * CPR)] = cmul_conj<T>(fr, fi, x[i]);
  }
}

// y[q] += f_q y_D[p(q)] for every 16-byte chunk (FP64 arithmetic).
template <typename T>
__global__ void k_flip_gather_add(int64_t dim, int CPR, typename CT<T>::V* __restrict__ y,
                                  const typename CT<T>::V* __restrict__ yd, const uint64_t* __restrict__ fmap,
                                  const __grid_constant__ FlipPhase ph) {
  const int64_t n = dim * CPR;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / CPR;
    int64_t p;
    double fr, fi;
    flip_coef(__ldg(fmap + row), ph, p, fr, fi);
    y[i] = cadd_mul<T>(y[i], fr, fi, yd[p * CPR + (i - row * CPR)]);
  }
}

template <typename W, typename R, typename T, int NV, int U, int MINB>
void launch_seg_t(Ctx& c, Ctx& t, const void* in, void* out, const double* scale, fx128* partial, int grid,
                  bool with_diag, unsigned long long* next_row) {
  HvParams<W> P;
  P.g = c.geom;
  if constexpr (sizeof(W) == 4) P.v = view32(t);
  else P.v = view64(t);
  using V = typename CT<T>::V;
  const R* gb = sizeof(R) == 4 ? reinterpret_cast<const R*>(c.binom32.p) : reinterpret_cast<const R*>(c.binom.p);
  k_hv_seg<W, R, T, NV, U, MINB><<<grid, kHvThreads, 0, c.stream>>>(P, static_cast<const V*>(in), static_cast<V*>(out),
                                                                    scale, partial, gb, with_diag ? 1 : 0, next_row);
}

// Variants of k_hv_seg (gather unroll U, CTAs per SM), as for k_hv; each runs one wave
// of sm_count x CTAs-per-SM CTAs (the grid does not change the results: the
// dot partials are exact fixed-point sums).
constexpr int kSegVariants = 5;
constexpr int kSegMinB[kSegVariants] = {4, 4, 3, 2, 2};

template <typename W, typename R, typename T, int NV>
void launch_seg_var(Ctx& c, Ctx& t, int var, const void* in, void* out, const double* scale, fx128* partial,
                    int grid, bool with_diag, unsigned long long* nr) {
  switch (var) {
    case 0: launch_seg_t<W, R, T, NV, 1, 4>(c, t, in, out, scale, partial, grid, with_diag, nr); return;
    case 1: launch_seg_t<W, R, T, NV, 2, 4>(c, t, in, out, scale, partial, grid, with_diag, nr); return;
    case 2: launch_seg_t<W, R, T, NV, 4, 3>(c, t, in, out, scale, partial, grid, with_diag, nr); return;
    case 3: launch_seg_t<W, R, T, NV, 4, 2>(c, t, in, out, scale, partial, grid, with_diag, nr); return;
    case 4: launch_seg_t<W, R, T, NV, 8, 2>(c, t, in, out, scale, partial, grid, with_diag, nr); return;
    default: break;
  }
  throw Error(FTLM_ERR_ARG, "bad H*V kernel variant");
}

template <typename W, typename R, typename T>
void launch_seg_nv(Ctx& c, Ctx& t, int var, const void* in, void* out, int nv, const double* scale, fx128* partial,
                   int grid, bool with_diag, unsigned long long* nr) {
  switch (nv) {
    case 1:
      if constexpr (sizeof(T) == 8) {
        launch_seg_var<W, R, T, 1>(c, t, var, in, out, scale, partial, grid, with_diag, nr);
        return;
      }
      break;
    case 2: launch_seg_var<W, R, T, 2>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 4: launch_seg_var<W, R, T, 4>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 8: launch_seg_var<W, R, T, 8>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 16: launch_seg_var<W, R, T, 16>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 32: launch_seg_var<W, R, T, 32>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 64: launch_seg_var<W, R, T, 64>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    case 128: launch_seg_var<W, R, T, 128>(c, t, var, in, out, scale, partial, grid, with_diag, nr); return;
    default: break;
  }
  throw Error(FTLM_ERR_ARG, "unsupported vectors per sweep: " + std::to_string(nv));
}

// Rows come from this sweep's counter (zeroed here, on the stream), or grid-stride.
void launch_seg(Ctx& c, Ctx& t, int var, const void* in, void* out, int nv, bool fp32, const double* scale,
                fx128* partial, int grid, bool with_diag, int counter_slot) {
  unsigned long long* nr = nullptr;
  if (c.seg_dynamic) {
    c.seg_counter.ensure(sizeof(unsigned long long) * 4);
    nr = c.seg_counter.as<unsigned long long>() + counter_slot;
    FTLM_CUDA(cudaMemsetAsync(nr, 0, sizeof(unsigned long long), c.stream));
  }
  if (c.wide) {
    if (fp32) launch_seg_nv<uint64_t, uint64_t, float>(c, t, var, in, out, nv, scale, partial, grid, with_diag, nr);
    else launch_seg_nv<uint64_t, uint64_t, double>(c, t, var, in, out, nv, scale, partial, grid, with_diag, nr);
  } else {
    if (fp32) launch_seg_nv<uint32_t, uint32_t, float>(c, t, var, in, out, nv, scale, partial, grid, with_diag, nr);
    else launch_seg_nv<uint32_t, uint32_t, double>(c, t, var, in, out, nv, scale, partial, grid, with_diag, nr);
  }
  FTLM_LAUNCH_CHECK();
}

// ---- wide stencil sweeps
// Stencil rows of a unit: more rows share more gathers in L1, fewer balance
// better. 4x4 (8,8), 64 vectors (1.3 M units of 8 rows and 64 chunks): 16 rows
// 11.3 ms per H*V, 8 rows 11.8, 32 rows 12.6; 6x3 (5,5), 16 vectors (130 k
// units): 1.65, 1.63, 1.80; 4x4 (4,4), 5 FP64 vectors (4 k): 0.109, 0.087, 0.154.
int stn_rows(int64_t dim, int cpr) { return dim * cpr >= (int64_t(1) << 27) ? 16 : 8; }

// Whether a row's hops are added in fours or in one chain. A chain rounds a growing sum at
// every hop, fours a quarter as often. The line lies where the error of H*V stays that of
// the kernels that shared a row among 32 / chunks groups of lanes (8 below 5 chunks) and so
// added sums as short. Relative to 64 bits, lane groups / chain / fours: 4x4 (3,4), FP32, 8
// vectors 4.84e-8 / 6.83e-8 / 4.95e-8, 16 5.06 / 6.83 / 4.95, 32 5.67 / 6.83 / 4.95, 64 6.83 / 6.83 /
// 4.95; FP64, 8 vectors 1.02e-16 / 1.33e-16 / 1.02e-16. Per H*V, chain / fours: 6x3 (5,5) 16 FP32
// vectors 1.64 / 1.70 ms, 4x4 (4,4) 5 FP64 0.084 / 0.088, 4x4 (6,6) 2 FP32 0.283 / 0.278, 4x4 (5,5)
// 128 2.32 / 2.5. Narrower sweeps all add in the same order, so a vector's product does
// not depend on how many others there are.
bool stn_fours(int nv, bool fp32) { return (fp32 ? nv / 2 : nv) < 32; }

template <typename T>
StnJob<T> stn_job(Ctx& t, const void* in, void* out, bool with_diag, const StnPanels& pan, int rows) {
  StnJob<T> j;
  j.in = static_cast<const typename CT<T>::V*>(in);
  j.out = static_cast<typename CT<T>::V*>(out);
  j.diag = with_diag ? t.stn_diag.as<T>() : nullptr;
  j.srow = t.stn_row.as<int2>();
  j.ent = t.stn_ent4.as<uint4>();
  j.coef = t.stn_coef.as<typename CoefT<T>::C>();
  j.cls = t.stn_cls.as<StnClass>();
  int64_t units = 0;
  for (size_t k = 0; k + 1 < t.stn_classes.size(); k += 2)
    units += stn_chunks(t.stn_classes[k + 1], rows) * pan.count(t.stn_classes[k]);
  j.units = static_cast<int32_t>(units);
  return j;
}

struct StnSweep {  // the two sweeps of one H*V: block order (with the diagonal), flipped order
  Ctx* t[2];
  const void* in[2];
  void* out[2];
  int n;
};

template <typename T, int LPL, int U, int NT, int MINB, bool FOURS>
int launch_stn_t(Ctx& c, const StnSweep& w, int nv, const double* scale, fx128* partial, unsigned int* counter) {
  StnJobs<T> P;
  P.njobs = w.n;
  P.nv = nv;
  P.pan = stn_panels(nv / CT<T>::VPL, 32 * LPL);
  P.rows = stn_rows(c.blk.dim, nv / CT<T>::VPL);
  for (int k = 0; k < kStnCoefs; ++k) {  // shift 0 (phase 1), ratio 1
    const double sg = k & 1 ? -1.0 : 1.0;
    P.c0[k].x = static_cast<T>(sg * c.geom.amp_re[k / 2]);
    P.c0[k].y = static_cast<T>(sg * c.geom.amp_im[k / 2]);
  }
  int64_t units = 0;
  for (int i = 0; i < w.n; ++i) {
    P.j[i] = stn_job<T>(*w.t[i], w.in[i], w.out[i], i == 0, P.pan, P.rows);
    units += P.j[i].units;
  }
  const int64_t items = (units + NT / 32 - 1) / (NT / 32);
  const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(items, int64_t(c.sm_count) * MINB)));
  // the rest of the SM's 228 KB serves as L1, where most of the gather reuse is
  constexpr size_t kSmem = sizeof(fx128) * NT / 32 * kStnSlots + 2048;
  constexpr int kCarve = static_cast<int>((kSmem * MINB * 100 + 228 * 1024 - 1) / (228 * 1024));
  FTLM_CUDA(cudaFuncSetAttribute(k_hv_stn<T, LPL, U, NT, MINB, FOURS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 kCarve));
  k_hv_stn<T, LPL, U, NT, MINB, FOURS><<<grid, NT, 0, c.stream>>>(P, scale, partial, counter);
  return grid;
}

// Variants: chunks per lane (more amortise the entry load, fewer leave
// registers for warps), gathers in flight, CTA shape. All sum a row's hops in
// the same order, and the same dot terms.
template <typename T, bool FOURS>
int launch_stn_var(Ctx& c, int var, const StnSweep& w, int nv, const double* scale, fx128* partial, unsigned int* nr) {
  switch (var) {
    case 0: return launch_stn_t<T, 2, 4, 256, 3, FOURS>(c, w, nv, scale, partial, nr);
    case 1: return launch_stn_t<T, 2, 8, 256, 2, FOURS>(c, w, nv, scale, partial, nr);
    case 2: return launch_stn_t<T, 1, 8, 256, 3, FOURS>(c, w, nv, scale, partial, nr);
    case 3: return launch_stn_t<T, 1, 4, 256, 4, FOURS>(c, w, nv, scale, partial, nr);
    case 4: return launch_stn_t<T, 2, 8, 256, 3, FOURS>(c, w, nv, scale, partial, nr);
    default: break;
  }
  throw Error(FTLM_ERR_ARG, "bad H*V kernel variant");
}

// Returns the grid, which is the number of rows of dot partials.
int launch_stn(Ctx& c, int var, const StnSweep& w, int nv, bool fp32, const double* scale, fx128* partial) {
  unsigned int* nr = nullptr;
  if (c.seg_dynamic) {
    c.seg_counter.ensure(sizeof(unsigned long long) * 4);
    nr = c.seg_counter.as<unsigned int>();
    FTLM_CUDA(cudaMemsetAsync(nr, 0, sizeof(unsigned int), c.stream));
  }
  auto run = [&](auto fours) {
    constexpr bool F = decltype(fours)::value;
    return fp32 ? launch_stn_var<float, F>(c, var, w, nv, scale, partial, nr)
                : launch_stn_var<double, F>(c, var, w, nv, scale, partial, nr);
  };
  const int grid = stn_fours(nv, fp32) ? run(std::true_type()) : run(std::false_type());
  FTLM_LAUNCH_CHECK();
  return grid;
}

int seg_grid(const Ctx& c, int var) {
  const int64_t by_rows = (c.blk.dim + kHvWarps - 1) / kHvWarps;
  const int64_t cap = static_cast<int64_t>(c.sm_count) * kSegMinB[var];
  return static_cast<int>(std::max<int64_t>(1, std::min(by_rows, cap)));
}

// The flipped tables: the context itself when N_up == N_down, else a
// companion context holding sector (N_down, N_up) of the same model.
Ctx& flipped_tables(Ctx& c) {
  if (c.sec.n_up == c.sec.n_dn) return c;
  if (!c.flipped) {
    c.flipped.reset(new Ctx());
    Ctx& f = *c.flipped;
    f.model = c.model;
    f.opts = c.opts;
    f.geom = c.geom;
    f.wide = c.wide;
    f.device = c.device;
    f.sm_count = c.sm_count;
    f.stream = c.stream;
    for (DBuf* b : table_bufs(f)) b->arena = &c.arena;
    f.binom = c.binom;  // shared, owned by c
    f.binom32 = c.binom32;
  }
  Ctx& f = *c.flipped;
  if (f.sec.n_up != c.sec.n_dn || f.sec.n_dn != c.sec.n_up) {
    sector_prepare(f, c.sec.n_dn, c.sec.n_up);
    c.prof.kernel_launches += f.prof.kernel_launches;
    f.prof.kernel_launches = 0;
  }
  block_prepare(f, c.blk.mx, c.blk.my);
  if (f.blk.dim != c.blk.dim) throw Error(FTLM_ERR_INTERNAL, "spin-flipped block has another dimension");
  return f;
}

// ---- entries of the wide sweeps

// Rounded-up entry counts (multiples of 4) for the row offsets.
__global__ void k_stn_round(const int64_t* __restrict__ rp, int64_t rows, int32_t* __restrict__ counts) {
  for (int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; r < rows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x)
    counts[r] = static_cast<int32_t>((rp[r + 1] - rp[r] + 3) & ~int64_t(3));
}

// The wide sweeps' entries from the packed ones, same order.
__global__ void k_stn_wide(int64_t rows, const int64_t* __restrict__ rp, const uint32_t* __restrict__ ent,
                           const uint8_t* __restrict__ row_deg, const __grid_constant__ StnRatios R,
                           const int64_t* __restrict__ rp4, int2* __restrict__ srow, uint32_t* __restrict__ out) {
  for (int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; r < rows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t h0 = rp[r];
    const int n = static_cast<int>(rp[r + 1] - h0), ds = row_deg[r];
    uint32_t* o = out + rp4[r];
    for (int k = 0; k < n; ++k) {
      const uint32_t e = ent[h0 + k];
      const int dt = static_cast<int>(e >> 26) + 1;
      uint32_t ratio = 0;
      while (R.num[ratio] * ds != R.den[ratio] * dt) ++ratio;
      const uint32_t id = ((ratio * 64 + ((e >> 20) & 63u)) * 8 + ((e >> 16) & 7u)) * 2 + ((e >> 19) & 1u);
      o[k] = (e & 0xFFFFu) | (id << 16);
    }
    srow[r] = make_int2(static_cast<int>(rp4[r] / 4), n);
  }
}

__global__ void k_stn_coef(const __grid_constant__ Geom g, const __grid_constant__ FlipPhase ph,
                           const __grid_constant__ StnRatios R, float2* __restrict__ c32, double2* __restrict__ c64) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= R.n * 64 * kStnCoefs) return;
  const int dir = (id >> 1) & 7, h = (id >> 4) & 63, ratio = id >> 10;
  double re = 0.0, im = 0.0;
  if (h < g.n) {
    const double q = g.sqrt_deg[R.num[ratio]] * (1.0 / g.sqrt_deg[R.den[ratio]]);
    re = (g.amp_re[dir] * ph.re[h] - g.amp_im[dir] * ph.im[h]) * q;
    im = (g.amp_re[dir] * ph.im[h] + g.amp_im[dir] * ph.re[h]) * q;
    if (id & 1) {
      re = -re;
      im = -im;
    }
  }
  if (c32) c32[id] = make_float2(static_cast<float>(re), static_cast<float>(im));
  else c64[id] = make_double2(re, im);
}

// Stabiliser size of every stencil row.
__global__ void k_stn_deg(int nclass, const int64_t* __restrict__ crb, int64_t c_dn,
                          const uint32_t* __restrict__ act_list, const uint64_t* __restrict__ dtab, int64_t rows,
                          uint8_t* __restrict__ deg) {
  for (int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; r < rows;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int c = 0;
    while (c + 1 < nclass && crb[c + 1] <= r) ++c;
    const int64_t base = static_cast<int64_t>(c - 1) * c_dn;
    deg[r] = c == 0 ? 1 : static_cast<uint8_t>((dtab[base + act_list[base + (r - crb[c])]] >> 48) & 0xFF);
  }
}

// The distinct values of deg_t / deg_s: orbit stabilisers are subgroups, so
// both divide the number of sites. False when there are more than the entry
// format numbers (a lattice with three prime factors such as 60 sites).
bool stn_ratios(int n, StnRatios& R) {
  R.n = 0;
  for (int dt = 1; dt <= n; ++dt)
    for (int ds = 1; ds <= n; ++ds) {
      if (n % dt || n % ds) continue;
      bool known = false;
      for (int k = 0; k < R.n; ++k) known = known || R.num[k] * ds == R.den[k] * dt;
      if (known) continue;
      if (R.n == kStnMaxRatios) return false;
      R.num[R.n] = static_cast<uint8_t>(dt);
      R.den[R.n] = static_cast<uint8_t>(ds);
      ++R.n;
    }
  return true;
}

bool stn_wide_build(Ctx& c, Ctx& t, int64_t rows) {
  StnRatios R;
  if (!stn_ratios(c.geom.n, R)) return false;
  const int grid = grid_rows(rows, 128);
  k_stn_round<<<grid, 128, 0, c.stream>>>(t.stn_rp.as<int64_t>(), rows, t.stn_cnt.as<int32_t>());
  t.stn_rp4.ensure(sizeof(int64_t) * (rows + 1));
  const int64_t total = scan_excl_i32_to_i64(c, t.stn_cnt.as<int32_t>(), t.stn_rp4.as<int64_t>(), rows);
  t.stn_ent4.ensure(sizeof(uint32_t) * (total + 8));  // sweeps read up to two quads past a row
  t.stn_row.ensure(sizeof(int2) * std::max<int64_t>(rows, 1));
  t.stn_deg.ensure(std::max<int64_t>(rows, 1));
  k_stn_deg<<<grid, 128, 0, c.stream>>>(t.sec.nclass, t.stn_crb.as<int64_t>(), t.sec.c_dn, t.blk.act_list.as<uint32_t>(),
                                        t.blk.dtab.as<uint64_t>(), rows, t.stn_deg.as<uint8_t>());
  k_stn_wide<<<grid, 128, 0, c.stream>>>(rows, t.stn_rp.as<int64_t>(), t.stn_ent.as<uint32_t>(), t.stn_deg.as<uint8_t>(),
                                         R, t.stn_rp4.as<int64_t>(), t.stn_row.as<int2>(), t.stn_ent4.as<uint32_t>());
  const bool fp32 = c.opts.precision == FTLM_PREC_MIXED;
  t.stn_coef.ensure((fp32 ? sizeof(float2) : sizeof(double2)) * R.n * 64 * kStnCoefs);
  k_stn_coef<<<R.n * 8, 128, 0, c.stream>>>(c.geom, flip_phase(t), R, fp32 ? t.stn_coef.as<float2>() : nullptr,
                                            fp32 ? nullptr : t.stn_coef.as<double2>());
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 4;
  return true;
}

// Position of every row of the block in the sweeps' order, S segments a group.
__global__ void k_stn_pos(const StnClass* __restrict__ cls, int ncls, int S, int64_t dim,
                          const int32_t* __restrict__ seg_ur, const int64_t* __restrict__ aoff,
                          uint32_t* __restrict__ pos) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < dim;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int c = 0;
    while (c + 1 < ncls && cls[c + 1].base <= i) ++c;
    const StnClass C = cls[c];
    const int64_t at = i - C.base, full = static_cast<int64_t>(S) * C.rows;
    const int g = static_cast<int>(at / full);
    const uint32_t in = static_cast<uint32_t>(at - g * full), nsg = min(S, C.nseg - g * S), a = in / nsg;
    pos[aoff[seg_ur[C.first + g * S + (in - a * nsg)]] + a] = static_cast<uint32_t>(i);
  }
}

// Class stencils of the prepared block of tables t (its own sector and
// block); false when a class has more than kStencilMaxRows rows.
template <typename W>
bool stencil_build_t(Ctx& c, Ctx& t) {
  const SectorTables& S = t.sec;
  const BlockTables& B = t.blk;
  if (S.c_dn > kStencilMaxRows) return false;
  std::vector<int64_t> crb(S.nclass + 1, 0);
  for (int k = 0; k < S.nclass; ++k) crb[k + 1] = crb[k] + (k == 0 ? S.c_dn : B.cls_nact[k]);
  const int64_t rows = crb[S.nclass];
  t.stn_crb.ensure(sizeof(int64_t) * (S.nclass + 1));
  FTLM_CUDA(cudaMemcpyAsync(t.stn_crb.p, crb.data(), sizeof(int64_t) * crb.size(), cudaMemcpyHostToDevice, c.stream));
  t.stn_cnt.ensure(sizeof(int32_t) * std::max<int64_t>(rows, 1));
  t.stn_rp.ensure(sizeof(int64_t) * (rows + 1));
  const int grid = grid_rows(rows, 128);
  k_stencil<W><<<grid, 128, 0, c.stream>>>(0, c.geom, S.nclass, t.stn_crb.as<int64_t>(), S.c_dn,
                                           B.act_list.as<uint32_t>(), B.dtab.as<uint64_t>(), S.dns.as<W>(),
                                           c.binom.as<uint64_t>(), rows, t.stn_cnt.as<int32_t>(), nullptr, nullptr);
  FTLM_LAUNCH_CHECK();
  const int64_t total = scan_excl_i32_to_i64(c, t.stn_cnt.as<int32_t>(), t.stn_rp.as<int64_t>(), rows);
  if (total > 0x7fffffffLL) return false;  // the sweeps keep 32-bit entry offsets
  FTLM_CUDA(cudaMemcpyAsync(t.stn_rp.as<int64_t>() + rows, &total, sizeof(int64_t), cudaMemcpyHostToDevice,
                            c.stream));
  t.stn_ent.ensure(sizeof(uint32_t) * std::max<int64_t>(total, 1));
  k_stencil<W><<<grid, 128, 0, c.stream>>>(1, c.geom, S.nclass, t.stn_crb.as<int64_t>(), S.c_dn,
                                           B.act_list.as<uint32_t>(), B.dtab.as<uint64_t>(), S.dns.as<W>(),
                                           c.binom.as<uint64_t>(), rows, nullptr, t.stn_rp.as<int64_t>(),
                                           t.stn_ent.as<uint32_t>());
  if (!stn_wide_build(c, t, rows)) return false;
  // segments by class, and the classes that have rows in this block
  std::vector<int32_t> seg(S.nur);
  std::vector<int64_t> first(S.nclass + 1, 0);
  for (int64_t u = 0; u < S.nur; ++u) ++first[S.h_ur_class[u] + 1];
  for (int k = 0; k < S.nclass; ++k) first[k + 1] += first[k];
  std::vector<int64_t> at(first.begin(), first.end() - 1);
  for (int64_t u = 0; u < S.nur; ++u) seg[at[S.h_ur_class[u]]++] = static_cast<int32_t>(u);
  std::vector<StnClass> cls;
  int64_t base = 0;
  t.stn_classes.clear();
  for (int k = 0; k < S.nclass; ++k) {
    const int64_t nseg = first[k + 1] - first[k], nrow = crb[k + 1] - crb[k];
    if (nseg == 0 || nrow == 0) continue;
    cls.push_back({static_cast<int32_t>(nseg), static_cast<int32_t>(nrow), k == 0 ? 1 : 0,
                   static_cast<int32_t>(first[k]), crb[k], base});
    base += nseg * nrow;
    t.stn_classes.push_back(nseg);
    t.stn_classes.push_back(nrow);
  }
  t.stn_seg.ensure(sizeof(int32_t) * std::max<int64_t>(S.nur, 1));
  t.stn_cls.ensure(sizeof(StnClass) * std::max<size_t>(cls.size(), 1));
  FTLM_CUDA(cudaMemcpyAsync(t.stn_seg.p, seg.data(), sizeof(int32_t) * seg.size(), cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaMemcpyAsync(t.stn_cls.p, cls.data(), sizeof(StnClass) * cls.size(), cudaMemcpyHostToDevice, c.stream));
  if (base != B.dim) throw Error(FTLM_ERR_INTERNAL, "stencil classes do not cover the block");
  FTLM_LAUNCH_CHECK();
  FTLM_CUDA(cudaStreamSynchronize(c.stream));
  c.prof.kernel_launches += 5;
  return true;
}

// Diagonal energy of every row of the prepared block, in the sweeps' type and order.
template <typename W, typename T>
__global__ void k_row_diag(const __grid_constant__ HvParams<W> P, const uint32_t* __restrict__ pos,
                           T* __restrict__ diag) {
  const BlockView<W>& v = P.v;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < v.dim;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    diag[pos[i]] = static_cast<T>(diag_energy(v.ur_bits[v.row_meta[i] & 0x3FFFFFFu], v.row_dn[i], P.g));
}

template <typename W>
void row_diag_build(Ctx& c) {
  HvParams<W> P;
  P.g = c.geom;
  if constexpr (sizeof(W) == 4) P.v = view32(c);
  else P.v = view64(c);
  const int64_t D = c.blk.dim;
  if (c.opts.precision == FTLM_PREC_MIXED) {
    c.stn_diag.ensure(sizeof(float) * D);
    k_row_diag<W, float><<<grid_rows(D, 256), 256, 0, c.stream>>>(P, c.stn_pos.as<uint32_t>(), c.stn_diag.as<float>());
  } else {
    c.stn_diag.ensure(sizeof(double) * D);
    k_row_diag<W, double><<<grid_rows(D, 256), 256, 0, c.stream>>>(P, c.stn_pos.as<uint32_t>(), c.stn_diag.as<double>());
  }
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
}

// Stencils of tables t for its prepared block, built once per (sector
// generation, block).
void stencil_prepare(Ctx& c, Ctx& t) {
  const int64_t key[3] = {t.sec_gen, t.blk.mx, t.blk.my};
  if (std::memcmp(key, t.stn_for, sizeof key) == 0) return;
  t.stn_pos_seg = 0;
  t.stn_ok = c.wide ? stencil_build_t<uint64_t>(c, t) : stencil_build_t<uint32_t>(c, t);
  std::memcpy(t.stn_for, key, sizeof key);
}

// Positions of the block's rows (and the diagonal in that order) for groups of S segments.
void order_prepare(Ctx& c, Ctx& t, int S) {
  if (t.stn_pos_seg == S) return;
  const int64_t D = t.blk.dim;
  t.stn_pos.ensure(sizeof(uint32_t) * std::max<int64_t>(D, 1));
  k_stn_pos<<<grid_rows(D, 256), 256, 0, c.stream>>>(t.stn_cls.as<StnClass>(), static_cast<int>(t.stn_classes.size() / 2),
                                                     S, D, t.stn_seg.as<int32_t>(), t.blk.aoff.as<int64_t>(),
                                                     t.stn_pos.as<uint32_t>());
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
  if (&t == &c) {
    if (c.wide) row_diag_build<uint64_t>(c);
    else row_diag_build<uint32_t>(c);
  }
  t.stn_pos_seg = S;
}

template <typename W>
void flip_map_build_t(Ctx& c, Ctx& f) {
  HvParams<W> P;
  P.g = c.geom;
  BlockView<W> vd;
  if constexpr (sizeof(W) == 4) {
    P.v = view32(c);
    vd = view32(f);
  } else {
    P.v = view64(c);
    vd = view64(f);
  }
  const int64_t D = c.blk.dim;
  c.flip_map.ensure(sizeof(uint64_t) * std::max<int64_t>(D, 1) + 64);
  int* bad = reinterpret_cast<int*>(c.flip_map.as<uint64_t>() + D);
  FTLM_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), c.stream));
  const uint32_t* pos = c.split_wide ? c.stn_pos.as<uint32_t>() : nullptr;
  const uint32_t* pos_d = c.split_wide ? f.stn_pos.as<uint32_t>() : nullptr;
  k_flip_map<W><<<grid_rows(D, 128), 128, 0, c.stream>>>(P, vd, c.binom.as<uint64_t>(), pos, pos_d,
                                                         c.flip_map.as<uint64_t>(), bad);
  FTLM_LAUNCH_CHECK();
  int hbad = 0;
  FTLM_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  FTLM_CUDA(cudaStreamSynchronize(c.stream));
  c.prof.kernel_launches += 1;
  if (hbad) throw Error(FTLM_ERR_INTERNAL, "spin flip: " + std::to_string(hbad) + " rows without an image");
}

}  // namespace

FlipPhase flip_phase(const Ctx& c) {
  FlipPhase ph;
  std::memcpy(ph.re, c.blk.phase_re, sizeof ph.re);
  std::memcpy(ph.im, c.blk.phase_im, sizeof ph.im);
  return ph;
}

void split_order(Ctx& c, int nv, bool fp32) {
  Ctx& f = c.sec.n_up == c.sec.n_dn ? c : *c.flipped;
  const int S = c.split_wide ? stn_group(fp32 ? nv / 2 : nv) : 0;
  if (S) {
    order_prepare(c, c, S);
    if (&f != &c) order_prepare(c, f, S);
  }
  const int key[5] = {c.sec.n_up, c.sec.n_dn, c.blk.mx, c.blk.my, S};
  if (std::memcmp(key, c.flip_for, sizeof key) == 0 && c.flip_gen == c.sec_gen) return;
  if (c.wide) flip_map_build_t<uint64_t>(c, f);
  else flip_map_build_t<uint32_t>(c, f);
  std::memcpy(c.flip_for, key, sizeof key);
  c.flip_gen = c.sec_gen;
}

bool split_stencils(const Ctx& c) {
  StnRatios R;
  return c.split_stencil && std::max(c.sec.c_up, c.sec.c_dn) <= kStencilMaxRows && stn_ratios(c.geom.n, R);
}

bool split_prepare(Ctx& c, int nv, bool fp32) {
  const int64_t D = c.blk.dim;
  if (D <= 0) return false;
  if (D > 0x7fffffffLL) return false;  // the flip map keeps 32-bit rows
  // memory: two extra vector arrays (flipped x and y), the 8-byte map, and per
  // row two positions and the diagonal
  const size_t esize = fp32 ? 8 : 16;
  // the on-the-fly sweeps take powers of two; the stencil ones, which nearly
  // every lattice takes, as many as there are
  int pow2 = fp32 ? 2 : 1;
  while (pow2 < nv) pow2 <<= 1;
  const size_t vec = static_cast<size_t>(D) * (split_stencils(c) ? nv : pow2) * esize;
  const bool two = c.sec.n_up != c.sec.n_dn;
  const size_t need = 2 * vec + (sizeof(uint64_t) + (two ? 2 : 1) * sizeof(uint32_t) + esize / 2) * D;
  const size_t have = c.vec_xd.cap + c.vec_yd.cap + c.flip_map.cap + c.stn_pos.cap + c.stn_diag.cap +
                      (two && c.flipped ? c.flipped->stn_pos.cap : 0);
  if (need > have) {  // keep 2 GiB headroom
    size_t free_b = 0, total_b = 0;
    FTLM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    if (need + (size_t(2) << 30) > free_b + have) return false;
  }
  Ctx& f = flipped_tables(c);
  c.split_wide = false;
  if (c.split_stencil) {
    stencil_prepare(c, c);
    if (&f != &c) stencil_prepare(c, f);
    c.split_wide = c.stn_ok && f.stn_ok;
  }
  split_order(c, nv, fp32);
  const size_t used = static_cast<size_t>(D) * (c.split_wide ? nv : pow2) * esize;
  c.vec_xd.ensure(used + kSweepPad);
  c.vec_yd.ensure(used);
  return true;
}

int seg_variant(Ctx& c, const StnSweep& both, int nv, bool fp32, const double* scale, fx128* partial) {
  if (c.hv_forced >= 0 && c.hv_forced < kSegVariants) return c.hv_forced;
  int width = 1;  // the wide sweeps take any number of vectors: one measurement per power of two
  while (width < nv) width <<= 1;
  const bool fours = c.split_wide && stn_fours(nv, fp32);
  const uint64_t key = static_cast<uint64_t>((c.wide ? 1 : 0) | (fours ? 2 : 0) | 4 | (c.split_wide ? 8 : 0)) |
                       (static_cast<uint64_t>(fp32 ? 1 : 0) << 4) |
                       (static_cast<uint64_t>(width) << 8) |
                       (static_cast<uint64_t>(hv_size_class(c.blk.dim)) << 20) |
                       (static_cast<uint64_t>(c.device) << 32);
  int best = -1;
  if (hv_tuned_lookup(c, key, best)) return best;
  if (c.blk.dim < (1 << 15)) return 1;  // too small to measure
  cudaEvent_t e0, e1;
  FTLM_CUDA(cudaEventCreate(&e0));
  FTLM_CUDA(cudaEventCreate(&e1));
  // best of several single-launch timings per variant, variants interleaved: of 3
  // after a warm run, or of 2 for the stencil sweeps, whose times repeat to 1% (a
  // few steps of 2 vectors cost less than 20 launches). Sums of fours (stn_fours) take
  // more registers: of their variants 1, with 128 registers, or 2, with one chunk a lane,
  // was the fastest on every block (us per H*V, variants 0-4: 5x3 (12,5) 2 FP32 vectors 48
  // 37 35 44 48, 4x3 (5,7) 4 FP64 43 31 32 35 52, 4x4 (12,5) 3 FP32 96 91 85 103 99, 6x3
  // (14,14) 43 FP32 527 487 564 590 554). Only those two are timed, warm, by three launches
  // of both sweeps with their dot products: cold single launches of one sweep picked the
  // slower on 4x4 (12,5) and 5x3 (3,9) (91 for 85 us, 47 for 43) and variant 3 on 5x3 (12,5).
  const bool wide = c.split_wide;
  auto timed = [&](int v) { return !fours || v == 1 || v == 2; };
  const void* in = both.in[0];
  void* out = both.out[0];
  const StnSweep one{{&c, nullptr}, {in, nullptr}, {out, nullptr}, 1};
  auto run = [&](int v) {
    if (fours) launch_stn(c, v, both, nv, fp32, scale, partial);
    else if (wide) launch_stn(c, v, one, nv, fp32, nullptr, nullptr);
    else launch_seg(c, c, v, in, out, nv, fp32, nullptr, nullptr, seg_grid(c, v), true, 0);
  };
  float best_ms[kSegVariants];
  for (int v = 0; v < kSegVariants; ++v) {
    best_ms[v] = 1e30f;
    if (!wide) run(v);  // warm
  }
  for (int rep = 0; rep < (fours ? 1 : wide ? 2 : 3); ++rep)
    for (int v = 0; v < kSegVariants; ++v) {
      if (!timed(v)) continue;
      if (fours) run(v);
      FTLM_CUDA(cudaEventRecord(e0, c.stream));
      for (int k = 0; k < (fours ? 3 : 1); ++k) run(v);
      FTLM_CUDA(cudaEventRecord(e1, c.stream));
      FTLM_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      FTLM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best_ms[v] = std::min(best_ms[v], ms);
    }
  best = 0;
  for (int v = 1; v < kSegVariants; ++v)
    if (best_ms[v] < best_ms[best]) best = v;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  c.prof.tune_runs += 1;
  c.prof.kernel_launches += fours ? 4 * 2 : wide ? 2 * kSegVariants : 4 * kSegVariants;
  hv_tuned_store(c, key, best);
  return best;
}

int hv_apply_split(Ctx& c, const void* in, const void* in_d, void* out, void* out_d, int nv, bool fp32,
                   const double* scale, fx128* partial) {
  Ctx& f = flipped_tables(c);
  const StnSweep both{{&c, &f}, {in, in_d}, {out, out_d}, 2};
  const int var = seg_variant(c, both, nv, fp32, scale, partial);
  c.prof.hv_variant = var;
  if (c.split_wide) {
    const int rows = launch_stn(c, var, both, nv, fp32, scale, partial);
    c.prof.kernel_launches += 1;
    return rows;
  }
  const int grid = seg_grid(c, var);
  // flipped sweep first: its partials follow this block's in the array
  launch_seg(c, f, var, in_d, out_d, nv, fp32, scale, partial ? partial + static_cast<int64_t>(grid) * nv : nullptr,
             grid, false, 1);
  launch_seg(c, c, var, in, out, nv, fp32, scale, partial, grid, true, 0);
  c.prof.kernel_launches += 2;
  return 2 * grid;
}

// vec[pos[q]][v] = raw[q - row0][v], zero for v >= nvec (pos null: q), for `rows`
// rows from row0, one thread per element.
template <typename T2>
__global__ void k_vectors_in(int64_t row0, int64_t rows, int nvec, int NV, const uint32_t* __restrict__ pos,
                             const double2* __restrict__ raw, T2* __restrict__ vec) {
  const int64_t n = rows * NV;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / NV, q = row0 + row;
    const int v = static_cast<int>(i - row * NV);
    T2 z{0, 0};
    if (v < nvec) {
      const double2 r = raw[row * nvec + v];
      z.x = static_cast<decltype(z.x)>(r.x);
      z.y = static_cast<decltype(z.x)>(r.y);
    }
    vec[(pos ? pos[q] : q) * NV + v] = z;
  }
}

template <typename T2>
__global__ void k_vectors_out(int64_t row0, int64_t rows, int nvec, int NV, const uint32_t* __restrict__ pos,
                              const T2* __restrict__ vec, double2* __restrict__ raw) {
  const int64_t n = rows * nvec;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / nvec, q = row0 + row;
    const T2 z = vec[(pos ? pos[q] : q) * NV + (i - row * nvec)];
    raw[i] = make_double2(z.x, z.y);
  }
}

// f(first row, rows) for the chunks of a block.
template <typename F>
void convert_chunks(Ctx& c, int nvec, F&& f) {
  const int64_t D = c.blk.dim;
  int64_t step = std::min(D, std::max<int64_t>(1, kConvertChunk / nvec));
  while (true) {
    try {
      c.host_start.ensure(sizeof(double2) * static_cast<size_t>(step) * nvec);
      break;
    } catch (const Error&) {  // beside vectors that fill the memory: smaller chunks
      if (step * nvec <= kConvertLeast) throw;
      cudaGetLastError();
      step = (step + 1) / 2;
    }
  }
  for (int64_t r = 0; r < D; r += step) f(r, std::min(step, D - r));
}

void vectors_from_host(Ctx& c, int nvec, int NV, bool fp32, const double* in, void* vec) {
  convert_chunks(c, nvec, [&](int64_t r, int64_t rows) {
    double2* raw = c.host_start.as<double2>();
    FTLM_CUDA(cudaMemcpyAsync(raw, in + 2 * r * nvec, sizeof(double2) * rows * nvec, cudaMemcpyHostToDevice, c.stream));
    const int grid = grid_rows(rows * NV, 256);
    if (fp32) k_vectors_in<<<grid, 256, 0, c.stream>>>(r, rows, nvec, NV, sweep_pos(c), raw, static_cast<float2*>(vec));
    else k_vectors_in<<<grid, 256, 0, c.stream>>>(r, rows, nvec, NV, sweep_pos(c), raw, static_cast<double2*>(vec));
    FTLM_LAUNCH_CHECK();
    c.prof.kernel_launches += 1;
  });
}

void vectors_to_host(Ctx& c, int nvec, int NV, bool fp32, const void* vec, double* out) {
  convert_chunks(c, nvec, [&](int64_t r, int64_t rows) {
    double2* raw = c.host_start.as<double2>();
    const int grid = grid_rows(rows * nvec, 256);
    if (fp32)
      k_vectors_out<<<grid, 256, 0, c.stream>>>(r, rows, nvec, NV, sweep_pos(c), static_cast<const float2*>(vec), raw);
    else
      k_vectors_out<<<grid, 256, 0, c.stream>>>(r, rows, nvec, NV, sweep_pos(c), static_cast<const double2*>(vec), raw);
    FTLM_LAUNCH_CHECK();
    FTLM_CUDA(cudaMemcpyAsync(out + 2 * r * nvec, raw, sizeof(double2) * rows * nvec, cudaMemcpyDeviceToHost, c.stream));
    c.prof.kernel_launches += 1;
  });
}

const uint32_t* sweep_pos(const Ctx& c) { return c.split_active && c.split_wide ? c.stn_pos.as<uint32_t>() : nullptr; }

int hv_split_max_grid(const Ctx& c) { return 2 * c.sm_count * 4; }

void flip_scatter(Ctx& c, const void* x, void* xd, int nv, bool fp32) {
  const int64_t D = c.blk.dim;
  const int CPR = fp32 ? nv / 2 : nv;
  const int grid = grid_rows(D * CPR, 256);
  if (fp32)
    k_flip_scatter<float><<<grid, 256, 0, c.stream>>>(D, CPR, static_cast<const float4*>(x), static_cast<float4*>(xd),
                                                      c.flip_map.as<uint64_t>(), flip_phase(c));
  else
    k_flip_scatter<double><<<grid, 256, 0, c.stream>>>(D, CPR, static_cast<const double2*>(x),
                                                       static_cast<double2*>(xd), c.flip_map.as<uint64_t>(),
                                                       flip_phase(c));
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
}

void flip_gather_add(Ctx& c, void* y, const void* yd, int nv, bool fp32) {
  const int64_t D = c.blk.dim;
  const int CPR = fp32 ? nv / 2 : nv;
  const int grid = grid_rows(D * CPR, 256);
  if (fp32)
    k_flip_gather_add<float><<<grid, 256, 0, c.stream>>>(D, CPR, static_cast<float4*>(y), static_cast<const float4*>(yd),
                                                         c.flip_map.as<uint64_t>(), flip_phase(c));
  else
    k_flip_gather_add<double><<<grid, 256, 0, c.stream>>>(D, CPR, static_cast<double2*>(y),
                                                          static_cast<const double2*>(yd), c.flip_map.as<uint64_t>(),
                                                          flip_phase(c));
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
}

}  // namespace ftlm
