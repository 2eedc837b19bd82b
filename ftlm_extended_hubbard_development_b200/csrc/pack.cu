// Small sectors: the tables of all momentum blocks in one launch, and the
// rows of many blocks (dense matrices, small-block Lanczos entries) in one
// launch each.
//
// A curve on a small lattice visits hundreds of blocks of a few to a few
// thousand rows. Building each block's tables with its own scans costs a
// dozen launches and four host round trips per block, and a row builder with
// one thread per row leaves the GPU idle (50 us per block on 4x2 and 3x3, most
// of it a chain of dependent table lookups). Here one CTA per momentum builds
// that block's tables (activity, lookup entries, row offsets, row list) with
// no host round trip, and a warp per row resolves 32 candidate hops at once.
// Rows and matrices per curve: 4x2 35 ms in 1240 launches -> 1.0 in 153, 3x3
// 66 ms -> 1.6.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ftlm_internal.h"
#include "hv_common.cuh"

namespace ftlm {

namespace {

constexpr int kPackThreads = 512;
constexpr int kPackWarps = kPackThreads / 32;
constexpr int64_t kPackMaxWords = int64_t(1) << 22;  // class words x momenta
constexpr int64_t kPackMaxRows = int64_t(1) << 20;   // rows of all blocks

// Exclusive CTA scan of one int per thread; total to every thread.
__device__ __forceinline__ int pack_scan(int v, int* warp_tot, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // warp_tot of the previous scan is no longer read
  if (lane == 31) warp_tot[wid] = inc;
  __syncthreads();
  int pre = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kPackWarps; ++w) {
    const int t = warp_tot[w];
    if (w < wid) pre += t;
    all += t;
  }
  total = all;
  return pre + inc - v;
}

struct PackArgs {
  int nclass;
  int64_t c_dn, nur;
  const int32_t* canon;
  const uint64_t* d_stab;
  const uint64_t* d_chi;
  const uint32_t* d_star;
  const uint16_t* d_hs;
  const uint16_t* ur_class;
  const int64_t* row0;  // [n_k + 1] first row of each block in the row arrays
  int32_t* act;         // [n_k][tot]
  uint32_t* act_list;   // [n_k][tot]
  uint64_t* dtab;       // [n_k][tot]
  int64_t* aoff;        // [n_k][nur + 1]
  int32_t* nact;        // [n_k][nclass]
  int64_t* dims;        // [n_k]
  uint32_t* row_meta;
};

// CTA k: the tables block_prepare builds for momentum (k % lx, k / lx).
template <typename W>
__global__ void __launch_bounds__(kPackThreads) k_pack_tables(const __grid_constant__ PackArgs A,
                                                             const __grid_constant__ Geom g,
                                                             const W* __restrict__ dns, W* __restrict__ row_dn) {
  __shared__ int warp_tot[kPackWarps];
  const int k = blockIdx.x, tid = threadIdx.x;
  const int mx = k % g.lx, my = k / g.lx;
  const int64_t tot = static_cast<int64_t>(A.nclass - 1) * A.c_dn;
  int32_t* act = A.act + k * tot;
  uint32_t* act_list = A.act_list + k * tot;
  uint64_t* dtab = A.dtab + k * tot;
  int64_t* aoff = A.aoff + k * (A.nur + 1);
  int32_t* nact = A.nact + k * A.nclass;
  // active canonical words of every class, in rank order
  for (int c = 1; c < A.nclass; ++c) {
    const int64_t base = static_cast<int64_t>(c - 1) * A.c_dn;
    int run = 0;
    for (int64_t t0 = 0; t0 < A.c_dn; t0 += kPackThreads) {
      const int64_t t = t0 + tid;
      const int f = t < A.c_dn && A.canon[base + t] &&
                    char_trivial(A.d_stab[base + t], A.d_chi[base + t], mx, my, g);
      int all;
      const int pos = run + pack_scan(f, warp_tot, all);
      if (t < A.c_dn) act[base + t] = f ? pos : -1;
      if (f) act_list[base + pos] = static_cast<uint32_t>(t);
      run += all;
    }
    if (tid == 0) nact[c] = run;
  }
  if (tid == 0) nact[0] = static_cast<int32_t>(A.c_dn);
  __syncthreads();
  for (int64_t t = tid; t < tot; t += kPackThreads) {
    const int64_t s = (t / A.c_dn) * A.c_dn + A.d_star[t];
    const uint16_t hs = A.d_hs[t];
    dtab[t] = pack_dtab(act[s], hs & 0xFF, hs >> 8, __popcll(A.d_stab[s]));
  }
  // row offsets of the up representatives
  int run = 0;
  for (int64_t u0 = 0; u0 < A.nur; u0 += kPackThreads) {
    const int64_t u = u0 + tid;
    const int n = u < A.nur ? nact[A.ur_class[u]] : 0;
    int all;
    const int pos = run + pack_scan(n, warp_tot, all);
    if (u < A.nur) aoff[u] = pos;
    run += all;
  }
  if (tid == 0) {
    aoff[A.nur] = run;
    A.dims[k] = run;
  }
  if (run != A.row0[k + 1] - A.row0[k]) return;  // the host reports the mismatch; no row is written
  __syncthreads();
  const int lane = tid & 31;
  for (int64_t u = tid >> 5; u < A.nur; u += kPackWarps) {
    const int c = A.ur_class[u];
    const int64_t r0 = A.row0[k] + aoff[u], n = aoff[u + 1] - aoff[u];
    const int64_t base = static_cast<int64_t>(c - 1) * A.c_dn;
    for (int64_t t = lane; t < n; t += 32) {
      const int64_t j = c == 0 ? t : static_cast<int64_t>(act_list[base + t]);
      const int deg = c == 0 ? 1 : __popcll(A.d_stab[base + j]);
      A.row_meta[r0 + t] = static_cast<uint32_t>(u) | (static_cast<uint32_t>(deg - 1) << 26);
      row_dn[r0 + t] = dns[j];
    }
  }
}

// What resolve() reads of one block.
template <typename W>
struct PackView {
  const uint64_t* up_info;
  const uint16_t* ur_class;
  const int64_t* aoff;
  const uint64_t* dtab;
  int64_t c_dn;
};

template <typename W>
struct RowArgs {
  Geom g;
  const uint64_t* up_info;
  const uint16_t* ur_class;
  const W* ur_bits;
  int64_t c_dn;
  int n_up, n_dn;
  const uint64_t* binom;
  const PackItem* items;
};

// A warp resolves the row's candidate hops 32 at a time, in the reference's
// order (up spin first, occupied sites ascending, directions 0..7). `emit` is
// called by the whole warp once per 32 candidates with each lane's hop.
template <typename W, typename F>
__device__ __forceinline__ void pack_row(const RowArgs<W>& P, const PackItem& it, int64_t i, bool nonzero_only,
                                         F&& emit) {
  const Geom& g = P.g;
  const int lane = threadIdx.x & 31;
  const uint32_t meta = it.row_meta[i];
  const uint32_t ur = meta & 0x3FFFFFFu;
  const int deg_s = static_cast<int>(meta >> 26) + 1;
  const W u = P.ur_bits[ur], d = static_cast<const W*>(it.row_dn)[i];
  const PackView<W> v{P.up_info, P.ur_class, it.aoff, it.dtab, P.c_dn};
  const int ncand = 8 * (P.n_up + P.n_dn);
  for (int q0 = 0; q0 < ncand; q0 += 32) {
    const int q = q0 + lane;
    bool ok = false;
    int64_t col = -1;
    int shift = 0, sgn = 0, deg_t = 1, par = 0, dir = q & 7;
    if (q < ncand) {
      const int p = q >> 3;
      const bool down = p >= P.n_up;
      const W bits = down ? d : u;
      const int from = kth_bit(bits, down ? p - P.n_up : p);
      const int to = g.nb[from][dir];
      if (!((bits >> to) & 1) && !(nonzero_only && g.amp_re[dir] == 0.0 && g.amp_im[dir] == 0.0)) {
        const W moved = bits ^ (static_cast<W>(1) << from) ^ (static_cast<W>(1) << to);
        ok = resolve<W, uint64_t>(down ? u : moved, down ? moved : d, !down, ur, v, g, P.binom, col, shift, sgn,
                                  deg_t);
        par = jw_parity(bits, from, to) ^ sgn;
      }
    }
    emit(u, d, deg_s, ok, static_cast<int>(col), dir, par, shift, deg_t);
  }
}

// Rows of dense column-major matrices (zeroed): the diagonal, then the hops in
// reference order, so the sums are those of adding the CSR's entries in order.
template <typename W>
__global__ void __launch_bounds__(256) k_pack_dense(const __grid_constant__ RowArgs<W> P, double2* __restrict__ arena) {
  const PackItem it = P.items[blockIdx.y];
  const int64_t i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= it.n) return;
  const int lane = threadIdx.x & 31;
  double2* A = arena + it.off;
  if (lane == 0) {
    const uint32_t ur = it.row_meta[i] & 0x3FFFFFFu;
    A[i + i * it.n].x = __dadd_rn(0.0, diag_energy(P.ur_bits[ur], static_cast<const W*>(it.row_dn)[i], P.g));
  }
  __syncwarp();
  pack_row<W>(P, it, i, false, [&](W, W, int deg_s, bool ok, int col, int dir, int par, int shift, int deg_t) {
    double re = 0.0, im = 0.0;
    if (ok) {
      // ((amp * sign) * phase) * ratio, the operation order of main.cpp:794-797
      const double ar = par ? -P.g.amp_re[dir] : P.g.amp_re[dir];
      const double ai = par ? -P.g.amp_im[dir] : P.g.amp_im[dir];
      const double pr = it.phase[2 * shift], pi = it.phase[2 * shift + 1];
      const double ratio = __ddiv_rn(P.g.sqrt_deg[deg_t], P.g.sqrt_deg[deg_s]);
      re = __dmul_rn(__dsub_rn(__dmul_rn(ar, pr), __dmul_rn(ai, pi)), ratio);
      im = __dmul_rn(__dadd_rn(__dmul_rn(ar, pi), __dmul_rn(ai, pr)), ratio);
    }
    // lanes with the same target: the first of them adds all, in lane order
    const unsigned same = __match_any_sync(0xffffffffu, ok ? col : -1 - lane);
    const bool lead = ok && __ffs(same) - 1 == lane;
    double2 a = make_double2(0.0, 0.0);
    if (lead) {
      a = A[i + static_cast<int64_t>(col) * it.n];
      a.x = __dadd_rn(a.x, re);
      a.y = __dadd_rn(a.y, im);
    }
    const int most = __reduce_max_sync(0xffffffffu, __popc(same));
    unsigned rest = same & (same - 1);
    for (int r = 1; r < most; ++r) {
      const int src = rest ? __ffs(rest) - 1 : lane;
      const double xr = __shfl_sync(0xffffffffu, re, src), xi = __shfl_sync(0xffffffffu, im, src);
      if (lead && rest) {
        a.x = __dadd_rn(a.x, xr);
        a.y = __dadd_rn(a.y, xi);
      }
      rest &= rest - 1;
    }
    if (lead) A[i + static_cast<int64_t>(col) * it.n] = a;
    __syncwarp();  // a later batch of this row may add to the same entry
  });
}

// (M + M^H)/2 with a real diagonal (main.cpp:875-886).
__global__ void __launch_bounds__(256) k_pack_herm(const PackItem* __restrict__ items, double2* __restrict__ arena) {
  const int64_t n = items[blockIdx.y].n;
  double2* A = arena + items[blockIdx.y].off;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < n * n;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = t % n, j = t / n;
    if (i > j) continue;
    if (i == j) {
      A[i + i * n].y = 0.0;
      continue;
    }
    const double2 a = A[i + j * n], b = A[j + i * n];
    const double re = 0.5 * (a.x + b.x), im = 0.5 * (a.y - b.y);
    A[i + j * n] = make_double2(re, im);
    A[j + i * n] = make_double2(re, -im);
  }
}

// Rows of small FTLM blocks: entry k of row i at ent[off + k * n + i]
// (nonzero-amplitude hops, reference order), its length and diagonal.
template <typename W>
__global__ void __launch_bounds__(256) k_pack_entries(const __grid_constant__ RowArgs<W> P,
                                                     const __grid_constant__ SmallRatios R,
                                                     uint32_t* __restrict__ ent, int32_t* __restrict__ cnt,
                                                     double* __restrict__ diag) {
  const PackItem it = P.items[blockIdx.y];
  const int64_t i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= it.n) return;
  const int lane = threadIdx.x & 31;
  uint32_t* e = ent + it.off + i;
  int len = 0;
  pack_row<W>(P, it, i, true, [&](W, W, int deg_s, bool ok, int col, int dir, int par, int shift, int deg_t) {
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      int ratio = 0;
      while (R.num[ratio] * deg_s != R.den[ratio] * deg_t) ++ratio;
      e[static_cast<int64_t>(len + __popc(m & ((1u << lane) - 1))) * it.n] =
          small_entry(col, dir, par, shift, ratio);
    }
    len += __popc(m);
  });
  if (lane == 0) {
    const uint32_t ur = it.row_meta[i] & 0x3FFFFFFu;
    cnt[it.off2 + i] = len;
    diag[it.off2 + i] = diag_energy(P.ur_bits[ur], static_cast<const W*>(it.row_dn)[i], P.g);
  }
}

// e^{i k.s} of every momentum, computed as block_prepare does
// (main.cpp:736-743), once per context: [n_k][64] complex.
void pack_phases(Ctx& c) {
  if (c.pack.phase.p) return;
  const Geom& g = c.geom;
  std::vector<double> h(static_cast<size_t>(g.n) * 128, 0.0);
  for (int k = 0; k < g.n; ++k) block_phases(g, k % g.lx, k / g.lx, h.data() + 128 * k, h.data() + 128 * k + 1, 2);
  c.pack.phase.ensure(sizeof(double) * h.size());
  FTLM_CUDA(cudaMemcpyAsync(c.pack.phase.p, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, c.stream));
  FTLM_CUDA(cudaStreamSynchronize(c.stream));
}

template <typename W>
void pack_build(Ctx& c, int64_t rows) {
  SectorTables& S = c.sec;
  SectorPack& K = c.pack;
  const int nk = c.geom.n;
  const int64_t tot = static_cast<int64_t>(S.nclass - 1) * S.c_dn;
  const size_t words = static_cast<size_t>(std::max<int64_t>(tot * nk, 1));
  K.act.ensure(sizeof(int32_t) * words);
  K.act_list.ensure(sizeof(uint32_t) * words);
  K.dtab.ensure(sizeof(uint64_t) * words);
  K.aoff.ensure(sizeof(int64_t) * (S.nur + 1) * nk);
  K.nact.ensure(sizeof(int32_t) * S.nclass * nk);
  K.dims.ensure(sizeof(int64_t) * (2 * nk + 1));
  K.row_meta.ensure(sizeof(uint32_t) * rows);
  K.row_dn.ensure(sizeof(W) * rows);
  int64_t* row0 = K.dims.as<int64_t>() + nk;
  FTLM_CUDA(cudaMemcpyAsync(row0, K.row0.data(), sizeof(int64_t) * (nk + 1), cudaMemcpyHostToDevice, c.stream));
  PackArgs A{S.nclass, S.c_dn, S.nur, S.canon.as<int32_t>(), S.d_stab.as<uint64_t>(), S.d_chi.as<uint64_t>(),
             S.d_star.as<uint32_t>(), S.d_hs.as<uint16_t>(), S.ur_class.as<uint16_t>(), row0, K.act.as<int32_t>(),
             K.act_list.as<uint32_t>(), K.dtab.as<uint64_t>(), K.aoff.as<int64_t>(), K.nact.as<int32_t>(),
             K.dims.as<int64_t>(), K.row_meta.as<uint32_t>()};
  k_pack_tables<W><<<nk, kPackThreads, 0, c.stream>>>(A, c.geom, S.dns.as<W>(), K.row_dn.as<W>());
  FTLM_LAUNCH_CHECK();
  c.prof.kernel_launches += 1;
  std::vector<int64_t> dims(nk);
  FTLM_CUDA(cudaMemcpyAsync(dims.data(), K.dims.p, sizeof(int64_t) * nk, cudaMemcpyDeviceToHost, c.stream));
  FTLM_CUDA(cudaStreamSynchronize(c.stream));
  for (int k = 0; k < nk; ++k)
    if (dims[k] != c.block_dims[k])
      throw Error(FTLM_ERR_INTERNAL, "block dimension from the orbit tables differs from the character count");
}

// All blocks' tables of the prepared sector, once per sector; false when the
// sector is too large for them.
bool sector_pack(Ctx& c) {
  SectorPack& K = c.pack;
  const int nk = c.geom.n;
  if (K.gen == c.sec_gen) return K.ok;
  K.gen = -1;
  const int64_t tot = static_cast<int64_t>(c.sec.nclass - 1) * c.sec.c_dn;
  K.row0.assign(nk + 1, 0);
  for (int k = 0; k < nk; ++k) K.row0[k + 1] = K.row0[k] + c.block_dims[k];
  K.ok = tot * nk <= kPackMaxWords && K.row0[nk] <= kPackMaxRows;
  if (K.ok) {
    if (c.wide) pack_build<uint64_t>(c, K.row0[nk]);
    else pack_build<uint32_t>(c, K.row0[nk]);
  }
  K.gen = c.sec_gen;
  return K.ok;
}

// Runs `launch(first, count, max rows)` over the items: all at once on the
// sector's tables, or one by one on block_prepare's.
template <typename F>
void for_items(Ctx& c, std::vector<PackItem>& items, F&& launch) {
  if (items.empty()) return;
  pack_phases(c);
  const bool all = sector_pack(c);
  const int lx = c.geom.lx;
  int64_t most = 0;
  for (PackItem& it : items) {
    const int k = it.my * lx + it.mx;
    it.phase = c.pack.phase.as<double>() + 128 * k;
    most = std::max<int64_t>(most, it.n);
    if (!all) continue;
    it.aoff = c.pack.aoff.as<int64_t>() + static_cast<int64_t>(k) * (c.sec.nur + 1);
    it.dtab = c.pack.dtab.as<uint64_t>() + static_cast<int64_t>(k) * (c.sec.nclass - 1) * c.sec.c_dn;
    it.row_meta = c.pack.row_meta.as<uint32_t>() + c.pack.row0[k];
    it.row_dn = c.wide ? static_cast<const void*>(c.pack.row_dn.as<uint64_t>() + c.pack.row0[k])
                       : static_cast<const void*>(c.pack.row_dn.as<uint32_t>() + c.pack.row0[k]);
  }
  c.pack.items.ensure(sizeof(PackItem) * items.size());
  PackItem* d = c.pack.items.as<PackItem>();
  if (all) {
    FTLM_CUDA(cudaMemcpyAsync(d, items.data(), sizeof(PackItem) * items.size(), cudaMemcpyHostToDevice, c.stream));
    launch(d, static_cast<int>(items.size()), most);
  } else {
    for (size_t i = 0; i < items.size(); ++i) {
      PackItem& it = items[i];
      block_prepare(c, it.mx, it.my);
      it.aoff = c.blk.aoff.as<int64_t>();
      it.dtab = c.blk.dtab.as<uint64_t>();
      it.row_meta = c.blk.row_meta.as<uint32_t>();
      it.row_dn = c.blk.row_dn.p;
      FTLM_CUDA(cudaMemcpyAsync(d + i, &it, sizeof(PackItem), cudaMemcpyHostToDevice, c.stream));
      launch(d + i, 1, it.n);
    }
  }
}

template <typename W>
RowArgs<W> row_args(Ctx& c, const PackItem* items) {
  return {c.geom, c.sec.up_info.as<uint64_t>(), c.sec.ur_class.as<uint16_t>(), c.sec.ur_bits.as<W>(), c.sec.c_dn,
          c.sec.n_up, c.sec.n_dn, c.binom.as<uint64_t>(), items};
}

}  // namespace

void pack_dense(Ctx& c, std::vector<PackItem>& items, double2* arena) {
  for_items(c, items, [&](const PackItem* d, int count, int64_t most) {
    const dim3 grid(static_cast<unsigned>((most + 7) / 8), count);
    if (c.wide) k_pack_dense<uint64_t><<<grid, 256, 0, c.stream>>>(row_args<uint64_t>(c, d), arena);
    else k_pack_dense<uint32_t><<<grid, 256, 0, c.stream>>>(row_args<uint32_t>(c, d), arena);
    const dim3 hgrid(static_cast<unsigned>(std::min<int64_t>((most * most + 255) / 256, 4096)), count);
    k_pack_herm<<<hgrid, 256, 0, c.stream>>>(d, arena);
    FTLM_LAUNCH_CHECK();
    c.prof.kernel_launches += 2;
  });
}

SmallRatios small_ratios(int n) {
  SmallRatios R{};
  for (int dt = 1; dt <= n; ++dt)
    for (int ds = 1; ds <= n; ++ds) {
      if (n % dt || n % ds) continue;
      bool known = false;
      for (int k = 0; k < R.n; ++k) known = known || R.num[k] * ds == R.den[k] * dt;
      if (known) continue;
      if (R.n == kSmallRatios) throw Error(FTLM_ERR_INTERNAL, "too many orbit-size ratios");
      R.num[R.n] = static_cast<uint8_t>(dt);
      R.den[R.n] = static_cast<uint8_t>(ds);
      ++R.n;
    }
  return R;
}

void pack_entries(Ctx& c, std::vector<PackItem>& items, uint32_t* ent, int32_t* cnt, double* diag) {
  const SmallRatios R = small_ratios(c.geom.n);
  for_items(c, items, [&](const PackItem* d, int count, int64_t most) {
    const dim3 grid(static_cast<unsigned>((most + 7) / 8), count);
    if (c.wide) k_pack_entries<uint64_t><<<grid, 256, 0, c.stream>>>(row_args<uint64_t>(c, d), R, ent, cnt, diag);
    else k_pack_entries<uint32_t><<<grid, 256, 0, c.stream>>>(row_args<uint32_t>(c, d), R, ent, cnt, diag);
    FTLM_LAUNCH_CHECK();
    c.prof.kernel_launches += 1;
  });
}

}  // namespace ftlm
