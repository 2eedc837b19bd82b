// Internal host-side structures of the B200 FTLM engine (not part of the ABI).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ftlm_gpu.h"
#include "dbuf.h"
#include "ftlm_device.cuh"

namespace ftlm {

#define FTLM_LAUNCH_CHECK() FTLM_CUDA(cudaGetLastError())

// Lets `kernel` be launched with up to `most` bytes of dynamic shared memory. The
// limit belongs to the function in the device, for all contexts and host threads,
// so `most` is the same in every call: a limit set to one launch's size would refuse
// a larger launch that another thread has just set it for. It does not affect
// occupancy, which follows from the launch's own size.
template <typename K>
inline void smem_limit(K* kernel, size_t most) {
  FTLM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)));
}

// Translation-orbit tables of one (N_up, N_down) sector.
//
// Representatives are the lexicographic minima of (up, down) orbits
// (main.cpp:643-675 keeps the first member met in an (up, down) ascending
// sweep). Hence the representative's up word is the minimum of its up
// orbit ("up representative" ur), and its down word is minimal among the
// images of the down word under the stabiliser H of ur. Up representatives
// with equal (H, sign character of H on the up word) form a class; each
// non-trivial class owns a table over all down words. Parents are ordered
// by (ur, canonical down), which is the reference's parent order.
struct SectorTables {
  int n_up = -1, n_dn = -1;
  int64_t c_up = 0, c_dn = 0, full_dim = 0, parents = 0;
  int64_t nur = 0;      // number of up representatives
  int nclass = 0;       // classes; class 0 is the trivial stabiliser
  std::vector<uint64_t> cls_stab, cls_sig;   // per class: H mask, sign mask
  std::vector<int64_t> cls_ncanon;           // canonical downs per class
  std::vector<uint16_t> h_ur_class;          // host copy of ur -> class
  DBuf ups, dns;         // W[c_up], W[c_dn] bit words in ascending order
  DBuf up_info;          // uint64[c_up]
  DBuf ur_bits;          // W[nur]
  DBuf ur_class;         // uint16[nur]
  DBuf ur_poff;          // int64[nur+1] parent offsets
  // per non-trivial class c (index c-1), over all down ranks
  DBuf d_star;           // uint32[(nclass-1)*c_dn] rank of the canonical image
  DBuf d_hs;             // uint16[(nclass-1)*c_dn] h | sign<<8 (T_h d* = d)
  DBuf d_stab, d_chi;    // uint64[(nclass-1)*c_dn] for canonical words
  DBuf d_cidx;           // int32[(nclass-1)*c_dn] canonical index (scan)
  DBuf canon;            // int32[(nclass-1)*c_dn] 1 for canonical words
  DBuf tmp_a, tmp_b, tmp_c, tmp_d, tmp_e;  // build scratch
};

// Tables of one momentum block (mx, my) of the prepared sector.
struct BlockTables {
  int mx = -1, my = -1;
  int64_t dim = 0;
  std::vector<int64_t> cls_nact;  // active canonical downs per class
  DBuf act;       // int32[(nclass-1)*c_dn] active index of canonical words (-1)
  DBuf act_list;  // uint32[(nclass-1)*c_dn] ranks of active canonical words
  DBuf aoff;      // int64[nur+1] active row offsets
  DBuf dtab;      // uint64[(nclass-1)*c_dn] packed lookup entries
  DBuf row_meta;  // uint32[dim]: ur | (deg-1)<<26
  DBuf row_dn;    // W[dim]
  double phase_re[64], phase_im[64];
};

// Everything the H*V / CSR kernels need about one block.
template <typename W>
struct BlockView {
  const uint64_t* up_info;
  const W* ur_bits;
  const uint16_t* ur_class;
  const int64_t* aoff;
  const uint64_t* dtab;
  const uint32_t* row_meta;
  const W* row_dn;
  int64_t c_dn;
  int64_t dim;
  int n_up, n_dn;
  double phase_re[64], phase_im[64];
};

// Device-resident spectrum of one block.
struct Spectrum {
  int64_t ev_off = 0;  // eigenvalues at spectra[ev_off .. ev_off+count)
  int64_t w_off = -1;  // weights at spectra[w_off ..), -1 for exact blocks
  int64_t count = 0;   // number of eigenvalues
  bool exact = false;
  double prefactor = 1.0;
  int particles = 0;
  int64_t dim = 0;
  int pending = -1;       // exact block queued for a deferred solve: index into Ctx::defer_items
  int pending_small = -1;  // small FTLM block whose solve is deferred: index into Ctx::defer_small
};

// An exact block whose dense matrix waits in the deferred pool.
struct DeferItem {
  int n_up, n_dn, mx, my;
  int64_t n, aoff;   // dimension, offset (complex entries) of its matrix in defer_arena
  int64_t sec_gen;   // sector generation it was assembled in
};

// One block of a small-block Lanczos launch (smallblock.cu): offsets into the
// context's sb_* arrays.
struct SmallBlockDesc {
  int64_t ent_off;    // entry k of row i at ent[ent_off + k * dim + i]
  int64_t row_off;    // row lengths and diagonal
  int64_t ab_off;     // alpha/beta [K][ld]
  int64_t start_off;  // reference start vectors [R][dim] complex, -1: Philox
  int64_t steps_off;  // steps[steps_off + r]
  uint64_t seed;      // block seed (Philox key)
  int32_t dim, K, ld, k;  // k: momentum index my * lx + mx
};

// A small FTLM block whose rows wait in the deferred pool.
struct DeferSmall {
  int n_up, n_dn, mx, my;
  SmallBlockDesc d;
  int64_t sec_gen;
};

// Entries of small-block rows: column : 12 | direction * 2 + parity : 4 |
// shift : 6 | number of the orbit-size ratio deg_t / deg_s : 6.
constexpr int kSmallRatios = 64;
struct SmallRatios {
  int n;
  uint8_t num[kSmallRatios], den[kSmallRatios];  // deg_t, deg_s of the first pair with that ratio
};
__host__ __device__ inline uint32_t small_entry(int col, int dir, int par, int shift, int ratio) {
  return static_cast<uint32_t>(col) | (static_cast<uint32_t>(dir * 2 + par) << 12) |
         (static_cast<uint32_t>(shift) << 16) | (static_cast<uint32_t>(ratio) << 22);
}

// Tables of every momentum block of a small sector (pack.cu).
struct SectorPack {
  int64_t gen = -1;  // sector generation they belong to
  bool ok = false;
  std::vector<int64_t> row0;  // [n_k + 1] first row of each block
  DBuf act, act_list, dtab, aoff, nact, dims, row_meta, row_dn;
  DBuf phase;  // [n_k][64] complex e^{i k.s}, the context's
  DBuf items;
};

// A block whose rows are built: dense matrix at arena + off, or entries at
// ent + off with lengths and diagonal at off2.
struct PackItem {
  int32_t mx, my;
  int64_t n, off, off2;
  const int64_t* aoff;
  const uint64_t* dtab;
  const uint32_t* row_meta;
  const void* row_dn;
  const double* phase;
};

// A queued accumulation: an exact (small = false) or FTLM block of the pool.
struct DeferAcc {
  bool small;
  int idx;
};

struct Profile {
  double hv_ms = 0.0;       // summed CUDA-event time of H*V launches
  int64_t hv_launches = 0;
  double hv_bytes = 0.0;    // algorithmic bytes of those launches
  double update_ms = 0.0;
  int64_t update_launches = 0;
  double eig_ms = 0.0;
  double dense_ms = 0.0;
  double thermo_ms = 0.0;
  double sector_ms = 0.0;
  double block_ms = 0.0;
  int64_t kernel_launches = 0;
  int64_t h2d_bytes = 0, d2h_bytes = 0;
  int hv_variant = -1;  // H*V kernel variant of the last launch
  int tune_runs = 0;    // autotuner measurements made by this context
  double small_ms = 0.0;     // device time of small-block Lanczos launches
  int64_t small_tasks = 0;   // (block, random vector) pairs they ran
  double hv_hops = 0.0;      // nonzero hop x vector products of the timed H*V launches
  double hv_min_bytes = 0.0; // their compulsory bytes D * (2 nv s + 8) per launch
  int hv_source = -1;        // operator source of the last sweep (kSrcFly / kSrcList / kSrcSplit)
};

// Momentum phases e^{i k.s} of a block, by translation index s.
struct FlipPhase {
  double re[64], im[64];
};

// Largest block dimension the small-block Lanczos launch takes (two FP64 complex
// vectors of this length, 128 KB, live in shared memory; an entry keeps 12 bits of column).
constexpr int64_t kSmallMaxDim = 4096;

struct Ctx {
  Arena arena;  // small buffers of this context and its spin-flipped companion
  ftlm_model model{};
  ftlm_run_opts opts{};
  Geom geom{};
  bool wide = false;  // 64-bit spin words (more than 32 sites)
  int hv_forced = -1; // H*V kernel variant forced by FTLM_HV_VARIANT (-1: autotune)
  bool hv_retune = false;  // FTLM_HV_RETUNE=1: tune once per context, ignoring the process-wide choices
  std::map<uint64_t, int> tuned_local;  // variants chosen by this context's tuner runs
  int hv_mode = -1;   // H*V operator source: -1 auto, 0 on-the-fly lookups, 1 cached hop list,
                      // 2 split-spin segment sweeps (FTLM_HV_MODE=fly|list|split)
  bool hl_active = false;  // H*V kernels read the cached hop list of the prepared block
  bool split_active = false;  // H*V runs as the two segment sweeps of split.cu
  std::unique_ptr<Ctx> flipped;  // tables of sector (N_down, N_up) when N_up != N_down
  DBuf flip_map;      // uint64 per row: flipped row | shift << 32 | sign << 38 (+ an error word)
  int flip_for[5] = {-1, -1, -1, -1, -1};  // (n_up, n_dn, mx, my, stn_pos_seg) the flip map belongs to
  int64_t flip_gen = -1, sec_gen = 0;  // sector generation of the flip map / of the tables
  DBuf vec_xd, vec_yd;  // Lanczos vector and H*V output in the spin-flipped row order
  bool seg_dynamic = true;  // segment sweeps take rows from a shared counter (FTLM_SEG_ROWS=stride: grid-stride)
  DBuf seg_counter;         // the row counters of the two sweeps
  DBuf gauss_jobs;          // Gaussian start vectors to draw
  bool split_stencil = true;  // segment sweeps read the class stencils (FTLM_SPLIT_OP=fly: on-the-fly lookups)
  bool split_wide = false;    // the prepared sweeps are the stencil ones, their vectors in stn_pos order
  // class stencils of this context's prepared block (split.cu)
  bool stn_ok = false;
  int64_t stn_for[3] = {-1, -1, -1};  // (sector generation, mx, my) they belong to
  DBuf stn_crb, stn_rp, stn_ent, stn_cnt;
  DBuf stn_rp4, stn_row, stn_ent4, stn_deg, stn_coef;  // entries of the wide sweeps in runs of one coefficient
  DBuf stn_seg, stn_cls;           // segments by class, class list
  DBuf stn_pos;                    // position of every row in the sweeps' order,
  int stn_pos_seg = 0;             // segments per group of that order (0: not built)
  DBuf stn_diag;                   // diagonal per position, in the sweeps' type
  std::vector<int64_t> stn_classes;  // per class with rows: number of segments, rows per segment
  bool hv_rows = true;  // narrow sweeps on the hop list: 8 lanes per row (FTLM_HV_ROWS=0: warp per row)
  bool small_blocks = true;  // batched FTLM runs blocks <= kSmallMaxDim in one launch (FTLM_SMALL_BLOCKS=0: off)
  int64_t hl_nnz = 0;
  DBuf hl_ptr, hl_ent;     // hop list: int64 row pointers, packed uint64 entries
  int device = 0;
  int sm_count = 148;
  cudaStream_t stream = nullptr;
  std::string last_error;
  DBuf binom;         // uint64 [65*65]
  DBuf binom32;       // uint32 [65*65]
  SectorTables sec;
  std::vector<int64_t> block_dims;  // dimension of every k-block of the prepared sector (k = my*lx + mx)
  BlockTables blk;
  // Lanczos work space
  DBuf vec_a, vec_b, vec_h, partial, lz_alpha, lz_beta, lz_scale, lz_state, host_start;
  DBuf ritz_tmp, ritz_out, ritz_meta, scan_tmp;
  // exact batch
  DBuf dense_arena, dense_meta, dense_out, dense_vecs;
  // deferred block spectra (ftlm_spectra_defer): dense matrices of exact
  // blocks and rows of small FTLM blocks of any number of sectors, solved
  // together by flush_deferred, then the queued accumulations
  bool spectra_defer = false;
  DBuf defer_arena, defer_ev, defer_work;
  int64_t defer_asz = 0;
  std::vector<DeferItem> defer_items;
  std::vector<DeferSmall> defer_small;
  std::vector<DeferAcc> defer_acc;
  // small FTLM blocks, running or pooled: entries, row lengths, diagonals,
  // start vectors, Lanczos coefficients, step counts, task lists. A pooled
  // sector's Lanczos runs on a side stream while the next sectors' tables are
  // built; the buffers move only when the side streams are idle, and c.stream
  // waits for them before the Ritz stage.
  DBuf sb_ent, sb_cnt, sb_diag, sb_start, sb_alpha, sb_beta, sb_steps, sb_meta;
  int64_t sb_ent_used = 0, sb_row_used = 0, sb_start_used = 0, sb_ab_used = 0, sb_st_used = 0, sb_meta_used = 0;
  static constexpr int kSide = 8;
  cudaStream_t side[kSide] = {};
  cudaEvent_t side_ev = nullptr;
  int side_next = 0;
  SectorPack pack;
  // spectra of the current sector's blocks (device arena)
  DBuf spectra;
  int64_t spectra_used = 0;
  std::map<std::pair<int, int>, Spectrum> spec;
  // thermo
  int nbeta = 0, nmu = 0;
  DBuf th_beta, th_mu, th_state;  // state: [4][nbeta][nmu] emin, z, n, n2
  // instrumentation
  bool timing = false;
  Profile prof;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // last Lanczos run (debug readback)
  int last_kdim = 0, last_nv = 0;
};

// ---- launchers implemented in the .cu files
void sector_prepare(Ctx& c, int n_up, int n_dn);
void block_prepare(Ctx& c, int mx, int my);
// Dimensions of every block k = my*lx + mx of sector (n_up, n_dn) on the host,
// by character counting: (1/N) sum_s e^{-ik.s} tr_up(T_s) tr_dn(T_s).
std::vector<int64_t> block_dims_by_characters(Ctx& c, int n_up, int n_dn);
void debug_parents(Ctx& c, uint64_t* up, uint64_t* dn, int32_t* deg, double* diag);
void debug_relations(Ctx& c, int32_t* parent, int32_t* shift, int32_t* sign);
void block_csr(Ctx& c, std::vector<int32_t>& row_ptr, std::vector<int32_t>& col,
               std::vector<double>& val, std::vector<double>& diag);
// Device CSR of the prepared block (reference entry order); returns nnz.
int64_t block_csr_device(Ctx& c, DBuf& row_ptr, DBuf& col, DBuf& val, DBuf& diag);
// e^{i k.s} of momentum (mx, my) for every translation s, at re/im[s * stride].
void block_phases(const Geom& g, int mx, int my, double* re, double* im, int stride);
// ---- rows of many blocks of the prepared sector (pack.cu); items carry mx,
// my, n and the offsets, the rest is filled in. No host synchronisation beyond
// one per sector.
// Dense Hermitian matrices (M + M^H)/2, column-major, at arena + off (zeroed).
void pack_dense(Ctx& c, std::vector<PackItem>& items, double2* arena);
// Entries, row lengths and diagonals of small blocks.
void pack_entries(Ctx& c, std::vector<PackItem>& items, uint32_t* ent, int32_t* cnt, double* diag);
SmallRatios small_ratios(int n);
// H*V of the prepared block on device arrays [dim][nv] complex (FP64 or FP32).
// partial_dev[grid][nv] receives each CTA's fixed-point sum of Re<s x, y>.
void hv_apply(Ctx& c, const void* in, void* out, int nv, bool fp32, const double* scale_dev,
              fx128* partial_dev, int nblocks_hint);
int hv_grid(Ctx& c, int nv, bool fp32);
// Chooses the operator source of sweeps of nv vectors over the prepared
// block (FTLM_HV_MODE or the automatic rule): on-the-fly lookups, the cached
// hop list (few vectors per sweep), or the split-spin segment sweeps (large
// blocks); builds what it needs and sets c.hl_active / c.split_active. The
// guard clears them again.
enum { kSrcFly = 0, kSrcList = 1, kSrcSplit = 2 };
constexpr int64_t kSplitMinDim = int64_t(1) << 15, kSplitMinDimFp64 = 12288;  // the latter for wide FP64 sweeps
int hv_select_source(Ctx& c, int nv, bool fp32);
struct HvSourceGuard {
  Ctx& c;
  ~HvSourceGuard() {
    c.hl_active = false;
    c.split_active = false;
  }
};
// Autotuner cache (hv.cu): variant chosen for a key by this context or the process.
int hv_size_class(int64_t dim);
bool hv_tuned_lookup(Ctx& c, uint64_t key, int& var);
void hv_tuned_store(Ctx& c, uint64_t key, int var);

// ---- split-spin H*V (split.cu)
// Prepares the spin-flipped tables and the flip map of the prepared block and
// the two flipped-order arrays for sweeps of nv vectors; false when they do
// not fit in device memory.
bool split_prepare(Ctx& c, int nv, bool fp32);
// Whether the prepared sector's split sweeps run on the class stencils: known
// before anything is built.
bool split_stencils(const Ctx& c);
// The prepared sweeps' row order for another number of vectors.
void split_order(Ctx& c, int nv, bool fp32);
// y = M x for x given in both row orders: out (this block's order, diagonal
// included) and out_d (flipped order) such that M x = out + S^T out_d.
// partial receives 2 x grid rows of fixed-point Re<s x, y> sums; returns
// that row count.
int hv_apply_split(Ctx& c, const void* in, const void* in_d, void* out, void* out_d, int nv, bool fp32,
                   const double* scale, fx128* partial);
// Row order of the stencil sweeps' vectors (split.cu): position of every row of
// the block, null where the active operator keeps the block order. Those sweeps
// take any number of vectors (FP32: an even one), leave y unscaled (the Lanczos
// update then applies the scale) and read up to kSweepPad bytes past the end of
// their input vectors.
const uint32_t* sweep_pos(const Ctx& c);
constexpr size_t kSweepPad = 2048;
inline int sweep_width(int nvec, bool fp32) { return fp32 ? (nvec + 1) / 2 * 2 : nvec; }
// Host vectors ([dim][nvec] complex FP64, block order) to [dim][NV] of the working
// precision in the operator's row order, and back, kConvertChunk elements at a
// time (256 MB on the device, whatever the block; less where that does not fit).
void vectors_from_host(Ctx& c, int nvec, int NV, bool fp32, const double* in, void* vec);
void vectors_to_host(Ctx& c, int nvec, int NV, bool fp32, const void* vec, double* out);
constexpr int64_t kConvertChunk = int64_t(1) << 24, kConvertLeast = int64_t(1) << 16;
// Whether the host converts `rows` x nvec elements, padded to NV vectors. Its loops and
// zero fill cost by the padded element, the device's way two launches and copies of 16
// bytes by the element: the difference follows rows (3 NV - 2 nvec). One vector is dearer on
// the host, and FP64 padding on the device needs no more than its elements. Whole calls,
// host / device (us), mixed precision:
//   1 vector   4036 rows 96 / 97, 5072 88 / 81, 14520 153 / 131
//   2 vectors  8008 rows 113 / 137, 14520 182 / 211
//   3 (4)      14520 rows 264-283 / 274-314
//   5 (8)      5072 rows 173 / 180, 8008 262 / 251, 14520 463 / 380
//   8 vectors  8008 rows 296 / 350, 14520 538 / 521
//   13 (16)    4368 rows 333 / 369
//   14 (16)    4036 rows 283 / 321, 5072 340 / 367, 8008 552 / 505
//   24 (32)    1176 rows 162 / 185, 4036 510 / 424
// FP64 with padding (else nothing is converted): 198 elements 37 / 42, 2744 55 / 57, 4256
// 68 / 71, 5292 77 / 74, 8820 113 / 87, 20180 216 / 147.
inline bool host_convert(int64_t rows, int nvec, int NV, bool fp32) {
  if (!fp32) return rows * nvec < 5000;
  return nvec == 1 ? rows < 4500 : rows * (3 * NV - 2 * nvec) < (NV < 32 ? 100000 : 84000);
}
int hv_split_max_grid(const Ctx& c);
// x_D[p(q)] = conj(f_q) x[q];  y[q] += f_q y_D[p(q)].
void flip_scatter(Ctx& c, const void* x, void* xd, int nv, bool fp32);
void flip_gather_add(Ctx& c, void* y, const void* yd, int nv, bool fp32);
FlipPhase flip_phase(const Ctx& c);
BlockView<uint32_t> view32(Ctx& c);
BlockView<uint64_t> view64(Ctx& c);

// Lanczos over the prepared block; results stored as a Spectrum.
void run_ftlm_block(Ctx& c, int n_up, int n_dn, int mx, int my, Spectrum& out,
                    const double* host_start /* [R][dim] complex or null */,
                    std::vector<double>* alpha_out, std::vector<double>* beta_out,
                    std::vector<int32_t>* steps_out);
// One block of a Ritz stage.
struct RitzJob {
  int R, nvmax, ld, K;
  const double* alpha;
  const double* beta;
  const int32_t* steps;
  Spectrum* out;
};
// FTLM spectra of several small blocks (dim <= kSmallMaxDim) of the prepared
// sector; stored like run_ftlm_block's, or pooled until flush_deferred.
void run_small_ftlm_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks);
// Empties the sb_* arrays. Makes c.stream wait for the side streams' Lanczos.
void small_rows_reset(Ctx& c);
void small_join(Ctx& c);
RitzJob small_ritz_job(Ctx& c, const SmallBlockDesc& d, Spectrum* out);
// Ritz values and weights of R Lanczos runs (alpha/beta [sweep][K][ld],
// nvmax vectors per sweep, steps[R] on the device) into the spectra arena.
void ritz_stage(Ctx& c, int R, int nvmax, int ld, int K, const double* alpha, const double* beta,
                const int32_t* steps, Spectrum& out);
// The same for several blocks with one host synchronisation.
void ritz_stage_many(Ctx& c, std::vector<RitzJob>& jobs);
// Exact spectra of several blocks of the prepared sector (one batched launch).
void run_exact_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks);
// Deferred form: assembles the blocks' matrices into the pool (flushing it
// first when they would push it past kDeferPoolBytes) and registers them as
// pending spectra of the current sector.
void queue_exact_blocks(Ctx& c, const std::vector<std::pair<int, int>>& blocks);
// Diagonalises the pooled matrices, runs Lanczos and the Ritz stage of the
// pooled FTLM blocks, then the queued accumulations in queue order, and turns the current sector's pending spectra into ordinary
// ones; empties the pool.
void flush_deferred(Ctx& c);
// Bytes held by the pool (matrices, small-block rows, start vectors and coefficients).
int64_t defer_pool_bytes(const Ctx& c);
constexpr int64_t kDeferPoolBytes = int64_t(4) << 30;
// Thermo
void thermo_configure(Ctx& c, int nbeta, const double* beta, int nmu, const double* mu);
void thermo_accumulate(Ctx& c, const Spectrum& s);
// Accumulates a spectrum already on the device (w null: unit weights).
void thermo_accumulate_dev(Ctx& c, const double* ev, const double* w, int64_t count, double pref, int particles);
void thermo_accumulate_host(Ctx& c, const double* ev, const double* w, int64_t count, double pref, int particles);
void thermo_read(Ctx& c, double* emin, double* z, double* n, double* n2);

// Seeds and reference start vectors (main.cpp:514-533, 1015-1025)
uint64_t block_seed(uint64_t seed, int n_up, int n_dn, int mx, int my);
// Reference Gaussian start vectors on c.stream (start.cu): the vector of `seed`
// to out[off .. off + dim), unit norm.
struct GaussJob {
  uint64_t seed;
  int64_t dim, off;
};
void gaussian_starts(Ctx& c, const std::vector<GaussJob>& jobs, double2* out);
// Seed of sample `sample` of the block with seed bseed (main.cpp:1015).
uint64_t sample_seed(uint64_t bseed, int sample);
// The buffers of a context's sector, block and stencil tables.
std::vector<DBuf*> table_bufs(Ctx& c);
// Nonzero-amplitude hops with active targets in the prepared block (the
// h_nz * dim of the H*V byte model).
int64_t block_nonzero_hops(Ctx& c);
// Builds the cached hop list of the prepared block; false when it does not fit in memory.
bool hoplist_build(Ctx& c);

// Spectra arena
int64_t spectra_alloc(Ctx& c, int64_t count);  // returns offset (doubles) of 2*count slots
void spectra_reset(Ctx& c);

// Scan helpers (exclusive, in place on device, returns total)
int64_t scan_excl_i32_to_i64(Ctx& c, const int32_t* flags, int64_t* out, int64_t n);

}  // namespace ftlm
