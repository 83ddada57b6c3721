// Host-side declarations shared by the library's translation units (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstddef>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "edgpu_internal.cuh"

namespace edgpu {

// Number of kernels this library has launched in the process (every launch site increments it).
long long launch_count();
// Persistent grid: as many blocks of `fn` (block threads, smem dynamic bytes) as are resident on the
// current GPU at once -- one wave, blocks walk their work in a grid-stride loop -- but never more than
// `nitems`.  Cached per (device, kernel, shared memory).
int occupancy_grid(const void *fn, int block, size_t smem, int nitems);
void note_launch(long long n = 1);

// A launch that may start while the kernel before it in the stream still runs (programmatic dependent launch); the
// kernel calls pdl_enter (edgpu_internal.cuh) before it reads anything, so only the launch itself and the set-up of
// shared memory overlap.  The recurrences' steps of three or four small kernels gain by it; the eigen-solver's do not (its
// Gram-Schmidt passes' stages and the operator's L1 want the same memory: 12-orbital solve 5 % slower, 8-site ring 1 %
// faster).
template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  note_launch();
}
// cudaFuncAttributeMaxDynamicSharedMemorySize of a kernel raised to `bytes` on the current device (remembered).
void opt_in_smem(const void *fn, size_t bytes);

inline long long binom_at_host(int n, int k) {
  if (n < 0 || k < 0 || k > n) return 0;
  long long r = 1;
  for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
  return r;
}

// Caching device allocator of a context: blocks are kept per size after free and reused, so the
// steady state of a solve performs no cudaMalloc.  Tracks the bytes held against an HBM budget.
class DeviceAllocator {
 public:
  void *alloc(size_t bytes);
  void free(void *p);
  void release_all();
  size_t in_use() const { return in_use_; }
  size_t held() const { return held_; }
  size_t budget = 0;  // 0 = unlimited
  std::string last_error;

 private:
  std::multimap<size_t, void *> free_;
  std::map<void *, size_t> live_;
  size_t in_use_ = 0, held_ = 0;
};

// items: every operator kernel walks a sector in "items" (row groups) so that batches of uneven
// sectors share one launch and per-item partial sums are reduced in a fixed order.
constexpr int kItemElems = 2048;  // target vector elements per item

template <typename T>
struct SectorItems {
  int nitems;
  int srs_rows;  // SRS: up-rows per item
};

// ---- tables.cu
void build_tables(const DevModel &m, long long *basis_off_host, int *basis, int *ninv, cudaStream_t st);
long long scan_tmp_size(long long n);
void exclusive_scan(const long long *in, long long *out, long long n, long long *tmp, cudaStream_t st);
void launch_spin_csr(const DevModel &m, int spin, int k, long long rows, const int *basis_k, long long *count,
                     long long *rp, long long *scan_tmp, int *rp32, int **col, double **val64, float **val32,
                     long long *nnz_out, int *err, DeviceAllocator &alloc, cudaStream_t st);
// k-major ("ELL") copy of a per-spin CSR: len[d], col/val[k * ld + d]; the padding stays as memset (0)
void launch_spin_ell(const int *rp, const int *col, const double *v64, const float *v32, int rows, int ld, int *len,
                     int *ell_col, double *ell_v64, float *ell_v32, cudaStream_t st);
// one-spin halves of the product interaction terms: up entries of the rows with k up electrons, and the down hops of the
// rows with k down electrons (SectorOp::vu_*, vd_to)
void launch_vprod_up(const DevModel &m, const DevVProd &vp, int k, int rows, const int *basis_k, int *cnt, int4 *ent,
                     cudaStream_t st);
void launch_vprod_dn(const DevModel &m, const DevVProd &vp, int k, int rows, int ld, const int *basis_k, int *to,
                     cudaStream_t st);
// (column, value) pairs of n table entries
template <typename T>
void launch_pack_hops(const int *col, const T *val, long long n, Hop<T> *out, cudaStream_t st);
// slot[i] = tile_slot of column ell_col[i], for tiles of C columns per lane
void launch_tile_slots(const int *ell_col, int n, int rows, int C, unsigned short *slot, cudaStream_t st);
// The k-major matrix of a spin in the order of the two-pass kernels (see k_long_schedule): order[k * ld + d] = the entry
// of row d taken as its k-th, or -1 for a filler, slot the column it reads, and tlen[d] how many entries, fillers among
// them, row d has.
void launch_long_schedule(const int *ell_col, const int *len, int rows, int ld, int kmax, unsigned short *slot, short *order,
                          int *tlen, cudaStream_t st);
// out[k * ld + d] = val[order[k * ld + d] * ld + d], 0 for fillers
template <typename T>
void launch_order_values(const T *val, const short *order, int ld, int kmax, T *out, cudaStream_t st);
void launch_crs(const DevModel &m, const SectorOp<double> &op, long long *count, long long *rp, long long *scan_tmp,
                int **col, double **val64, float **val32, long long *nnz_out, int *err, DeviceAllocator &alloc,
                cudaStream_t st);
void launch_diag(const DevModel &m, const SectorOp<double> &op, double *d64, float *d32, cudaStream_t st);
void launch_socrs_check(const DevModel &m, const SectorOp<double> &op, int *err, cudaStream_t st);

// ---- spmv.cuh / krylov.cu : batched operator kernels
// SMs of a GB300: item sizes aim at one or two items per SM where a sector is small.
constexpr int kSms = 152;
// SRS sectors whose rows (down-spin dimension) are at least this long are swept in tiles of four rows; of shorter rows a
// thread takes one column of a few rows at a time (spmv.cuh: srs_tile, srs_short).
constexpr int kSrsLongRow = 128;
constexpr int kSrsVeryLong = 4096;  // rows from here on do not go four at a time into a tile's shared memory
constexpr int kTileRows = 64;       // most up-spin rows of a tiled item (kSrsLongRow <= row < kSrsVeryLong)
// Sectors of very long rows and many of them take two passes over X (spmv.cuh, k_srs_long): whole rows in shared
// memory for the down-spin hops, then whole columns for the up-spin ones, 16 bytes of interleaved rows or columns
// per place, so both dimensions are held to the 224 KB a block has.  In one pass each up hop reads its source row
// from L2 or beyond (4x4 cluster, sector (8,8): 72 ps per state in one pass, 34 in two); sectors with fewer up rows
// fit L2 and give the second pass too few rows to work on.
constexpr int kLongUp = 512, kLongMax = 224 * 1024 / 16, kLongRows = 4;
__host__ __device__ inline bool srs_two_pass(int up_rows, int dn_rows) {
  return dn_rows >= kSrsVeryLong && dn_rows <= kLongMax && up_rows >= kLongUp && up_rows <= kLongMax;
}
// Up-spin rows per SRS work item.  Rows of kSrsLongRow to kSrsVeryLong - 1 states go in groups of four, 8192 elements per
// item (EDGPU_SRS_ITEM_ELEMS: 512 to 24576, cut to kTileElems), but no fewer items than one per SM where that leaves four
// rows each; longer rows one to three per item (or kLongRows in two passes); of shorter ones about kItemElems elements, in
// sectors that would leave SMs idle 512.  The size of tiled items hardly matters for the batch of all sectors of the
// 12-orbital impurity (its solve 283 ms with 2048 elements, 278 with 4096, 279 with 6144, 281 with 8192, 289 with 12288),
// more for single large sectors (their recurrences 27.9, 27.9, 27.9, 26.2, 30.5 ms).
// most elements of a tiled item: with 8-byte ones 96 KB, which leaves room for the item's up hops (up to 64 rows of 100,
// 16 bytes each, when every site of 20 is bound to every other) in the 227 KB of a block
constexpr int kTileElems = 12288;
inline int srs_item_elems() {
  static const int target = [] {  // elements per item of long rows (EDGPU_SRS_ITEM_ELEMS, for measurements)
    const char *e = getenv("EDGPU_SRS_ITEM_ELEMS");
    const int v = e ? atoi(e) : 0;
    return v >= 512 && v <= 24576 ? std::min(v, kTileElems) : 8192;
  }();
  return target;
}
inline int srs_item_rows(int up_rows, int dn_rows) {
  if (srs_two_pass(up_rows, dn_rows)) return kLongRows;
  const int target = srs_item_elems();
  int r;
  if (dn_rows >= kSrsLongRow && dn_rows < kSrsVeryLong) r = std::max(4, target / dn_rows & ~3);
  else if (dn_rows >= kSrsLongRow) r = std::max(1, 24576 / dn_rows);  // very long rows: as many as stage in 96 KB
  else r = kItemElems / std::max(1, dn_rows);
  // small sectors of short rows, which leave SMs idle: 512 elements or four rows
  if (dn_rows < kSrsLongRow && (long long)up_rows * dn_rows <= 8192) r = std::min(r, std::max(4, 512 / dn_rows & ~3));
  // sectors of too few rows for an item per SM of that size: about one item per SM, of at least four rows
  if (dn_rows >= kSrsLongRow && dn_rows < kSrsVeryLong)
    r = std::min({r, kTileRows, std::max(4, ((up_rows + kSms - 1) / kSms + 3) & ~3)});
  return std::max(1, std::min(r, up_rows));
}

// Rows per item of a recurrence.  Its sums are formed item by item, so the item size is part of the values: not by the
// number of SMs or the storage's needs, as srs_item_rows and row_item, but from the row length alone.
inline int lz_item_rows(int storage, int up_rows, int dn_rows) {
  if (storage != kSRS) return kItemElems;
  if (dn_rows >= kSrsVeryLong) return srs_item_rows(up_rows, dn_rows);
  const int r = dn_rows < kSrsLongRow ? kItemElems / std::max(1, dn_rows)
                                      : std::min(kTileRows, std::max(4, srs_item_elems() / dn_rows & ~3));
  return std::max(1, std::min(r, up_rows));
}

// SRS rows per item of a product of nvec vectors of one sector (edgpu_spmv): the sector's own, or, where those make too few
// items for two per SM, as few as that takes, in groups of four.
inline int vec_item_rows(int srs_rows, int up_rows, int dn_rows, int nitems, long long nvec) {
  if (dn_rows >= kSrsVeryLong || nvec * nitems >= 2 * kSms) return srs_rows;
  return (int)std::min<long long>(srs_rows, std::max<long long>(4, (nvec * up_rows / (2 * kSms) + 3) / 4 * 4));
}

// Room in shared memory for the up hops of an item (entries): of any srs_rows consecutive rows, from the longest row,
// because a product may cut the sector at other rows than multiples of srs_rows (18-site impurity, sector (4,2), two
// vectors: items of 20 rows with up to 220 hops, where groups of 24 from row 0 on have at most 216).  Tiles read their
// hops from there alone; short rows with more than 1024 per item read them from global memory.
inline int item_hop_room(int srs_rows, int dn_rows, int kmax) {
  if (dn_rows >= kSrsVeryLong) return 0;
  const int n = srs_rows * kmax;
  return dn_rows < kSrsLongRow ? std::min(n, 1024) : n;
}

// Rows per item of CRS or SOCRS products over `rows` rows in all: about three items per SM, of `least` to 256 rows, one per
// thread (4900 rows in items of 2048 left all but three SMs idle; 48 vectors of them in items of 64 left three quarters of
// each block's threads idle, 43 instead of 32 us; 15 vectors of 63,504 rows in items of 2048 make one wave with a tail,
// 37 instead of 31 us).
inline int row_item(long long rows, int least) {
  return (int)std::min<long long>(256, std::max<long long>(least, (rows / (3 * kSms) + 63) / 64 * 64));
}
template <typename T>
__host__ __device__ inline void item_range(const SectorOp<T> &op, int srs_rows, long long li, long long &lo, long long &hi) {
  if (op.storage == kSRS) {
    long long u0 = li * srs_rows;
    long long u1 = u0 + srs_rows;
    if (u1 > op.up_rows) u1 = op.up_rows;
    lo = u0 * op.dn_rows;
    hi = u1 * op.dn_rows;
  } else {
    lo = li * (long long)srs_rows;
    hi = lo + srs_rows;
    if (hi > op.dim) hi = op.dim;
  }
}

// One Hamiltonian-times-vector work unit of a batch: y = H x (+ c z), optional per-item <x,y>.
template <typename T>
struct MvTask {
  const SectorOp<T> *op;  // device pointer
  int srs_rows;
  int item_begin;
  const T *x;
  T *y;
  const T *z;
  double c;
};

// Plain Lanczos recurrence (include/edlib/Lanczos.h:36-77) over rotating buffers.
template <typename T>
struct LzTask {
  const SectorOp<T> *op;
  int srs_rows;
  int item_begin;
  int nitems;
  T *buf[3];
  double *alpha;      // [nlanc]
  double *beta;       // [nlanc + 1]
  double *part_a;     // [nitems]
  double *part_b;     // [nitems]
  double *scal;       // [0] bet
  int *state;         // [0] 0, or the step (from 1) that finished it, [1] nlanc
  int nlanc_max;
  int mv_rows;        // rows per item and first item of the product, where it has items of its own (LzBatch::split)
  int mv_begin;
};

// A batch of recurrences for launch_lz_step.  split: the product has its own, smaller items (mv_items of them) and <v, w>
// a pass of its own over the recurrences' items, which are too few where rows are short or stored row by row.
template <typename T>
struct LzBatch {
  const LzTask<T> *tasks;
  const int *item_task;
  int nitems;
  bool split = false;
  const int *mv_item_task = nullptr;
  int mv_items = 0;
};

// Restarted Lanczos eigen-solver task with full classical Gram-Schmidt (twice).
#ifndef EDGPU_CGS_STAGES
#define EDGPU_CGS_STAGES 4  // shared-memory stages of the FP32 Gram-Schmidt slice stream
#endif
#ifndef EDGPU_CGS_MIN_BLOCKS
#define EDGPU_CGS_MIN_BLOCKS 2
#endif
// Vector elements per Gram-Schmidt chunk, in every precision: sums over a vector are formed chunk by chunk, so the length
// is part of the values (FP64 chunks of 512 or 2048, shorter by the vector's length, gave other last bits).  FP64 passes
// are bound by FP64 issue (two lanes per clock and SM) and a chunk is one SM's work, so where chunks are few the dot pass
// divides a chunk's columns and the restart its elements among blocks (krylov.cu: dot_parts, launch_eig_restart).
constexpr int kCgsChunk = 4096;
constexpr int kCgsSup = 64;                  // chunks per split of the dot pass's partials reduction
__host__ __device__ inline int cgs_nsup(int nchunks) { return (nchunks + kCgsSup - 1) / kCgsSup; }
constexpr int kMaxLd = 128;      // largest projected-matrix dimension (ncv + 1)
constexpr int kGramPairs = 64 * 65 / 2;  // pairs of a restart Gram block: basis of at most 64 vectors
constexpr int kGramSmem = 64 * 1024;         // shared memory of one Gram slice
constexpr int kEigDone = -0x40000000;  // restart code of a finished sector (k_eig_reset)

template <typename T>
struct EigTask {
  const SectorOp<T> *op;
  int srs_rows;
  int item_begin;
  int nitems;
  int chunk_begin;   // first entry of this task in the chunk map
  int nchunks;       // ceil(n / kCgsChunk)
  long long n;
  long long ldv;     // column stride of V (n rounded up to 16 bytes)
  int m;             // basis vectors before a restart (ncv, clamped to n)
  int ld;            // leading dimension of Tm (mmax + 1)
  T *V;              // (m + 1) columns, ldv apart
  T *w;              // ldv
  double *Tm;        // ld x ld column-major projected matrix
  double *hpart;     // [nchunks][ld] partials of s = V^T w
  double *hpart2;    // [nchunks][ld] partials of g = V^T V[j]
  double *spart;     // [nsup][2 ld + 2] superchunk sums of s, g and |w|^2 (kCgsSup chunks each)
  double *hv;        // [ld] projection coefficients h = (I - E) s of the step
  int *ord;          // [ld + 1] update order: [0] columns subtracted exactly, then the column indices
  int *cnt;          // [nsup + 1] arrival counters of the dot reduction, zero between launches
  double *npart;     // [2][nchunks] |w|^2 before and after the projection
  double *E;         // ld x ld Gram deviation V^T V - I of the basis (column-major)
  double *gpart;     // [nchunks][gstride] partial Gram blocks after a restart
  int gstride;       // (m + 1)(m + 2) / 2: pairs of the largest basis
  double *nsc;       // [0] |w|^2 of the step before the projection
  // st: [0] basis size j + 1 so far (-1 before the first vector), [1] mode (0 Lanczos, 1 orthogonalising a
  // random vector), [2] not growing (basis full or given up), [3] random draws, [5] sector finished,
  // [6] [0] as the step found it, [7] 0 where [2] held, else 1 + 2 [1] + 4 [3] as the step found them
  int *st;
  unsigned long long seed;
  const T *start;    // first basis vector (before orthogonalisation); nullptr: a seeded random vector
};

// FP64 Rayleigh-Ritz refinement of k FP32 Ritz vectors of one sector (items of kItemElems elements)
struct RrTask {
  long long n;
  int k;             // <= 32
  int item_begin, nitems;
  const double *X;   // k x n
  const double *W;   // k x n, H X
  double *part;      // [nitems][2 k k]
  double *theta;     // [k]
  double *Y;         // [k][k], column i = coefficients of refined vector i
  float *out;        // k x n refined vectors
  int *status;       // [1] 0 ok, 1 Gram matrix not positive definite
};
void launch_rr(const RrTask *tasks_dev, const int *item_task_dev, int nitems, int ntasks, double *work, cudaStream_t st);

// Shared-memory shape of an operator launch (all tasks of a launch share one storage kind):
// xs_elems vector elements for the staged rows of an item; plain = 1 when no task of a launch_mv has a
// z term or wants dot products.
struct MvShape {
  int storage;
  int xs_elems;       // staging elements of an item's own rows
  int hop_elems = 0;  // up hops of a tiled item
  int long_places = 0;  // rows or columns of the largest two-pass sector (0: none)
  int other = 0;        // some sector is not a two-pass one
  int short_rows = 0;   // one sector, of short rows
  int plain = 0;
  int mb = 2;         // resident blocks per SM of the eigen-step operator kernel: 2 or 3 (plain launches: 3)
};
// Operator variants the tuner chooses between for the eigen step (spmv.cuh, tune_eig_mv): resident blocks per SM
// {2, 3}; all compute the same sums in the same order, so the choice changes speed only.
struct OpTuning {
  int mb = 2;
  double ms = 0.0;  // time of the chosen variant on the tuning launch
  bool done = false;
};

// nvec vectors of one sector (edgpu_spmv): items of `rows` rows, `per` of them per vector
template <typename T>
struct Sector_mv {
  const SectorOp<T> *op;
  const T *x;
  T *y;
  long long ld;
  int nvec, rows, per;
  bool accumulate;
};
template <typename T>
void launch_mv_vectors(const Sector_mv<T> &v, MvShape sh, cudaStream_t st);
template <typename T>
void launch_mv(const MvTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, cudaStream_t st);

// One block that waits (bounded) on a bulk-copy barrier no copy completes: *gave_up_dev = 1 when both waits
// gave up (krylov.cu, k_wait_selftest).
void launch_wait_selftest(int rounds, int *gave_up_dev, cudaStream_t st);
// true (and cleared) when a bounded wait of the Gram-Schmidt dot pass gave up on a bulk copy
bool take_cgs_stall();
template <typename T>
void launch_lz_mv(const LzBatch<T> &b, int it, bool early, MvShape sh, cudaStream_t st);
template <typename T>
void launch_eig_mv(const EigTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, cudaStream_t st,
                   T *probe_y = nullptr);
// The operator tuner on an eigen-step batch: every variant timed on the batch's own tasks (probe mode: x =
// V[0] of every task, into the scratch probe_y of the largest task's length); returns the fastest.
template <typename T>
OpTuning tune_eig_mv(const EigTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, T *probe_y,
                     cudaStream_t st);
template <typename T>
void launch_lz_step(const LzBatch<T> &b, int it, MvShape sh, cudaStream_t st);
// Kernel attributes the step kernels need for this shape; call before launch_eig_step (and before a
// step is captured into a graph).
template <typename T>
void prepare_eig_step(MvShape sh);
template <typename T>
void prepare_eig_mv(MvShape sh);
template <typename T>
void launch_eig_step(const EigTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, const int *chunk_task_dev,
                     int nchunks, const int *leaders_dev, int nleaders, MvShape sh, cudaStream_t st);
template <typename T>
void launch_eig_jacobi(const EigTask<T> *tasks_dev, int ntasks, double *theta, double *Y, double *resid, int ld,
                       double *work, int *status, cudaStream_t st);
template <typename T>
void launch_eig_restart(const EigTask<T> *tasks_dev, const int *chunk_task_dev, int nchunks, const int *keep,
                        const double *Y, int ld, T *const *outV, cudaStream_t st);

template <typename T>
void launch_eig_reset(const EigTask<T> *tasks_dev, int ntasks, const int *rk, const double *theta, int ld,
                      cudaStream_t st);

// Fresh deterministic random vector in w of every task in restart mode (w <- hash(seed, draw, i) - 0.5)
template <typename T>
void launch_eig_random(const EigTask<T> *tasks_dev, const int *chunk_task_dev, int nchunks, cudaStream_t st);
// out[i] = sum_q coef[q] * vecs[q][i], i < n, vecs[q] FP64 where is64[q] else FP32 (Ritz vectors -> one FP64 vector)
void launch_seed_combine(const void *const *vecs, const int *is64, const double *coef, int k, long long n, double *out,
                         cudaStream_t st);
// y -= c[0] * x (c a device scalar)
void launch_axpy_dev(double *y, const double *x, const double *c, long long n, cudaStream_t st);
// The two Gram-Schmidt passes of an eigen-solver step on their own (launch_eig_step runs them).
template <typename T>
void launch_cgs_dot(const EigTask<T> *tasks_dev, const int *chunk_task_dev, int nchunks, cudaStream_t st);
// kernel attributes of launch_cgs_dot (its staging buffers); call once before launching or capturing it
template <typename T>
void prepare_cgs();
template <typename T>
void launch_cgs_upd(const EigTask<T> *tasks_dev, const int *chunk_task_dev, int nchunks, cudaStream_t st);
// between the two: the chunk partials of the dot pass reduced per task and the projection coefficients
template <typename T>
// leaders_dev: the chunk indices (into chunk_task_dev) whose chunk starts a split of kCgsSup chunks of its task
void launch_cgs_coef(const EigTask<T> *tasks_dev, const int *chunk_task_dev, const int *leaders_dev, int nleaders,
                     cudaStream_t st);
// Gram block of every restarted task's basis (rk[b] != 0, != kEigDone) into EigTask::E.
template <typename T>
void launch_eig_gram(const EigTask<T> *tasks_dev, const int *chunk_task_dev, int nchunks, int ntasks, const int *rk,
                     cudaStream_t st);
// The same Gram block from the old one and the restart's Y (before launch_eig_reset); see k_eig_gram_proj.
template <typename T>
void launch_eig_gram_proj(const EigTask<T> *tasks_dev, int ntasks, const int *rk, const double *Y, int ld,
                          cudaStream_t st);

// a / a+ (gather form), diagonal operators, dot products, scaling, continued fraction
template <typename T>
void launch_a_adag(const SectorOp<T> &src, const SectorOp<T> &dst, int im, int annihilate, const T *in, T *out,
                   int accumulate, cudaStream_t st, double weight = 1.0);
template <typename T>
void launch_diag_op(const SectorOp<T> &op, int opkind, int mu, int nu, const T *in, T *out, cudaStream_t st);
template <typename T>
void launch_dot_partials(const T *a, const T *b, long long n, double *partial, int nparts, cudaStream_t st);
void launch_reduce(const double *partial, int nparts, double *out, cudaStream_t st);
template <typename T>
void launch_scale(T *x, long long n, const double *norm2, int divide_sqrt, cudaStream_t st);
template <typename T>
void launch_convert(const double *in, T *out, long long n, cudaStream_t st);
template <typename T>
void launch_to_double(const T *in, double *out, long long n, cudaStream_t st);

struct CfJob {
  const double *alpha;
  const double *beta;
  const int *state;     // [1] = nlanc
  double expectation;   // <n|O+O|n>
  double E, E0;
  int isign;
  int sym;              // 0: fermionic fraction; 1: symmetrised bosonic fraction
  double *out;          // complex (re, im) output array base
  long long out_stride; // complex elements between consecutive frequencies
};
// real = 0: z = i omega (Matsubara, static term at index 0 of a symmetrised fraction); real = 1: z = omega + i pi/beta
// res: scratch of njobs * nw complex values
void launch_cf(const CfJob *jobs_dev, int njobs, const double *omega, int nw, double beta_T, int real, double2 *res,
               cudaStream_t st);
void launch_chi_tail(double *chi, long long stride, int nw, const double *omega, double beta_T, double avg,
                     cudaStream_t st);

}  // namespace edgpu
