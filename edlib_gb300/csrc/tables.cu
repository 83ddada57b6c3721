// Sector bookkeeping on the device: combinadic tables, per-spin hopping CSR, full CSR, diagonal.
//
// * basis / ninv        -- SzSymmetry::initial_fill / next_basis (include/edlib/SzSymmetry.h:191-216):
//                          the r-th state with k particles is the r-th k-combination of bit positions in
//                          lexicographic order of the sorted position tuple; ninv is its inverse.
// * spin CSR            -- SpinResolvedStorage::fill_spin (include/edlib/SpinResolvedStorage.h:622-638)
//                          with CRSMatrix::addElement/endLine merging (include/edlib/CRSMatrix.h:46-98)
// * full CSR            -- CRSStorage::fill / addElement (include/edlib/CRSStorage.h:66-83, 169-205)
// * diagonal            -- Model::diagonal for every state of a sector
// * SOCRS collision test -- SOCRSStorage::addElement (include/edlib/SOCRSStorage.h:303-317)
#include "edgpu_kernels.h"

namespace edgpu {

// ------------------------------------------------------------------ combinadic tables
__global__ void k_unrank(int ns, int k, long long count, const long long *binom, int *out) {
  long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= count) return;
  int mask = 0, x = 0;
  long long rem = r;
  for (int i = 0; i < k; ++i) {
    while (true) {
      long long c = binom_at(binom, ns - 1 - x, k - 1 - i);
      if (rem < c) break;
      rem -= c;
      ++x;
    }
    mask |= 1 << x;
    ++x;
  }
  out[r] = mask;
}

__global__ void k_ninv(int ns, const long long *binom, int *ninv) {
  long long mask = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (mask >= (1ll << ns)) return;
  int k = __popc((unsigned)mask);
  long long r = 0;
  int x = 0, i = 0;
  for (int p = 0; p < ns; ++p) {
    if (!((mask >> p) & 1)) continue;
    for (int y = x; y < p; ++y) r += binom_at(binom, ns - 1 - y, k - 1 - i);
    x = p + 1;
    ++i;
  }
  ninv[((long long)k << ns) | mask] = (int)r;
}

void build_tables(const DevModel &m, long long *basis_off_host, int *basis, int *ninv, cudaStream_t st) {
  for (int k = 0; k <= m.ns; ++k) {
    long long cnt = binom_at_host(m.ns, k);
    if (cnt == 0) continue;
    k_unrank<<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(m.ns, k, cnt, m.binom, basis + basis_off_host[k]); note_launch();
  }
  long long nm = 1ll << m.ns;
  cudaMemsetAsync(ninv, 0, sizeof(int) * (size_t)(m.ns + 1) * nm, st);
  k_ninv<<<(unsigned)((nm + 255) / 256), 256, 0, st>>>(m.ns, m.binom, ninv); note_launch();
}

// ------------------------------------------------------------------ exclusive scan (int64)
__global__ void k_scan_block(const long long *in, long long *out, long long n, long long *block_sums) {
  __shared__ long long s[1024];
  long long i = blockIdx.x * 1024ll + threadIdx.x;
  long long v = i < n ? in[i] : 0;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    long long t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < n) out[i] = s[threadIdx.x] - v;
  if (threadIdx.x == 1023) block_sums[blockIdx.x] = s[1023];
}

__global__ void k_scan_add(long long *out, long long n, const long long *block_prefix) {
  long long i = blockIdx.x * 1024ll + threadIdx.x;
  if (i < n) out[i] += block_prefix[blockIdx.x];
}

__global__ void k_scan_total(const long long *in, long long *out, long long n) { out[n] = out[n - 1] + in[n - 1]; }

// out[0..n] = exclusive scan of in[0..n), out[n] = total.  tmp must hold 2*ceil(n/1024)+2 values.
void exclusive_scan(const long long *in, long long *out, long long n, long long *tmp, cudaStream_t st) {
  long long nb = (n + 1023) / 1024;
  if (nb <= 0) {
    cudaMemsetAsync(out, 0, sizeof(long long), st);
    return;
  }
  k_scan_block<<<(unsigned)nb, 1024, 0, st>>>(in, out, n, tmp); note_launch();
  if (nb > 1) {
    exclusive_scan(tmp, tmp + nb + 1, nb, tmp + 2 * nb + 2, st);  // recursion on block sums
    k_scan_add<<<(unsigned)nb, 1024, 0, st>>>(out, n, tmp + nb + 1); note_launch();
  }
  // total = out[n-1] + in[n-1]
  k_scan_total<<<1, 1, 0, st>>>(in, out, n); note_launch();
}

long long scan_tmp_size(long long n) {
  long long s = 0;
  while (n > 1) {
    long long nb = (n + 1023) / 1024;
    s += 2 * nb + 2;
    n = nb;
  }
  return s + 4;
}

// ------------------------------------------------------------------ per-spin hopping CSR
constexpr int kRowMax = 256;

// Builds row r of the spin-s hopping matrix for k particles; count_only -> write count.
__device__ int spin_row(const DevModel &m, int spin, int k, int mask, int *cols, double *vals, int *err) {
  const int shift = spin == 0 ? m.ns : 0;
  const state_t nst = (state_t)mask << shift;
  int len = 0;
  for (int q = 0; q < m.nT; ++q) {
    const Transition &tr = m.T[q];
    if (!trans_valid(tr, nst, m.ip)) continue;
    int sign;
    state_t kk = trans_apply(tr, nst, m.ip, sign);
    int col = m.ninv[((long long)k << m.ns) | (int)(kk >> shift)];
    double t = tr.value;
    if (fabs(t) == 0) continue;
    int found = -1;
    for (int e = 0; e < len; ++e)
      if (cols[e] == col) found = e;
    if (found >= 0) {
      vals[found] += sign * t;
    } else {
      if (len >= kRowMax) { atomicExch(err, 1); return len; }
      cols[len] = col;
      vals[len] = sign * t;
      ++len;
    }
  }
  // CRSMatrix::compress: drop |v| < 1e-15; the element shifted into a removed slot is not re-tested
  for (int e = 0; e < len; ++e) {
    if (fabs(vals[e]) < 1e-15) {
      for (int r = e; r < len - 1; ++r) { vals[r] = vals[r + 1]; cols[r] = cols[r + 1]; }
      --len;
    }
  }
  return len;
}

__global__ void k_spin_count(DevModel m, int spin, int k, long long rows, const int *basis_k, long long *count, int *err) {
  long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  int cols[kRowMax];
  double vals[kRowMax];
  count[r] = spin_row(m, spin, k, basis_k[r], cols, vals, err);
}

__global__ void k_spin_fill(DevModel m, int spin, int k, long long rows, const int *basis_k, const long long *rp,
                            int *rp32, int *col, double *val64, float *val32, int *err) {
  long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  int cols[kRowMax];
  double vals[kRowMax];
  int len = spin_row(m, spin, k, basis_k[r], cols, vals, err);
  long long o = rp[r];
  rp32[r] = (int)o;
  if (r == rows - 1) rp32[rows] = (int)(o + len);
  for (int e = 0; e < len; ++e) {
    col[o + e] = cols[e];
    val64[o + e] = vals[e];
    val32[o + e] = (float)vals[e];
  }
}

// ------------------------------------------------------------------ full CSR of a sector
__device__ int crs_row(const DevModel &m, const SectorOp<double> &op, long long i, int *cols, double *vals, int *err) {
  state_t nst = sector_state(op, i);
  int len = 1;
  cols[0] = (int)i;
  vals[0] = model_diagonal(m, nst);
  for (int pass = 0; pass < 2; ++pass) {
    const Transition *L = pass == 0 ? m.T : m.V;
    int nL = pass == 0 ? m.nT : m.nV;
    for (int q = 0; q < nL; ++q) {
      const Transition &tr = L[q];
      if (!trans_valid(tr, nst, m.ip)) continue;
      int sign;
      state_t kk = trans_apply(tr, nst, m.ip, sign);
      int col = (int)sector_index(op, kk);
      int found = -1;
      for (int e = 0; e < len; ++e)
        if (cols[e] == col) found = e;
      if (found >= 0) {
        vals[found] += sign * tr.value;
      } else {
        if (len >= kRowMax) { atomicExch(err, 1); return len; }
        cols[len] = col;
        vals[len] = sign * tr.value;
        ++len;
      }
    }
  }
  return len;
}

__global__ void k_crs_count(DevModel m, SectorOp<double> op, long long *count, int *err) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= op.dim) return;
  int cols[kRowMax];
  double vals[kRowMax];
  count[i] = crs_row(m, op, i, cols, vals, err);
}

__global__ void k_crs_fill(DevModel m, SectorOp<double> op, const long long *rp, int *col, double *val64,
                           float *val32, int *err) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= op.dim) return;
  int cols[kRowMax];
  double vals[kRowMax];
  int len = crs_row(m, op, i, cols, vals, err);
  long long o = rp[i];
  for (int e = 0; e < len; ++e) {
    col[o + e] = cols[e];
    val64[o + e] = vals[e];
    val32[o + e] = (float)vals[e];
  }
}

// ------------------------------------------------------------------ diagonal, collisions
__global__ void k_diag(DevModel m, SectorOp<double> op, double *d64, float *d32) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= op.dim) return;
  double v = model_diagonal(m, sector_state(op, i));
  d64[i] = v;
  d32[i] = (float)v;
}

// SOCRS refuses a transition that lands on the diagonal or twice on the same column
__global__ void k_socrs_check(DevModel m, SectorOp<double> op, int *err) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= op.dim) return;
  state_t nst = sector_state(op, i);
  long long cols[kRowMax];
  int len = 0;
  for (int pass = 0; pass < 2; ++pass) {
    const Transition *L = pass == 0 ? m.T : m.V;
    int nL = pass == 0 ? m.nT : m.nV;
    for (int q = 0; q < nL; ++q) {
      if (!trans_valid(L[q], nst, m.ip)) continue;
      int sign;
      long long c = sector_index(op, trans_apply(L[q], nst, m.ip, sign));
      if (c == i) { atomicExch(err, 2); return; }
      for (int e = 0; e < len; ++e)
        if (cols[e] == c) { atomicExch(err, 3); return; }
      if (len < kRowMax) cols[len++] = c;
    }
  }
}

__global__ void k_spin_ell(const int *rp, const int *col, const double *v64, const float *v32, int rows, int ld,
                           int *len, int *ell_col, double *ell_v64, float *ell_v32) {
  for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < rows; d += gridDim.x * blockDim.x) {
    const int j0 = rp[d], j1 = rp[d + 1];
    len[d] = j1 - j0;
    for (int j = j0; j < j1; ++j) {
      const long long e = (long long)(j - j0) * ld + d;
      ell_col[e] = col[j];
      ell_v64[e] = v64[j];
      ell_v32[e] = v32[j];
    }
  }
}

template <typename T>
__global__ void k_pack_hops(const int *col, const T *val, long long n, Hop<T> *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    Hop<T> h{};
    h.c = col[i];
    h.v = val[i];
    out[i] = h;
  }
}
template <typename T>
void launch_pack_hops(const int *col, const T *val, long long n, Hop<T> *out, cudaStream_t st) {
  if (n <= 0) return;
  k_pack_hops<T><<<(unsigned)std::min<long long>(1024, (n + 255) / 256), 256, 0, st>>>(col, val, n, out); note_launch();
}
template void launch_pack_hops<float>(const int *, const float *, long long, Hop<float> *, cudaStream_t);
template void launch_pack_hops<double>(const int *, const double *, long long, Hop<double> *, cudaStream_t);
template void launch_pack_hops<ffloat>(const int *, const ffloat *, long long, Hop<ffloat> *, cudaStream_t);

__global__ void k_tile_slots(const int *ell_col, int n, int rows, int C, unsigned short *slot) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    slot[i] = (unsigned short)tile_slot(ell_col[i], rows, C);
}
void launch_tile_slots(const int *ell_col, int n, int rows, int C, unsigned short *slot, cudaStream_t st) {
  k_tile_slots<<<std::max(1, std::min(1024, (n + 255) / 256)), 256, 0, st>>>(ell_col, n, rows, C, slot); note_launch();
}

// The order of a row's hops in the two-pass kernels, one row per lane.  A 16-byte shared-memory load of a warp runs in
// four phases of eight lanes; lanes whose places agree modulo 8 (but differ) take one wavefront more each.  The eight
// lanes of a phase may take their entries in any order, so per group of eight rows entries are dealt in rounds: lanes with
// most entries left first, each the entry whose bank is least used in this round, among those the bank with most entries
// left; a lane that would meet a conflict and has rounds to spare waits, reading its own place (value 0), so that an element
// that is not finite reaches no row it is not bound to (what the round's first lane reads, without a conflict of its own,
// is 3 % faster on the 4x4 cluster).  (The tiles keep the matrix' order: eigen-solves and recurrences add in it, and sums in another order are other
// values.  There a load takes 1.8 to 2.5 wavefronts; dealt out it took 1.1 to 1.8.)
__global__ void k_long_schedule(const int *ell_col, const int *len, int rows, int ld, int kmax, unsigned short *slot,
                                short *order, int *tlen) {
  // the group's columns at hand: lane q's entry e at at[(e * 8 + q) * 32], for rows of at most 64 entries
  extern __shared__ unsigned short schedule_smem[];
  unsigned short *at = schedule_smem + threadIdx.x;
  const int ngroups = (rows + 7) / 8;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
    int col[8], left[8], cnt[8];
    unsigned long long rem[8];
    int nmax = 0;
    for (int b = 0; b < 8; ++b) cnt[b] = 0;
    for (int q = 0; q < 8; ++q) {
      const int d = 8 * g + q;
      col[q] = d < rows ? d : -1;
      left[q] = d < rows ? len[d] : 0;
      rem[q] = left[q] >= 64 ? ~0ull : (1ull << left[q]) - 1;
      nmax = max(nmax, left[q]);
      for (int e = 0; e < left[q]; ++e) {
        const int s = ell_col[e * ld + d];
        if (e < 64) at[(e * 8 + q) * 32] = (unsigned short)s;
        ++cnt[s & 7];
      }
    }
    for (int q = 0; q < 8; ++q)
      if (col[q] >= 0) tlen[col[q]] = nmax;
    for (int k = 0; k < kmax; ++k) {
      int used[8], pick[8];
      for (int b = 0; b < 8; ++b) used[b] = 0, pick[b] = -1;
      unsigned todo = 0xff;
      for (int turn = 0; turn < 8 && k < nmax; ++turn) {
        int q = -1;
        for (int i = 0; i < 8; ++i)
          if ((todo >> i & 1) && (q < 0 || left[i] > left[q])) q = i;
        todo &= ~(1u << q);
        if (left[q] == 0) continue;
        int best = -1, bu = 0, bc = 0;
        if (nmax > 64) best = len[col[q]] - left[q];  // long rows keep their order
        for (unsigned long long m = nmax > 64 ? 0 : rem[q]; m; m &= m - 1) {
          const int e = __ffsll((long long)m) - 1, b = at[(e * 8 + q) * 32] & 7;
          if (best < 0 || used[b] < bu || (used[b] == bu && cnt[b] > bc)) best = e, bu = used[b], bc = cnt[b];
        }
        if (nmax <= 64 && bu > 0 && left[q] < nmax - k) continue;
        const int s = best < 64 ? at[(best * 8 + q) * 32] : ell_col[best * ld + col[q]];
        ++used[s & 7];
        --cnt[s & 7];
        --left[q];
        rem[q] &= ~(1ull << (best & 63));
        pick[q] = best;
      }
      for (int q = 0; q < 8; ++q) {
        if (col[q] < 0) continue;
        const int o = k * ld + col[q];
        order[o] = (short)pick[q];
        slot[o] = (unsigned short)(pick[q] < 0 ? col[q]
                                   : pick[q] < 64 ? at[(pick[q] * 8 + q) * 32] : ell_col[pick[q] * ld + col[q]]);
      }
    }
  }
}
void launch_long_schedule(const int *ell_col, const int *len, int rows, int ld, int kmax, unsigned short *slot, short *order,
                          int *tlen, cudaStream_t st) {
  const int ngroups = (rows + 7) / 8;
  k_long_schedule<<<(ngroups + 31) / 32, 32, sizeof(unsigned short) * 32 * 8 * std::min(kmax, 64), st>>>(ell_col, len, rows, ld, kmax, slot, order, tlen); note_launch();
}

template <typename T>
__global__ void k_order_values(const T *val, const short *order, int ld, int kmax, T *out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kmax * ld; i += gridDim.x * blockDim.x)
    out[i] = order[i] >= 0 ? val[order[i] * ld + i % ld] : T(0);
}
template <typename T>
void launch_order_values(const T *val, const short *order, int ld, int kmax, T *out, cudaStream_t st) {
  k_order_values<T><<<std::max(1, std::min(1024, (kmax * ld + 255) / 256)), 256, 0, st>>>(val, order, ld, kmax, out); note_launch();
}
template void launch_order_values<float>(const float *, const short *, int, int, float *, cudaStream_t);
template void launch_order_values<double>(const double *, const short *, int, int, double *, cudaStream_t);
template void launch_order_values<ffloat>(const ffloat *, const short *, int, int, ffloat *, cudaStream_t);

// ------------------------------------------------------------------ product interaction terms
// c+_I c_K on one spin's mask: target mask and sign (orbital m is bit ns - 1 - m); false when not allowed.
__device__ inline bool spin_hop(int ns, int mask, int I, int K, int &to, int &sign) {
  const int bk = 1 << (ns - 1 - K), bi = 1 << (ns - 1 - I);
  if (!(mask & bk)) return false;
  const int m1 = mask ^ bk;
  if (m1 & bi) return false;
  to = m1 | bi;
  sign = ((__popc(mask >> (ns - K)) + __popc(m1 >> (ns - I))) & 1) ? -1 : 1;
  return true;
}

__global__ void k_vprod_up(DevModel m, DevVProd vp, int k, int rows, const int *basis_k, int *cnt, int4 *ent) {
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < rows; u += gridDim.x * blockDim.x) {
    int n = 0;
    for (int q = 0; q < vp.nW; ++q) {
      int to, sign;
      if (!spin_hop(m.ns, basis_k[u], vp.upI[q], vp.upK[q], to, sign)) continue;
      ent[(long long)u * vp.nW + n++] = make_int4(m.ninv[((long long)k << m.ns) | to], vp.g[q], vp.t[q], sign < 0);
    }
    cnt[u] = n;
  }
}

__global__ void k_vprod_dn(DevModel m, DevVProd vp, int k, int rows, int ld, const int *basis_k, int *to_) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < rows * vp.ng; t += gridDim.x * blockDim.x) {
    const int g = t / rows, d = t - g * rows;
    int to, sign;
    const bool ok = spin_hop(m.ns, basis_k[d], vp.dnJ[g], vp.dnL[g], to, sign);
    to_[g * ld + d] = ok ? m.ninv[((long long)k << m.ns) | to] << 1 | (sign < 0 ? 1 : 0) : -1;
  }
}

void launch_vprod_up(const DevModel &m, const DevVProd &vp, int k, int rows, const int *basis_k, int *cnt, int4 *ent,
                     cudaStream_t st) {
  k_vprod_up<<<std::max(1, std::min(1024, (rows + 127) / 128)), 128, 0, st>>>(m, vp, k, rows, basis_k, cnt, ent); note_launch();
}

void launch_vprod_dn(const DevModel &m, const DevVProd &vp, int k, int rows, int ld, const int *basis_k, int *to,
                     cudaStream_t st) {
  const int n = rows * vp.ng;
  k_vprod_dn<<<std::max(1, std::min(1024, (n + 127) / 128)), 128, 0, st>>>(m, vp, k, rows, ld, basis_k, to); note_launch();
}

void launch_spin_ell(const int *rp, const int *col, const double *v64, const float *v32, int rows, int ld, int *len,
                     int *ell_col, double *ell_v64, float *ell_v32, cudaStream_t st) {
  const int blocks = std::max(1, std::min(1024, (rows + 255) / 256));
  k_spin_ell<<<blocks, 256, 0, st>>>(rp, col, v64, v32, rows, ld, len, ell_col, ell_v64, ell_v32); note_launch();
}

void launch_spin_csr(const DevModel &m, int spin, int k, long long rows, const int *basis_k, long long *count,
                     long long *rp, long long *scan_tmp, int *rp32, int **col, double **val64, float **val32,
                     long long *nnz_out, int *err, DeviceAllocator &alloc, cudaStream_t st) {
  unsigned g = (unsigned)((rows + 127) / 128);
  k_spin_count<<<g, 128, 0, st>>>(m, spin, k, rows, basis_k, count, err); note_launch();
  exclusive_scan(count, rp, rows, scan_tmp, st);
  long long nnz = 0;
  cudaMemcpyAsync(&nnz, rp + rows, sizeof(long long), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  *nnz_out = nnz;
  *col = (int *)alloc.alloc(sizeof(int) * (size_t)(nnz > 0 ? nnz : 1));
  *val64 = (double *)alloc.alloc(sizeof(double) * (size_t)(nnz > 0 ? nnz : 1));
  *val32 = (float *)alloc.alloc(sizeof(float) * (size_t)(nnz > 0 ? nnz : 1));
  k_spin_fill<<<g, 128, 0, st>>>(m, spin, k, rows, basis_k, rp, rp32, *col, *val64, *val32, err); note_launch();
}

void launch_crs(const DevModel &m, const SectorOp<double> &op, long long *count, long long *rp, long long *scan_tmp,
                int **col, double **val64, float **val32, long long *nnz_out, int *err, DeviceAllocator &alloc,
                cudaStream_t st) {
  unsigned g = (unsigned)((op.dim + 127) / 128);
  k_crs_count<<<g, 128, 0, st>>>(m, op, count, err); note_launch();
  exclusive_scan(count, rp, op.dim, scan_tmp, st);
  long long nnz = 0;
  cudaMemcpyAsync(&nnz, rp + op.dim, sizeof(long long), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  *nnz_out = nnz;
  *col = (int *)alloc.alloc(sizeof(int) * (size_t)(nnz > 0 ? nnz : 1));
  *val64 = (double *)alloc.alloc(sizeof(double) * (size_t)(nnz > 0 ? nnz : 1));
  *val32 = (float *)alloc.alloc(sizeof(float) * (size_t)(nnz > 0 ? nnz : 1));
  k_crs_fill<<<g, 128, 0, st>>>(m, op, rp, *col, *val64, *val32, err); note_launch();
}

void launch_diag(const DevModel &m, const SectorOp<double> &op, double *d64, float *d32, cudaStream_t st) {
  if (op.dim == 0) return;
  k_diag<<<(unsigned)((op.dim + 255) / 256), 256, 0, st>>>(m, op, d64, d32); note_launch();
}

void launch_socrs_check(const DevModel &m, const SectorOp<double> &op, int *err, cudaStream_t st) {
  if (op.dim == 0) return;
  k_socrs_check<<<(unsigned)((op.dim + 127) / 128), 128, 0, st>>>(m, op, err); note_launch();
}

}  // namespace edgpu
