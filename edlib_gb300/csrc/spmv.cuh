// Hamiltonian-times-vector kernels for the three storages, batched over work items.
//
// * SRS   -- SpinResolvedStorage::av (include/edlib/SpinResolvedStorage.h:58-115): the sector vector is the
//            row-major N_up x N_dn matrix X (d fastest) and
//            Y = D o X + X H_dn^T + H_up X + H_loc X,
//            accumulated per element in the reference order (diagonal, down hops, up hops, interaction).
//            A work item is a group of up-rows; its rows of X are staged in shared memory, so that the H_dn
//            gather reads shared memory, and the H_up term reads whole rows of X (coalesced in d).  Rows of
//            kSrsLongRow to kSrsVeryLong - 1 states in tiles of 4 rows over row-interleaved shared memory (srs_tile);
//            longer rows one at a time (srs_longrow) or, in sectors of many of them, in two passes (k_srs_long);
//            shorter ones a column of a few rows or one element per thread (srs_short, srs_flat).
//            The off-diagonal interaction (H_loc): from tables of its terms' one-spin halves, or matrix-free from the
//            transition list.
//            Element types: FP32, FP64, and float-float pairs (the mixed mode's recurrences).
// * CRS   -- CRSStorage::av (include/edlib/CRSStorage.h:57-64): a thread per row.
// * SOCRS -- SOCRSStorage::av (include/edlib/SOCRSStorage.h:46-87): matrix-free; each row re-derives its
//            state from the combinadic tables, tests every transition by its masks, ranks the target with ninv
//            and takes the fermion sign from one popc; nothing but the tables is stored.  A thread per row.
// Every kernel is instantiated per storage (a launch covers one storage); the recurrences' emit <x, y> per item (FP64 /
// float-float accumulation, fixed order).
//
// The order of every sum is part of the values.  Eigen-solves stop and restart on them, and two kinds of results magnify a
// last bit: a continued fraction that has not converged (of a state that is not the lowest of its neighbouring sectors;
// by up to 1e11), and the last, near-degenerate pairs of a solve.

#pragma once
#include "edgpu_kernels.h"

namespace edgpu {

constexpr int kMvBlock = 256;
static_assert(kSrsLongRow >= 128, "a tile's 128 columns lie inside a row");

__host__ __device__ inline size_t align16(size_t b) { return (b + 15) & ~size_t(15); }

// a b, rounded by itself, and a b + c with one rounding (float-float: its own product and sum): written out where the
// compiler could contract either of two products with their sum, so that a value does not depend on which it takes.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ ffloat mul_rn(ffloat a, ffloat b) { return a * b; }
__device__ __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double madd(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ ffloat madd(ffloat a, ffloat b, ffloat c) { return c += a * b; }

template <typename T>
__device__ __forceinline__ T transitions_term(const SectorOp<T> &op, state_t s, const Transition *L, const T *vals, int nL,
                                              const T *x, T acc) {
  for (int q = 0; q < nL; ++q) {
    if (!trans_valid(L[q], s, op.ip)) continue;
    int sign;
    state_t k = trans_apply(L[q], s, op.ip, sign);
    acc += vals[q] * (T)sign * x[sector_index(op, k)];
  }
  return acc;
}

// C elements of a row in registers
template <typename T, int C>
struct RowPart {
  T v[C];
};

// Off-diagonal interaction of C elements of an SRS row, columns d0, d0 + S, ... (those below Nd), added to a in the order of
// the terms: each up entry of the row (source row, down hop, term) by the entry of the down hop in each column, or, for a
// model without these tables, the transitions.  A Kanamori impurity has about four up entries per row, one in four of which
// meets a down hop of a column, where testing every transition on every state cost 24 state tests with two rank lookups
// per hit.  (Not inlined: models without such terms keep the registers.)
template <typename T, int C, int S>
__device__ __noinline__ RowPart<T, C> srs_vloc(const SectorOp<T> *opp, int u, int d0, const T *x, RowPart<T, C> a) {
  const SectorOp<T> &op = *opp;
  constexpr int U = 4;  // entries in flight
  const int Nd = op.dn_rows, ne = op.nW ? ldg_t(op.vu_cnt + u) : 0;
  for (int e = 0; e < ne; e += U) {
    int4 en[U];
    int to[U][C];
    T v[U], xv[U][C];
#pragma unroll
    for (int q = 0; q < U; ++q) en[q] = e + q < ne ? __ldg(op.vu_ent + (long long)u * op.nW + e + q) : make_int4(0, 0, -1, 0);
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const bool in = en[q].z >= 0;
      v[q] = in ? ldg_t(op.V_val + en[q].z) : T(0);
      if (en[q].w) v[q] = -v[q];
#pragma unroll
      for (int cc = 0; cc < C; ++cc) to[q][cc] = in && d0 + cc * S < Nd ? ldg_t(op.vd_to + en[q].y * op.dn_ld + d0 + cc * S) : -1;
    }
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int cc = 0; cc < C; ++cc)
        xv[q][cc] = to[q][cc] >= 0 ? x[(long long)en[q].x * Nd + (to[q][cc] >> 1)] : T(0);
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int cc = 0; cc < C; ++cc)
        if (to[q][cc] >= 0) a.v[cc] = madd(to[q][cc] & 1 ? -v[q] : v[q], xv[q][cc], a.v[cc]);
  }
  if (op.nV) {
    for (int cc = 0; cc < C; ++cc)
      if (d0 + cc * S < Nd) {
        const state_t s = ((state_t)op.up_basis[u] << op.ns) | (state_t)op.dn_basis[d0 + cc * S];
        T v = T(0);
#pragma unroll
        for (int q = 0; q < C; ++q)
          if (q == cc) v = a.v[q];
        v = transitions_term(op, s, op.V_, op.V_val, op.nV, x, v);
#pragma unroll
        for (int q = 0; q < C; ++q)
          if (q == cc) a.v[q] = v;
      }
  }
  return a;
}

// The same for R rows u, u + 1, ... (nr of them real) of one column: the rows' chains of loads run side by side.
template <typename T, int R>
__device__ __noinline__ RowPart<T, R> srs_vloc_rows(const SectorOp<T> *opp, int u, int nr, int d, const T *x,
                                                    RowPart<T, R> a) {
  const SectorOp<T> &op = *opp;
  constexpr int U = 2;
  int ne[R], nmax = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    ne[r] = op.nW && r < nr ? ldg_t(op.vu_cnt + u + r) : 0;
    nmax = max(nmax, ne[r]);
  }
  for (int e = 0; e < nmax; e += U) {
    int4 en[U][R];
    int to[U][R];
    T v[U][R], xv[U][R];
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r)
        en[q][r] = e + q < ne[r] ? __ldg(op.vu_ent + (long long)(u + r) * op.nW + e + q) : make_int4(0, 0, -1, 0);
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool in = en[q][r].z >= 0;
        v[q][r] = in ? ldg_t(op.V_val + en[q][r].z) : T(0);
        to[q][r] = in ? ldg_t(op.vd_to + en[q][r].y * op.dn_ld + d) : -1;
        if ((en[q][r].w ^ to[q][r]) & 1) v[q][r] = -v[q][r];
      }
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r)
        xv[q][r] = to[q][r] >= 0 ? x[(long long)en[q][r].x * op.dn_rows + (to[q][r] >> 1)] : T(0);
#pragma unroll
    for (int q = 0; q < U; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (to[q][r] >= 0) a.v[r] = madd(v[q][r], xv[q][r], a.v[r]);
  }
  if (op.nV) {
    for (int r = 0; r < nr; ++r) {
      const state_t s = ((state_t)op.up_basis[u + r] << op.ns) | (state_t)op.dn_basis[d];
      T v = T(0);
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (q == r) v = a.v[q];
      v = transitions_term(op, s, op.V_, op.V_val, op.nV, x, v);
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (q == r) a.v[q] = v;
    }
  }
  return a;
}

// What an item of a spin-resolved sector needs, in shared memory: one thread fetches it an item ahead, so that the
// chain of task, sector and pointers is off the block's critical path and out of its registers.
template <typename T>
struct SrsItem {
  const SectorOp<T> *op;
  const T *x, *xi, *dg, *z;  // the sector vector; its rows of this item, the diagonal's and z's (or null)
  T *y;
  const unsigned short *slot;
  const T *ev;
  const int *len, *urp;      // urp: from the item's first row on
  const Hop<T> *uh;
  double *dot;               // the item's part of <x, y>, or null
  T c;                       // y = H x + c z
  int Nd, ld, u0, nrows, vloc, skip;
  int together;              // short rows: a few rows of a column per thread (srs_short)
};

template <typename T>
__device__ __forceinline__ void fetch_item(SrsItem<T> &d, const SectorOp<T> *opp, int srs_rows, int li, const T *x, T *y,
                                           const T *z, T c, const LzTask<T> *lz) {
  const SectorOp<T> &op = *opp;
  const int Nd = op.dn_rows, u0 = li * srs_rows;
  const long long lo = (long long)u0 * Nd;
  d.op = opp;
  d.x = x;
  d.xi = x + lo;
  d.dg = op.diag + lo;
  d.z = z ? z + lo : nullptr;
  d.y = y + lo;
  d.slot = op.dn_slot;
  d.ev = op.dn_ell_val;
  d.len = op.dn_len;
  d.urp = op.up_rp + u0;
  d.uh = op.up_hop;
  d.dot = lz ? lz->part_a + li : nullptr;
  d.c = c;
  d.Nd = Nd;
  d.ld = op.dn_ld;
  d.u0 = u0;
  d.nrows = min(srs_rows, op.up_rows - u0);
  d.vloc = op.nW != 0 || op.nV != 0;
  d.together = sizeof(T) == 4 ? op.up_kmax <= 16 : d.vloc;
  d.skip = srs_two_pass(op.up_rows, Nd);  // k_srs_long's
}

// A recurrence's operator starts before the kernel that writes its x has ended (launch_pdl), and the read-only path
// (ldg_t) asks for data that nobody writes while the kernel lives: x and z are read by ordinary loads, tables and the
// diagonal through the read-only path.  Tiles of other launches read x through it too (RO; 495-state rows 106 instead of
// 111 us).

// C consecutive vector elements (16 bytes: 4 FP32 or 2 FP64) in one load when `vec` is set (the caller
// guarantees the alignment); a ragged end (n < C) is read element by element.
template <typename T>
__device__ __forceinline__ Lanes<T> load_lanes(const T *p, bool vec, int n) {
  Lanes<T> q;
  if (vec && n == Lanes<T>::C) {
    if constexpr (std::is_same<T, ffloat>::value) {
      const float4 f = ldg_t(reinterpret_cast<const float4 *>(p));
      q.v[0] = ffloat(f.x, f.y), q.v[1] = ffloat(f.z, f.w);
    } else if constexpr (sizeof(T) == 4) {
      const float4 f = ldg_t(reinterpret_cast<const float4 *>(p));
      q.v[0] = f.x, q.v[1] = f.y, q.v[2] = f.z, q.v[3] = f.w;
    } else {
      const double2 f = ldg_t(reinterpret_cast<const double2 *>(p));
      q.v[0] = f.x, q.v[1] = f.y;
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < Lanes<T>::C; ++cc) q.v[cc] = cc < n ? p[cc] : (T)0;
  }
  return q;
}

// C consecutive ints of a k-major table (16 bytes for C = 4, 8 for C = 2; always aligned: the table's
// leading dimension is a multiple of 4 and column tiles start at multiples of C).
template <int C>
__device__ __forceinline__ Lanes<int> load_ints(const int *p) {
  Lanes<int> q;
  if constexpr (C == 4) {
    const int4 f = ldg_t(reinterpret_cast<const int4 *>(p));
    q.v[0] = f.x, q.v[1] = f.y, q.v[2] = f.z, q.v[3] = f.w;
  } else {
    const int2 f = ldg_t(reinterpret_cast<const int2 *>(p));
    q.v[0] = f.x, q.v[1] = f.y;
  }
  return q;
}

// One hop table entry (column or source row, value) in one load.
__device__ __forceinline__ Hop<float> ldg_hop(const Hop<float> *p) {
  const int2 t = __ldg(reinterpret_cast<const int2 *>(p));
  return Hop<float>{t.x, __int_as_float(t.y)};
}
__device__ __forceinline__ Hop<double> ldg_hop(const Hop<double> *p) {
  const int4 t = __ldg(reinterpret_cast<const int4 *>(p));
  return Hop<double>{t.x, 0, __hiloint2double(t.w, t.z)};
}
__device__ __forceinline__ Hop<ffloat> ldg_hop(const Hop<ffloat> *p) {
  const int4 t = __ldg(reinterpret_cast<const int4 *>(p));
  return Hop<ffloat>{t.x, 0, ffloat(__int_as_float(t.z), __int_as_float(t.w))};
}

// 16 bytes through the read-only path
template <typename T>
__device__ __forceinline__ Lanes<T> ldg16(const T *p) {
  return load_lanes(p, true, Lanes<T>::C);
}
// A lane's C elements of a row: 16 consecutive bytes (VEC), or elements o apart from p; RO: through the read-only path
// (z may be the vector being written).
template <typename T, int C, bool VEC, bool RO = true>
__device__ __forceinline__ void ld_tile(const T *p, const int (&o)[C], T (&v)[C]) {
  if constexpr (VEC) {
    const Lanes<T> q = RO ? ldg16(p) : load16(p);
#pragma unroll
    for (int cc = 0; cc < C; ++cc) v[cc] = q.v[cc];
  } else {
#pragma unroll
    for (int cc = 0; cc < C; ++cc) v[cc] = RO ? ldg_t(p + o[cc]) : p[o[cc]];
  }
}

// Geometry of an SRS tile: R up rows x W = 32 C columns per warp.  In shared memory RI rows (16 bytes of one column)
// are interleaved: row r, column d of the item at xs[((r / RI) Nd + slot(d)) RI + r % RI], so that one 16-byte load
// fetches a down-hop's source column for RI rows.  slot (tile_slot) puts every C-th column side by side in rows of a
// multiple of C states, whose tiles hold C consecutive columns per lane; the hop tables name slots.
template <typename T>
struct TileGeom {
  static constexpr int R = 4, C = sizeof(T) == 4 ? 4 : 2, W = 32 * C, RI = 16 / (int)sizeof(T), NP = R / RI;
};

// How a tile's lanes hold columns: kVec, lane l the C columns from C l on, every global access 16 bytes per lane
// (rows of whole 16-byte pieces on aligned bases); kOdd, lane l columns l, l + 32, ..., rows of any other length;
// kOff, as kOdd for rows of whole 16-byte pieces off 16-byte bases.
enum TileMode { kVec, kOdd, kOff };

// Rows [0, nrows) of Nd elements from x into the interleaved layout; the interleaved slots past the last row are zero.
template <typename T, int M, bool RO>
__device__ __forceinline__ void stage_interleaved(T *xs, const T *x, int nrows, int Nd) {
  constexpr int RI = TileGeom<T>::RI, C = TileGeom<T>::C;
  const int nq = (nrows + RI - 1) / RI;
  Lanes<T> *out = reinterpret_cast<Lanes<T> *>(xs);
  if constexpr (M == kVec) {
    const int Nq = Nd / C;  // C consecutive columns of RI rows, transposed in registers
    int q = threadIdx.x / Nq, d = threadIdx.x - q * Nq;
#pragma unroll 1
    for (int e = threadIdx.x; e < nq * Nq; e += kMvBlock) {
      Lanes<T> v[RI];
#pragma unroll
      for (int i = 0; i < RI; ++i) v[i] = q * RI + i < nrows ? (RO ? ldg16(x + (q * RI + i) * Nd + C * d) : load16(x + (q * RI + i) * Nd + C * d)) : Lanes<T>{};
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        Lanes<T> w;
#pragma unroll
        for (int i = 0; i < RI; ++i) w.v[i] = v[i].v[cc];
        out[q * Nd + cc * Nq + d] = w;
      }
      for (d += kMvBlock; d >= Nq; d -= Nq) ++q;
    }
  } else {
    int q = threadIdx.x / Nd, d = threadIdx.x - q * Nd;
    const int qs = kMvBlock / Nd, ds = kMvBlock - qs * Nd;
#pragma unroll 4
    for (int e = threadIdx.x; e < nq * Nd; e += kMvBlock) {
      Lanes<T> v;
#pragma unroll
      for (int i = 0; i < RI; ++i) v.v[i] = q * RI + i < nrows ? (RO ? ldg_t(x + (q * RI + i) * Nd + d) : x[(q * RI + i) * Nd + d]) : T(0);
      out[q * Nd + (M == kOdd ? d : tile_slot(d, Nd, C))] = v;
      q += qs;
      d += ds;
      if (d >= Nd) d -= Nd, ++q;
    }
  }
}

// The C slots and values of one k-major entry row for a lane's columns (16-byte pieces when VEC).
template <typename T, int C, bool VEC>
__device__ __forceinline__ void ld_entry(const unsigned short *slot, const T *val, const int (&o)[C], int (&c)[C], T (&v)[C]) {
  if constexpr (VEC && C == 4) {
    const uint2 q = __ldg(reinterpret_cast<const uint2 *>(slot));
    c[0] = q.x & 0xffff, c[1] = q.x >> 16, c[2] = q.y & 0xffff, c[3] = q.y >> 16;
  } else if constexpr (VEC) {
    const unsigned q = __ldg(reinterpret_cast<const unsigned *>(slot));
    c[0] = q & 0xffff, c[1] = q >> 16;
  } else {
#pragma unroll
    for (int cc = 0; cc < C; ++cc) c[cc] = __ldg(slot + o[cc]);
  }
  ld_tile<T, C, VEC>(val, o, v);
}

// The up hops of an item in shared memory: row r's at [rp[r], rp[r + 1]), c = the source row's offset in x;
// one entry of value 0 behind them.
template <typename T>
struct ItemHops {
  Hop<T> *hop;
  int *rp;
};

// A thread's part of a tile of the SRS sweep: rows rg .. rg + 3 of the item (those below nrows), columns from c0 on
// (kVec: C consecutive ones; else 32 apart).  Columns below cb are another tile's, columns past the row's end (MD; `mine`
// says whether c0 is one) repeat the last, and so do rows past the item's end; all of them store nothing: every load is
// in bounds without a predicate.
// What bounds it: L1 and shared-memory wavefronts, then issue slots.  Rows apart in shared memory (each down-hop
// entry 16 address computations and 16 scalar loads per thread) took 110 thread instructions per state.  Here an
// entry is one 16-byte shared-memory load per column for RI rows, and the item's up hops come from shared memory, HB
// of them in flight per row.  Rows of 924 or 792 states start off 128-byte lines, where a warp's 4-byte accesses
// touch two lines each: those take 16-byte accesses (the 64-vector product of the 12-orbital sector (6,6): 428 us with
// 4-byte ones).
// Per element the sum runs diagonal, (c z), down hops and up hops each in the reference's order, interaction: another
// order (down hops dealt out so that a phase's eight lanes meet few bank conflicts) is faster, but the eigen-solver's
// and the recurrences' vectors are then others in the last bit, which unconverged quantities magnify.
template <typename T, int M, int HB, bool MZ, bool MD, bool RO>
__device__ __forceinline__ void srs_tile(const SrsItem<T> &it, const ItemHops<T> &hops, int rg, int cb, int c0, bool mine,
                                         const T *__restrict__ xs, DotAcc &acc) {
  using TG = TileGeom<T>;
  constexpr bool VEC = M == kVec;
  constexpr int R = TG::R, C = TG::C, RI = TG::RI, NP = TG::NP;
  const int Nd = it.Nd;
  const Lanes<T> *__restrict__ xv = reinterpret_cast<const Lanes<T> *>(xs) + (rg / RI) * Nd;
  int o[C];  // the columns, from c0
#pragma unroll
  for (int cc = 0; cc < C; ++cc) o[cc] = VEC ? cc : MD ? min(32 * cc, Nd - 1 - c0) : 32 * cc;
  auto own = [&](int cc) { return VEC ? true : MD ? c0 + 32 * cc < Nd : c0 + 32 * cc >= cb; };
  auto slot = [&](int cc) { return VEC ? c0 / C + cc * (Nd / C) : M == kOdd ? c0 + o[cc] : tile_slot(c0 + o[cc], Nd, C); };
  auto row = [&](int r) { return min(rg + r, it.nrows - 1) * Nd + c0; };
  T a[R][C];
#pragma unroll
  for (int r = 0; r < R; ++r) ld_tile<T, C, VEC>(it.dg + row(r), o, a[r]);
  if (MZ && it.z) {
    // a + c z; whole groups of four rows and rows of no whole 16-byte pieces round c z first, others the diagonal's term
    const bool first = !VEC || rg + R <= it.nrows;
    T zq[R][C];
#pragma unroll
    for (int r = 0; r < R; ++r) ld_tile<T, C, VEC, false>(it.z + row(r), o, zq[r]);
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        const Lanes<T> q = xv[p * Nd + slot(cc)];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          T &e = a[p * RI + i][cc];
          const T z = zq[p * RI + i][cc];
          if constexpr (std::is_same<T, ffloat>::value) e = e * q.v[i] + it.c * z;
          else e = first ? madd(e, q.v[i], mul_rn(it.c, z)) : madd(it.c, z, mul_rn(e, q.v[i]));
        }
      }
  } else {
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        const Lanes<T> q = xv[p * Nd + slot(cc)];
#pragma unroll
        for (int i = 0; i < RI; ++i) a[p * RI + i][cc] = mul_rn(a[p * RI + i][cc], q.v[i]);
      }
  }
  {
    int kk = 0;
#pragma unroll
    for (int cc = 0; cc < C; ++cc) kk = max(kk, ldg_t(it.len + c0 + o[cc]));
    if (!mine) kk = 0;  // lanes past the row's end sum nothing
    const unsigned short *__restrict__ es = it.slot + c0;
    const T *__restrict__ ev = it.ev + c0;
    const int ld = it.ld;
    int hc[C];
    T hv[C];
    if (kk > 0) ld_entry<T, C, VEC>(es, ev, o, hc, hv);
#pragma unroll 1
    for (int k = 0; k < kk; ++k) {
      int nc[C];
      T nv[C];
      es += ld;
      ev += ld;
      if (k + 1 < kk) ld_entry<T, C, VEC>(es, ev, o, nc, nv);
#pragma unroll
      for (int cc = 0; cc < C; ++cc)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const Lanes<T> q = xv[p * Nd + hc[cc]];
#pragma unroll
          for (int i = 0; i < RI; ++i) a[p * RI + i][cc] = madd(hv[cc], q.v[i], a[p * RI + i][cc]);
        }
#pragma unroll
      for (int cc = 0; cc < C; ++cc) hc[cc] = nc[cc], hv[cc] = nv[cc];
    }
  }
  {
    const int none = hops.rp[it.nrows];  // the entry past the item's hops: row 0, value 0
    int k0[R], n[R], nmax = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = min(rg + r, it.nrows - 1);
      k0[r] = hops.rp[q];
      n[r] = hops.rp[q + 1] - k0[r];
      nmax = max(nmax, n[r]);
    }
    if (!mine) nmax = 0;
    const T *xc = it.x + c0;
#pragma unroll 1
    for (int h = 0; h < nmax; h += HB) {
      T xq[R][HB][C], v[R][HB];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < HB; ++q) {
          const Hop<T> hp = hops.hop[h + q < n[r] ? k0[r] + h + q : none];
          v[r][q] = hp.v;
          ld_tile<T, C, VEC, RO>(xc + hp.c, o, xq[r][q]);
        }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < HB; ++q)
          if (h + q < n[r]) {  // uniform over the warp
#pragma unroll
            for (int cc = 0; cc < C; ++cc) a[r][cc] = madd(v[r][q], xq[r][q][cc], a[r][cc]);
          }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (rg + r >= it.nrows) continue;
    if (it.vloc) {
      RowPart<T, C> p;
#pragma unroll
      for (int cc = 0; cc < C; ++cc) p.v[cc] = a[r][cc];
      p = srs_vloc<T, C, VEC ? 1 : 32>(it.op, it.u0 + rg + r, c0, it.x, p);
#pragma unroll
      for (int cc = 0; cc < C; ++cc) a[r][cc] = p.v[cc];
    }
    T *__restrict__ y = it.y + row(r);
    if constexpr (VEC) {
      store_lanes(y, a[r]);
    } else {
#pragma unroll
      for (int cc = 0; cc < C; ++cc)
        if (own(cc)) y[o[cc]] = renorm(a[r][cc]);
    }
    if (MD && it.dot) {
#pragma unroll
      for (int cc = 0; cc < C; ++cc)
        if (own(cc)) dot_add(acc, xv[(r / RI) * Nd + slot(cc)].v[r % RI], a[r][cc]);
    }
  }
}

// The tiles of a staged item; the thread's part of <x, y>.  kVec: the item's units of 4 rows x C columns numbered through, a
// thread each, rows ending inside a warp.  (A warp per tile of 4 rows x W columns, the last columns taken twice past the
// row's end, is 1 % faster on FP32 rows of 220 or 560 states, the same on 252, 792, 816, 924 and 1716, and 25 % slower on
// 680.)  Other modes: a warp per tile, so that its accesses are whole lines; the last tile moves back to end with the row,
// but with dot products (MD), where a thread's elements are part of the sums' values, its columns past the end repeat the
// last.
template <typename T, int M, int HB, bool MZ, bool MD, bool RO>
__device__ __forceinline__ DotAcc srs_tiles(const SrsItem<T> &it, const ItemHops<T> &hops, const T *__restrict__ xs) {
  using TG = TileGeom<T>;
  constexpr int C = TG::C;
  constexpr bool linear = M == kVec;
  DotAcc acc;
  dot_init(acc);
  const int ngr = (it.nrows + TG::R - 1) / TG::R, per = linear ? it.Nd / C : (it.Nd + TG::W - 1) / TG::W;
#pragma unroll 1
  for (int unit = linear ? threadIdx.x : threadIdx.x >> 5; unit < ngr * per; unit += linear ? kMvBlock : kMvBlock / 32) {
    const int g = unit / per, q = unit - g * per, cb = linear ? 0 : q * TG::W;
    const int c0 = linear ? q * C : (MD ? cb : min(cb, it.Nd - TG::W)) + (threadIdx.x & 31);
    srs_tile<T, M, HB, MZ, MD, RO>(it, hops, g * TG::R, cb, c0, c0 < it.Nd, xs, acc);
  }
  return acc;
}
// tiles off 16-byte bases apart from the others, with registers of their own
template <typename T, bool MZ, bool MD, bool RO>
__device__ __noinline__ DotAcc srs_tiles_off(const SrsItem<T> &it, const ItemHops<T> &hops, const T *__restrict__ xs) {
  return srs_tiles<T, kOff, 1, MZ, MD, RO>(it, hops, xs);
}

// SRS item of very long rows (one to three rows per item, each staged in shared memory): one row at a time,
// its up-spin hop list (source-row offsets and values) copied once to shared memory for the whole block, and
// each thread sweeping C-column quads of the row: diagonal (c z), the down hops from the staged row through
// the k-major copy, the up hops as gathers of the quad from each source row (8-byte pieces when rows have an
// even length), the interaction.  The same sums in the same order as the tiled paths.  For rows of 10^4
// states a four-row tile does not stage in shared memory.  Rows with more than kLongHops up hops take the rest of
// the list from global memory.
constexpr int kLongHops = 128;
template <typename T, bool MZ, bool MD>
__device__ __noinline__ DotAcc srs_longrow(const SrsItem<T> &it, const T *__restrict__ xs) {
  const SectorOp<T> &op = *it.op;
  const T *x = it.x, *z = it.z;
  T *y = it.y;
  const T c = it.c;
  const int u0 = it.u0, nrows = it.nrows;
  DotAcc acc;
  dot_init(acc);
  constexpr int C = Lanes<T>::C;
  __shared__ long long hop_off[kLongHops];
  __shared__ T hop_val[kLongHops];
  const int Nd = op.dn_rows;
  const bool even = (Nd & 1) == 0 && ((uintptr_t)x & 7) == 0;
  const int *__restrict__ elen = op.dn_len;
  const int *__restrict__ ecol = op.dn_ell_col;
  const T *__restrict__ eval = op.dn_ell_val;
  const int eld = op.dn_ld;
  for (int r = 0; r < nrows; ++r) {
    const int u = u0 + r;
    const int k0 = ldg_t(op.up_rp + u), nall = ldg_t(op.up_rp + u + 1) - k0, nh = min(nall, kLongHops);
    __syncthreads();  // the previous row's hop list is no longer read
    for (int h = threadIdx.x; h < nh; h += blockDim.x) {
      hop_off[h] = (long long)ldg_t(op.up_col + k0 + h) * Nd;
      hop_val[h] = ldg_t(op.up_val + k0 + h);
    }
    __syncthreads();
    const T *__restrict__ xrow = xs + (long long)r * Nd;
    const long long rowbase = (long long)r * Nd;
    for (int d0 = C * threadIdx.x; d0 < Nd; d0 += C * blockDim.x) {
      const int nc = min(C, Nd - d0);
      T a[C];
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        const bool in = cc < nc;
        a[cc] = in ? ldg_t(it.dg + rowbase + d0 + cc) * xrow[d0 + cc] : (T)0;
        if (MZ && z && in) a[cc] = a[cc] + c * z[rowbase + d0 + cc];
      }
      {  // down hops: entry k of the quad's columns in one 16-byte load each of columns and values
        const Lanes<int> lq = load_ints<C>(elen + d0);
        int kk = lq.v[0];
#pragma unroll
        for (int cc = 1; cc < C; ++cc) kk = max(kk, lq.v[cc]);
        for (int k = 0; k < kk; ++k) {
          const Lanes<int> cq = load_ints<C>(ecol + k * eld + d0);
          const Lanes<T> vq = load_lanes(eval + k * eld + d0, true, C);
#pragma unroll
          for (int cc = 0; cc < C; ++cc)
            if (k < lq.v[cc]) a[cc] += vq.v[cc] * xrow[cq.v[cc]];
        }
      }
      // up hops: the quad of every source row, four hops' loads in flight
      if (nc == C && even) {
        for (int h = 0; h < nh; h += 4) {
          Lanes<T> xq[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int hq = h + q < nh ? h + q : h;
            const T *src = x + hop_off[hq] + d0;
            if constexpr (sizeof(T) == 4) {
              const float2 p0 = *reinterpret_cast<const float2 *>(src), p1 = *reinterpret_cast<const float2 *>(src + 2);
              xq[q].v[0] = p0.x, xq[q].v[1] = p0.y, xq[q].v[2] = p1.x, xq[q].v[3] = p1.y;
            } else {
              xq[q].v[0] = src[0];
              xq[q].v[1] = src[1];
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (h + q < nh) {
              const T v = hop_val[h + q];
#pragma unroll
              for (int cc = 0; cc < C; ++cc) a[cc] += v * xq[q].v[cc];
            }
        }
      } else {
        for (int h = 0; h < nh; ++h) {
          const T v = hop_val[h];
          const T *src = x + hop_off[h] + d0;
#pragma unroll
          for (int cc = 0; cc < C; ++cc)
            if (cc < nc) a[cc] += v * src[cc];
        }
      }
      for (int h = nh; h < nall; ++h) {
        const T v = ldg_t(op.up_val + k0 + h);
        const T *src = x + (long long)ldg_t(op.up_col + k0 + h) * Nd + d0;
#pragma unroll
        for (int cc = 0; cc < C; ++cc)
          if (cc < nc) a[cc] += v * src[cc];
      }
      if (op.nW != 0 || op.nV != 0) {
        RowPart<T, C> p;
#pragma unroll
        for (int cc = 0; cc < C; ++cc) p.v[cc] = a[cc];
        p = srs_vloc<T, C, 1>(&op, u, d0, x, p);
#pragma unroll
        for (int cc = 0; cc < C; ++cc) a[cc] = p.v[cc];
      }
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        if (cc < nc) {
          y[rowbase + d0 + cc] = renorm(a[cc]);
          if (MD && it.dot) dot_add(acc, xrow[d0 + cc], a[cc]);
        }
      }
    }
  }
  return acc;
}

// SRS item of short rows (below kSrsLongRow states), staged like a tile's (stage_interleaved, slots in column order):
// a thread takes one column of RI rows at a time, so that rows shorter than a warp keep every thread busy and each
// down-hop entry, loaded once, serves RI rows; or (srs_flat, rows as they are) one element at a time.  Per element the sums
// of the tiles, in the reference's order.  Columns of rows for FP32 vectors of few up hops per row (32 vectors, 12-orbital
// impurity, rows of 66 states 39 us, one element at a time 41; but 14-site ring, rows of 91: 160 and 147), which nothing is
// shared of where they are many (16-site square cluster, 8 vectors, rows of 16 states: 121 and 66 us); 8-byte types, bound by
// arithmetic, one element at a time (rows of 66 states 95 and 83 us) but with interaction terms, whose chains of loads run
// side by side for the rows (G of the 8-orbital Kanamori impurity 4.46 and 4.67 ms).
template <typename T, bool MZ>
__device__ __noinline__ void srs_short(const SrsItem<T> &it, const ItemHops<T> &hops, bool near, const T *__restrict__ xs) {
  constexpr int RI = Lanes<T>::C;
  const SectorOp<T> &op = *it.op;
  const Lanes<T> *__restrict__ xv = reinterpret_cast<const Lanes<T> *>(xs);
  const int Nd = it.Nd, ld = it.ld, n = (it.nrows + RI - 1) / RI * Nd;
  const int *__restrict__ ecol = op.dn_ell_col;
  const T *__restrict__ eval = op.dn_ell_val;
  int g = threadIdx.x / Nd, d = threadIdx.x - g * Nd;
  const int gs = kMvBlock / Nd, ds = kMvBlock - gs * Nd;
  for (int e = threadIdx.x; e < n; e += kMvBlock) {
    const int nr = min(RI, it.nrows - g * RI);
    const Lanes<T> *__restrict__ xg = xv + g * Nd;
    const Lanes<T> own = xg[d];
    int ro[RI];  // rows past the item's end repeat its last one and store nothing
#pragma unroll
    for (int r = 0; r < RI; ++r) ro[r] = (g * RI + min(r, nr - 1)) * Nd + d;
    T a[RI];
#pragma unroll
    for (int r = 0; r < RI; ++r) a[r] = mul_rn(ldg_t(it.dg + ro[r]), own.v[r]);
    if (MZ && it.z) {
#pragma unroll
      for (int r = 0; r < RI; ++r) a[r] = madd(it.c, it.z[ro[r]], a[r]);
    }
    const int kk = ldg_t(it.len + d);
#pragma unroll 4
    for (int k = 0; k < kk; ++k) {
      const Lanes<T> q = xg[ldg_t(ecol + k * ld + d)];
      const T v = ldg_t(eval + k * ld + d);
#pragma unroll
      for (int r = 0; r < RI; ++r) a[r] = madd(v, q.v[r], a[r]);
    }
    int k0[RI], nh[RI], nmax = 0;
#pragma unroll
    for (int r = 0; r < RI; ++r) {
      const int *p = it.urp + g * RI + min(r, nr - 1);
      k0[r] = ldg_t(p);
      nh[r] = ldg_t(p + 1) - k0[r];
      nmax = max(nmax, nh[r]);
    }
    const T *xd = it.x + d;
    const int first = ldg_t(it.urp);
#pragma unroll 1
    for (int h = 0; h < nmax; h += 4) {
      T v[4][RI], xq[4][RI];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < RI; ++r) {
          v[q][r] = xq[q][r] = T(0);
          if (h + q < nh[r]) {
            Hop<T> hp;
            if (near) {
              hp = hops.hop[k0[r] - first + h + q];
            } else {
              hp = ldg_hop(it.uh + k0[r] + h + q);
              hp.c *= Nd;
            }
            v[q][r] = hp.v;
            xq[q][r] = xd[hp.c];
          }
        }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < RI; ++r)
          if (h + q < nh[r]) a[r] = madd(v[q][r], xq[q][r], a[r]);
    }
    if (it.vloc) {
      RowPart<T, RI> p;
#pragma unroll
      for (int r = 0; r < RI; ++r) p.v[r] = a[r];
      p = srs_vloc_rows<T, RI>(it.op, it.u0 + g * RI, nr, d, it.x, p);
#pragma unroll
      for (int r = 0; r < RI; ++r) a[r] = p.v[r];
    }
#pragma unroll
    for (int r = 0; r < RI; ++r) {
      if (r >= nr) continue;
      it.y[ro[r]] = renorm(a[r]);
    }
    g += gs;
    d += ds;
    if (d >= Nd) d -= Nd, ++g;
  }
}

// A thread takes one element at a time, e = threadIdx.x, + kMvBlock, ... over the item, which with dot products (MD) is part
// of the value of <x, y>.  The item's rows are copied as they are: interleaved like the others' they came through registers
// and cost twice the shared-memory wavefronts (G of the 9-orbital impurity, FP64, 4.43 -> 4.19 ms).
template <typename T, bool MZ, bool MD>
__device__ __noinline__ DotAcc srs_flat(const SrsItem<T> &it, const ItemHops<T> &hops, bool near, const T *__restrict__ xs) {
  const SectorOp<T> &op = *it.op;
  const int Nd = it.Nd, ld = it.ld, n = it.nrows * Nd, first = ldg_t(it.urp);
  const int *__restrict__ ecol = op.dn_ell_col;
  const T *__restrict__ eval = op.dn_ell_val;
  DotAcc acc;
  dot_init(acc);
  int r = threadIdx.x / Nd, d = threadIdx.x - r * Nd;
  const int rs = kMvBlock / Nd, ds = kMvBlock - rs * Nd;
  for (int e = threadIdx.x; e < n; e += kMvBlock) {
    const T *__restrict__ xg = xs + r * Nd;
    const T xv = xg[d];
    T a = mul_rn(ldg_t(it.dg + e), xv);
    if (MZ && it.z) a = madd(it.c, it.z[e], a);
    const int kk = ldg_t(it.len + d);
#pragma unroll 4
    for (int k = 0; k < kk; ++k) a = madd(ldg_t(eval + k * ld + d), xg[ldg_t(ecol + k * ld + d)], a);
    const int k0 = ldg_t(it.urp + r), nh = ldg_t(it.urp + r + 1) - k0;
    const T *xd = it.x + d;
    if (near) {
#pragma unroll 4
      for (int h = 0; h < nh; ++h) {
        const Hop<T> hp = hops.hop[k0 - first + h];
        a = madd(hp.v, xd[hp.c], a);
      }
    } else {
#pragma unroll 8
      for (int h = 0; h < nh; ++h) {
        const Hop<T> hp = ldg_hop(it.uh + k0 + h);
        a = madd(hp.v, xd[hp.c * Nd], a);
      }
    }
    if (it.vloc) a = srs_vloc<T, 1, 1>(it.op, it.u0 + r, d, it.x, RowPart<T, 1>{{a}}).v[0];
    it.y[e] = renorm(a);
    if (MD && it.dot) dot_add(acc, xv, a);
    r += rs;
    d += ds;
    if (d >= Nd) d -= Nd, ++r;
  }
  return acc;
}

// One item of a sector: y[lo:hi) = (H x)[lo:hi) + c z[lo:hi), a thread per row, the row added in its own order, U of its
// entries (CRS) or transitions (SOCRS, tested by their masks: TransMask) with their loads in flight.  Items are small
// enough for every SM (row_item): 4900 rows of 17 entries, one FP64 vector, 27 us cold in three items of 2048 rows.
// Several lanes per row, reading its entries side by side, add by a butterfly (another sum) or hand all entries around,
// and then every lane adds all of them: FP64 issue, two lanes per clock and SM, bounds that (63,504 CRS rows, 15 FP64
// vectors: 129 us with four lanes per row).
template <typename T, int ST>
__device__ __forceinline__ void mv_item(const SectorOp<T> *opp, int rows, long long li, const T *x, T *y, const T *z, T c) {
  const SectorOp<T> &op = *opp;
  constexpr int U = ST == kCRS ? 4 : 4;
  long long lo, hi;
  item_range(op, rows, li, lo, hi);
  if constexpr (ST == kCRS) {
    for (long long i = lo + threadIdx.x; i < hi; i += kMvBlock) {
      const long long j1 = op.crs_rp[i + 1];
      T v = z ? mul_rn(c, z[i]) : T(0);
      for (long long j = op.crs_rp[i]; j < j1; j += U) {
        T a[U], b[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const bool in = j + k < j1;
          a[k] = in ? ldg_t(op.crs_val + j + k) : T(0);
          b[k] = in ? x[__ldg(op.crs_col + j + k)] : T(0);
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (j + k < j1) v = madd(a[k], b[k], v);
      }
      y[i] = v;
    }
  } else {
    const unsigned Nd = (unsigned)op.dn_rows;
    for (long long i = lo + threadIdx.x; i < hi; i += kMvBlock) {
      const long long u = op.dim <= 0xffffffffll ? (unsigned)i / Nd : i / Nd;
      const unsigned d = (unsigned)(i - u * Nd);
      const unsigned long long s = ((unsigned long long)__ldg(op.up_basis + u) << op.ns) | (unsigned)__ldg(op.dn_basis + d);
      T v = mul_rn(ldg_t(op.diag + i), x[i]);
      if (z) v = madd(c, z[i], v);
      for (int k0 = 0; k0 < op.nM; k0 += U) {
        T m[U], b[U];
        bool hit[U];
#pragma unroll
        for (int p = 0; p < U; ++p) {
          const int k = min(k0 + p, op.nM - 1);
          const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2 *>(op.M_ + k));
          const ulonglong2 f = __ldg(reinterpret_cast<const ulonglong2 *>(op.M_ + k) + 1);
          hit[p] = k0 + p < op.nM && (s & a.y) == a.x;
          const unsigned long long t = s ^ f.x;
          m[p] = ldg_t(op.M_val + k);
          if (__popcll(s & f.y) & 1) m[p] = -m[p];
          b[p] = T(0);
          if (hit[p])
            b[p] = x[(long long)__ldg(op.ninv_up + (t >> op.ns)) * Nd + __ldg(op.ninv_dn + (t & ((1ull << op.ns) - 1)))];
        }
#pragma unroll
        for (int p = 0; p < U; ++p)
          if (hit[p]) v = madd(m[p], b[p], v);
      }
      y[i] = v;
    }
  }
}

// <x, y> of an item into its recurrence's parts
template <int NT>
__device__ __forceinline__ void emit_dot(DotAcc &acc, double *dst, double *red) {
  const double s = block_sum<NT>(dot_value(acc), red);
  if (threadIdx.x == 0) *dst = s;
}

// ---------------------------------------------------------------- where an operator launch's items come from
// get(it, f): f(op, srs_rows, li, x, y, z, c, lz) for item it: y = H x + c z, <x, y> into lz's parts where lz is given, or
// false where its task has nothing to do.  kEarly: its launches may be launch_pdl's.

// generic batch: y = H x (+ c z)
template <typename T>
struct MvSource {
  static constexpr bool kEarly = false;
  const MvTask<T> *tasks;
  const int *item_task;
  template <class F>
  __device__ __forceinline__ bool get(int it, F &&f) const {
    const MvTask<T> &t = tasks[item_task[it]];
    const int li = it - t.item_begin;
    f(t.op, t.srs_rows, li, t.x, t.y, t.z, (T)t.c, (const LzTask<T> *)nullptr);
    return true;
  }
};

// nvec vectors of one sector, ld apart: y_q = H x_q, or y_q += H x_q -- no task list to build or copy
template <typename T>
struct VecSource {
  static constexpr bool kEarly = false;
  const SectorOp<T> *op;
  const T *x;
  T *y;
  long long ld;
  int rows, per;  // rows per item, items per vector
  bool acc;
  template <class F>
  __device__ __forceinline__ bool get(int it, F &&f) const {
    const int q = it / per;
    T *yq = y + q * ld;
    f(op, rows, it - q * per, x + q * ld, yq, acc ? yq : nullptr, T(1), (const LzTask<T> *)nullptr);
    return true;
  }
};

// Lanczos recurrence, phase 1.  Iteration iter (0-based) of Lanczos.h:44-68: v = buf[iter % 3],
// w = buf[(iter + 1) % 3] = H v - bet buf[(iter + 2) % 3], and <v, w> unless SPLIT (LzBatch); a finished recurrence has
// nothing to do.
template <typename T, bool SPLIT>
struct LzSource {
  static constexpr bool kEarly = true;
  const LzTask<T> *tasks;
  const int *item_task;
  int iter;
  template <class F>
  __device__ __forceinline__ bool get(int it, F &&f) const {
    const LzTask<T> &t = tasks[item_task[it]];
    if (t.state[0]) return false;
    f(t.op, SPLIT ? t.mv_rows : t.srs_rows, it - (SPLIT ? t.mv_begin : t.item_begin), t.buf[iter % 3], t.buf[(iter + 1) % 3],
      iter == 0 ? nullptr : t.buf[(iter + 2) % 3], (T)(-t.scal[0]), SPLIT ? (const LzTask<T> *)nullptr : &t);
    return true;
  }
};

// eigen-solver step, phase 1: w = H V[j] for tasks in Lanczos mode that still grow their basis.  probe_y (the
// operator tuner): every task, x = V[0], into probe_y (shared scratch: the values are not used).
template <typename T>
struct EigSource {
  static constexpr bool kEarly = false;
  const EigTask<T> *tasks;
  const int *item_task;
  T *probe_y;
  template <class F>
  __device__ __forceinline__ bool get(int it, F &&f) const {
    const EigTask<T> &t = tasks[item_task[it]];
    if (!probe_y && (t.st[2] || t.st[1] != 0)) return false;  // full, or orthogonalising a random vector
    f(t.op, t.srs_rows, it - t.item_begin, probe_y ? t.V : t.V + (long long)t.st[0] * t.ldv, probe_y ? probe_y : t.w,
      (const T *)nullptr, T(0), (const LzTask<T> *)nullptr);
    return true;
  }
};

// Spin-resolved items.  MZ / MD: the launch may carry a z term / may want dot products (false removes those paths
// at compile time); HB: up hops in flight per row of a tile; MB: resident blocks per SM its registers are held to.
template <typename T, class Src, bool MZ, bool MD, int HB, int MB>
__global__ void __launch_bounds__(kMvBlock, MB) k_srs_mv(Src src, int nitems, int xs_cap, int hop_cap) {
  constexpr bool RO = !Src::kEarly;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SrsItem<T> items[2];
  __shared__ double red[kMvBlock / 32];
  __shared__ int hop_rp[kTileRows + 1];
  T *xs = reinterpret_cast<T *>(smem_raw);
  const ItemHops<T> hops{reinterpret_cast<Hop<T> *>(smem_raw + align16(sizeof(T) * (size_t)xs_cap)), hop_rp};
  // items from the last on: the batches list their sectors by size, and the largest items first leave the shortest tail
  auto fetch = [&](int i, SrsItem<T> &d) {
    if (i < nitems && !src.get(nitems - 1 - i, [&](const SectorOp<T> *op, int srs_rows, int li, const T *x, T *y, const T *z, T c, const LzTask<T> *lz) {
          fetch_item<T>(d, op, srs_rows, li, x, y, MZ ? z : nullptr, c, MD ? lz : nullptr);
        }))
      d.skip = 1;
  };
  if constexpr (Src::kEarly) pdl_enter();
  if (threadIdx.x == 0) fetch(blockIdx.x, items[0]);
  __syncthreads();
  int p = 0;
#pragma unroll 1
  for (int i = blockIdx.x; i < nitems; i += gridDim.x, p ^= 1) {
    const SrsItem<T> &it = items[p];
    if (it.skip) {  // uniform over the block
      if (threadIdx.x == 0) fetch(i + gridDim.x, items[p ^ 1]);
      __syncthreads();
      continue;
    }
    const int Nd = it.Nd;
    const bool small = Nd < kSrsLongRow, flat = small && (MD || !it.together);
    bool tile = Nd >= kSrsLongRow && Nd < kSrsVeryLong;
    // 16-byte accesses: rows of whole 16-byte pieces on aligned bases
    const bool whole = (Nd * sizeof(T)) % 16 == 0;
    const bool vec = whole && (((uintptr_t)it.x | (uintptr_t)it.dg | (uintptr_t)it.y | (uintptr_t)it.z) & 15) == 0;
    const int nel = it.nrows * Nd;
    bool near = false;  // the item's hops fit in shared memory; tiles', always (item_hop_room)
    if (tile || small) {
      const int k0 = ldg_t(it.urp), nh = ldg_t(it.urp + it.nrows) - k0;
      near = nh <= hop_cap;
      // else row by row from global memory; so are a recurrence's last rows of 2048 states or more, fewer than a group of
      // four, whose <x, y> is summed in that order
      tile = tile && near && !(MD && it.dot && it.nrows < TileGeom<T>::R && Nd >= 2048);
      if (tile)
        for (int q = threadIdx.x; q <= it.nrows; q += kMvBlock) hop_rp[q] = ldg_t(it.urp + q) - k0;
      if (near)
        for (int q = threadIdx.x; q <= nh; q += kMvBlock) {
          Hop<T> hp{};
          if (q < nh) hp = ldg_hop(it.uh + k0 + q);
          hp.c *= Nd;
          hops.hop[q] = hp;
        }
    }
    if (tile) {
      if (vec) stage_interleaved<T, kVec, RO>(xs, it.xi, it.nrows, Nd);
      else if (!whole) stage_interleaved<T, kOdd, RO>(xs, it.xi, it.nrows, Nd);
      else stage_interleaved<T, kOff, RO>(xs, it.xi, it.nrows, Nd);
    } else if (small && !flat) {
      stage_interleaved<T, kOdd, RO>(xs, it.xi, it.nrows, Nd);
    } else if (nel <= xs_cap) {
      stage_async(xs, it.xi, nel);
    }
    if (threadIdx.x == kMvBlock - 32) fetch(i + gridDim.x, items[p ^ 1]);  // the next item's description
    if (!tile && (!small || flat)) cp_async_wait_all();
    __syncthreads();
    DotAcc acc{};
    if (tile) {
      if (vec) acc = srs_tiles<T, kVec, HB, MZ, MD, RO>(it, hops, xs);
      else if (!whole) acc = srs_tiles<T, kOdd, HB, MZ, MD, RO>(it, hops, xs);
      else acc = srs_tiles_off<T, MZ, MD, RO>(it, hops, xs);
    } else if (small) {
      if (flat) acc = srs_flat<T, MZ, MD>(it, hops, near, xs);
      else srs_short<T, MZ>(it, hops, near, xs);
    } else {
      acc = srs_longrow<T, MZ, MD>(it, nel <= xs_cap ? xs : it.xi);
    }
    if (MD && it.dot) emit_dot<kMvBlock>(acc, it.dot, red);
    __syncthreads();  // xs and items[p] are free, items[p ^ 1] is there
  }
}

// RI consecutive columns of a row, the first n of them (n < RI only at the row's end): wide 8 or 16 bytes at a time.
template <typename T, bool RO>
__device__ __forceinline__ Lanes<T> ld_cols(const T *p, int n, bool wide) {
  Lanes<T> q{};
  if (wide && n == Lanes<T>::C) {
    if constexpr (sizeof(T) == 4) {
      const float2 a = RO ? __ldg(reinterpret_cast<const float2 *>(p)) : *reinterpret_cast<const float2 *>(p);
      const float2 b = RO ? __ldg(reinterpret_cast<const float2 *>(p) + 1) : *(reinterpret_cast<const float2 *>(p) + 1);
      q.v[0] = a.x, q.v[1] = a.y, q.v[2] = b.x, q.v[3] = b.y;
    } else {
      q = RO ? ldg16(p) : load16(p);
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < Lanes<T>::C; ++cc)
      if (cc < n) q.v[cc] = RO ? ldg_t(p + cc) : p[cc];
  }
  return q;
}
template <typename T>
__device__ __forceinline__ void st_cols(T *p, const T (&v)[Lanes<T>::C], int n, bool wide) {
  if (wide && n == Lanes<T>::C) {
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
      *(reinterpret_cast<float2 *>(p) + 1) = make_float2(v[2], v[3]);
    } else {
      store_lanes(p, v);
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < Lanes<T>::C; ++cc)
      if (cc < n) p[cc] = renorm(v[cc]);
  }
}

// a += the hops of a place from the staged rows or columns xs (RI of them interleaved): entries of k-major slots and
// values, U at a time, the next U on their way meanwhile, to the longest of the warp's places.
template <typename T>
__device__ __forceinline__ void long_hops(const Lanes<T> *xs, const unsigned short *__restrict__ slot, const T *__restrict__ val,
                                          int ld, int kk, T (&a)[Lanes<T>::C]) {
  constexpr int RI = Lanes<T>::C, U = sizeof(T) == 4 ? 8 : 4;
  int c[U];
  T v[U];
  auto load = [&](int k) {
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const bool in = k + q < kk;  // uniform over the warp
      c[q] = in ? __ldg(slot + (k + q) * ld) : 0;
      v[q] = in ? ldg_t(val + (k + q) * ld) : T(0);
    }
  };
  load(0);
#pragma unroll 1
  for (int k = 0; k < kk; k += U) {
    int c0[U];
    T v0[U];
#pragma unroll
    for (int q = 0; q < U; ++q) c0[q] = c[q], v0[q] = v[q];
    load(k + U);
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const Lanes<T> x = xs[c0[q]];
      if (k + q < kk) {
#pragma unroll
        for (int i = 0; i < RI; ++i) a[i] += v0[q] * x.v[i];
      }
    }
  }
}

// Two-pass sectors (srs_two_pass).  Pass 1, per item of kLongRows rows: RI whole rows interleaved in shared memory,
// y = diagonal, (c z), down hops.  Pass 2, per item a share of the sector's groups of RI columns: those columns of
// all rows in shared memory, y += up hops, interaction; <x, y>.  Each hop is then one 16-byte shared-memory load for
// RI elements, and X crosses memory twice instead of once per up hop.  Per element the sum runs diagonal, (c z), down
// hops, then the sum of the up hops, interaction.  What bounds it: the latency of the hop entries
// (from L2: their tables do not fit beside 206 KB of places) and the shared-memory wavefronts of the gathers.  Sector
// (8,8) of the 4x4 cluster, 165,636,900 states, FP32: 12.4 -> 5.6 ms; (5,7): 5.8 -> 1.5 ms.
template <typename T, class Src, int PASS, bool MZ, bool MD, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_srs_long(Src src, int nitems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SrsItem<T> it;
  __shared__ double red[NT / 32];
  constexpr int RI = Lanes<T>::C;
  Lanes<T> *xs = reinterpret_cast<Lanes<T> *>(smem_raw);
  for (int i = blockIdx.x; i < nitems; i += gridDim.x) {
    __syncthreads();  // the previous item is no longer read
    if (threadIdx.x == 0) {
      it.skip = !src.get(i, [&](const SectorOp<T> *op, int srs_rows, int li, const T *x, T *y, const T *z, T c, const LzTask<T> *lz) {
        fetch_item<T>(it, op, srs_rows, li, x, y, MZ ? z : nullptr, c, MD ? lz : nullptr);
      }) || !it.skip;
    }
    __syncthreads();
    if (it.skip) continue;  // nothing to do, or not a two-pass sector (uniform over the block)
    const SectorOp<T> &op = *it.op;
    const int Nd = it.Nd, Nu = op.up_rows;
    const int *__restrict__ len = op.long_len[PASS == 1];
    const int ld = op.long_ld[PASS == 1], L = PASS == 1 ? Nd : Nu, Lw = (L + 31) / 32 * 32;
    DotAcc acc;
    dot_init(acc);
    if constexpr (PASS == 1) {
      for (int r0 = 0; r0 < it.nrows; r0 += RI) {
        const int nr = min(RI, it.nrows - r0);
        const long long base = (long long)r0 * Nd;
        __syncthreads();
#pragma unroll 2
        for (int d = threadIdx.x; d < Nd; d += NT) {
          Lanes<T> q;
#pragma unroll
          for (int r = 0; r < RI; ++r) q.v[r] = r < nr ? ldg_t(it.xi + base + (long long)r * Nd + d) : T(0);
          xs[d] = q;
        }
        __syncthreads();
        for (int d = threadIdx.x; d < Lw; d += NT) {
          const int dd = min(d, Nd - 1);
          const Lanes<T> q = xs[dd];
          T a[RI];
#pragma unroll
          for (int r = 0; r < RI; ++r) a[r] = ldg_t(it.dg + base + (long long)min(r, nr - 1) * Nd + dd) * q.v[r];
          if (MZ && it.z) {
#pragma unroll
            for (int r = 0; r < RI; ++r) a[r] = a[r] + it.c * it.z[base + (long long)min(r, nr - 1) * Nd + dd];
          }
          const int kk = __reduce_max_sync(0xffffffffu, ldg_t(len + dd));
          long_hops<T>(xs, op.long_slot[1] + dd, op.long_val[1] + dd, ld, kk, a);
          if (d < Nd) {
#pragma unroll
            for (int r = 0; r < RI; ++r)
              if (r < nr) it.y[base + (long long)r * Nd + d] = renorm(a[r]);
          }
        }
      }
    } else {
      const int per = (Nu + kLongRows - 1) / kLongRows, ncg = (Nd + RI - 1) / RI, share = (ncg + per - 1) / per;
      const int g0 = it.u0 / kLongRows * share, g1 = min(ncg, g0 + share);
      T *__restrict__ y = it.y - (long long)it.u0 * Nd;
      const bool whole = sizeof(T) == 4 ? Nd % 2 == 0 && (((uintptr_t)it.x | (uintptr_t)y) & 7) == 0
                                        : Nd % 2 == 0 && (((uintptr_t)it.x | (uintptr_t)y) & 15) == 0;
      for (int g = g0; g < g1; ++g) {
        const int d0 = g * RI, nc = min(RI, Nd - d0);
        __syncthreads();
#pragma unroll 2
        for (int u = threadIdx.x; u < Nu; u += NT) xs[u] = ld_cols<T, true>(it.x + (long long)u * Nd + d0, nc, whole);
        __syncthreads();
        for (int u = threadIdx.x; u < Lw; u += NT) {
          const int uu = min(u, Nu - 1);
          T *__restrict__ yr = y + (long long)uu * Nd + d0;
          const Lanes<T> y1 = ld_cols<T, false>(yr, nc, whole);  // pass 1's part, on its way while the hops are summed
          T a[RI];
#pragma unroll
          for (int r = 0; r < RI; ++r) a[r] = T(0);
          const int kk = __reduce_max_sync(0xffffffffu, ldg_t(len + uu));
          long_hops<T>(xs, op.long_slot[0] + uu, op.long_val[0] + uu, ld, kk, a);
#pragma unroll
          for (int r = 0; r < RI; ++r) a[r] = y1.v[r] + a[r];
          if (u < Nu) {
            if (it.vloc) {
              RowPart<T, RI> p;
#pragma unroll
              for (int r = 0; r < RI; ++r) p.v[r] = a[r];
              p = srs_vloc<T, RI, 1>(it.op, u, d0, it.x, p);
#pragma unroll
              for (int r = 0; r < RI; ++r) a[r] = p.v[r];
            }
            st_cols<T>(yr, a, nc, whole);
            if (MD && it.dot) {
              const Lanes<T> q = xs[u];
#pragma unroll
              for (int r = 0; r < RI; ++r)
                if (r < nc) dot_add(acc, q.v[r], a[r]);
            }
          }
        }
      }
      if (MD && it.dot) emit_dot<NT>(acc, it.dot, red);
    }
  }
}

// CRS and SOCRS items
template <typename T, class Src, int ST>
__global__ void __launch_bounds__(kMvBlock, 3) k_row_mv(Src src, int nitems) {
  if constexpr (Src::kEarly) pdl_enter();
  for (int i = blockIdx.x; i < nitems; i += gridDim.x)
    src.get(i, [&](const SectorOp<T> *op, int rows, int li, const T *x, T *y, const T *z, T c, const LzTask<T> *) {
      mv_item<T, ST>(op, rows, li, x, y, z, c);
    });
}

// up hops in flight and resident blocks per SM of the launches outside the eigen step: FP32 tiles are bound by L1 and
// want registers, 8-byte ones by arithmetic and want warps (float-float recurrences of the 12-orbital impurity 16.3 ms
// with two blocks, 15.5 with three)
template <typename T>
constexpr int kPlainHB = sizeof(T) == 4 ? 2 : 1;
template <typename T>
constexpr int kMvBlocks = sizeof(T) == 4 ? 2 : 3;

static int grid_for(const void *fn, size_t smem, int nitems) { return occupancy_grid(fn, kMvBlock, smem, nitems); }

// Opt a kernel in to `bytes` of dynamic shared memory (once per device and size).  Without the opt-in static and
// dynamic shared memory together are held to 48 KB; the operator kernels carry a few KB of static arrays, so the
// attribute is set from 32 KB of dynamic memory on.
template <typename K>
static void set_smem(K kernel, size_t bytes) {
  if (bytes > 32 * 1024) opt_in_smem((const void *)kernel, bytes);
}

template <typename T>
static size_t smem_bytes(const MvShape &sh) {
  return align16(sizeof(T) * (size_t)sh.xs_elems) + sizeof(Hop<T>) * (size_t)(sh.hop_elems + 1);
}

// shared memory of a two-pass launch; blocks of 512 threads two to an SM where it allows, else one of 1024
inline size_t long_smem(const MvShape &sh) { return (size_t)16 * sh.long_places; }
inline bool long_wide(const MvShape &sh) { return long_smem(sh) > 112 * 1024; }
template <typename T, class Src, int PASS, bool MZ, bool MD, int NT>
static void launch_long_pass(const Src &src, int nitems, const MvShape &sh, cudaStream_t st) {
  const auto k = k_srs_long<T, Src, PASS, MZ, MD, NT>;
  set_smem(k, long_smem(sh));
  k<<<occupancy_grid((const void *)k, NT, long_smem(sh), nitems), NT, long_smem(sh), st>>>(src, nitems);
  note_launch();
}
template <typename T, class Src, bool MZ, bool MD>
static void launch_long(const Src &src, int nitems, const MvShape &sh, cudaStream_t st) {
  if (long_wide(sh)) {
    launch_long_pass<T, Src, 1, MZ, MD, 1024>(src, nitems, sh, st);
    launch_long_pass<T, Src, 2, MZ, MD, 1024>(src, nitems, sh, st);
  } else {
    launch_long_pass<T, Src, 1, MZ, MD, 512>(src, nitems, sh, st);
    launch_long_pass<T, Src, 2, MZ, MD, 512>(src, nitems, sh, st);
  }
}

template <typename T, class Src, bool MZ, bool MD, int HB, int MB>
static void launch_srs(const Src &src, int nitems, const MvShape &sh, cudaStream_t st, bool early = false) {
  if (sh.long_places) launch_long<T, Src, MZ, MD>(src, nitems, sh, st);
  if (!sh.other) return;
  const size_t sm = smem_bytes<T>(sh);
  const auto k = k_srs_mv<T, Src, MZ, MD, HB, MB>;
  set_smem(k, sm);
  const int grid = grid_for((const void *)k, sm, nitems);
  if constexpr (Src::kEarly) {
    if (early && !sh.long_places) {
      launch_pdl(k, grid, kMvBlock, sm, st, src, nitems, sh.xs_elems, sh.hop_elems);
      return;
    }
  }
  k<<<grid, kMvBlock, sm, st>>>(src, nitems, sh.xs_elems, sh.hop_elems);
  note_launch();
}
template <typename T, class Src>
static void launch_rows(int storage, const Src &src, int nitems, cudaStream_t st, bool early = false) {
  const auto k = storage == kCRS ? k_row_mv<T, Src, kCRS> : k_row_mv<T, Src, kSOCRS>;
  const int grid = grid_for((const void *)k, 0, nitems);
  if constexpr (Src::kEarly) {
    if (early) {
      launch_pdl(k, grid, kMvBlock, 0, st, src, nitems);
      return;
    }
  }
  k<<<grid, kMvBlock, 0, st>>>(src, nitems);
  note_launch();
}

template <typename T>
void launch_mv(const MvTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, cudaStream_t st) {
  const MvSource<T> src{tasks_dev, item_task_dev};
  if (sh.storage != kSRS) launch_rows<T>(sh.storage, src, nitems_total, st);
  else if (sh.plain) launch_srs<T, MvSource<T>, false, false, kPlainHB<T>, kMvBlocks<T>>(src, nitems_total, sh, st);
  else launch_srs<T, MvSource<T>, true, false, 1, kMvBlocks<T>>(src, nitems_total, sh, st);
}

template <typename T>
void launch_mv_vectors(const Sector_mv<T> &v, MvShape sh, cudaStream_t st) {
  const VecSource<T> src{v.op, v.x, v.y, v.ld, v.rows, v.per, v.accumulate};
  const int n = v.per * v.nvec;
  if (sh.storage != kSRS) launch_rows<T>(sh.storage, src, n, st);
  // short rows wait on memory, not on L1: three blocks per SM for every type (16-site square cluster, FP32 rows of 16 states
  // 82 us with two, 66 with three)
  else if (sh.short_rows && v.accumulate) launch_srs<T, VecSource<T>, true, false, 1, 3>(src, n, sh, st);
  else if (sh.short_rows) launch_srs<T, VecSource<T>, false, false, 1, 3>(src, n, sh, st);
  else if (v.accumulate) launch_srs<T, VecSource<T>, true, false, 1, kMvBlocks<T>>(src, n, sh, st);
  else launch_srs<T, VecSource<T>, false, false, kPlainHB<T>, kMvBlocks<T>>(src, n, sh, st);
}

template <typename T>
void launch_lz_mv(const LzBatch<T> &b, int it, bool early, MvShape sh, cudaStream_t st) {
  if constexpr (!std::is_same<T, ffloat>::value) {  // float-float recurrences: spin-resolved storage only, never split
    if (b.split) {
      const LzSource<T, true> src{b.tasks, b.mv_item_task, it};
      if (sh.storage != kSRS) launch_rows<T>(sh.storage, src, b.mv_items, st, early);
      else launch_srs<T, LzSource<T, true>, true, false, 1, kMvBlocks<T>>(src, b.mv_items, sh, st, early);
      return;
    }
  }
  const LzSource<T, false> src{b.tasks, b.item_task, it};
  if constexpr (sizeof(T) == 8) {
    // few items: no more blocks per SM than registers for two rounds of up hops in flight allow (G of the 11-orbital
    // impurity, 99 items, float-float 7.6 -> 6.1 ms, FP64 8.8 -> 8.3); FP64, bound by arithmetic, one (198 items of the same
    // sizes: 11.9 ms with either)
    if (b.nitems <= (std::is_same<T, ffloat>::value ? 2 : 1) * kSms) {
      launch_srs<T, LzSource<T, false>, true, true, 2, 2>(src, b.nitems, sh, st, early);
      return;
    }
  }
  launch_srs<T, LzSource<T, false>, true, true, 1, kMvBlocks<T>>(src, b.nitems, sh, st, early);
}

// Kernel attributes of the eigen step's operator for a shape; called before a step is captured into a graph.
template <typename T>
void prepare_eig_mv(MvShape sh) {
  const size_t sm = smem_bytes<T>(sh);
  set_smem(k_srs_mv<T, EigSource<T>, false, false, 1, 3>, sm);
  set_smem(k_srs_mv<T, EigSource<T>, false, false, 2, 2>, sm);
  if (sh.long_places) {
    set_smem(k_srs_long<T, EigSource<T>, 1, false, false, 1024>, long_smem(sh));
    set_smem(k_srs_long<T, EigSource<T>, 2, false, false, 1024>, long_smem(sh));
    set_smem(k_srs_long<T, EigSource<T>, 1, false, false, 512>, long_smem(sh));
    set_smem(k_srs_long<T, EigSource<T>, 2, false, false, 512>, long_smem(sh));
  }
}

template <typename T>
void launch_eig_mv(const EigTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, cudaStream_t st,
                   T *probe_y) {
  const EigSource<T> src{tasks_dev, item_task_dev, probe_y};
  if (sh.storage != kSRS) launch_rows<T>(sh.storage, src, nitems_total, st);
  else if (sh.mb >= 3) launch_srs<T, EigSource<T>, false, false, 1, 3>(src, nitems_total, sh, st);
  else launch_srs<T, EigSource<T>, false, false, 2, 2>(src, nitems_total, sh, st);
}

template <typename T>
OpTuning tune_eig_mv(const EigTask<T> *tasks_dev, const int *item_task_dev, int nitems_total, MvShape sh, T *probe_y,
                     cudaStream_t st) {
  OpTuning best;
  best.done = true;
  best.ms = 1e30;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return best;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return best;
  }
  for (int mb = 2; mb <= 3; ++mb) {
    MvShape v = sh;
    v.mb = mb;
    prepare_eig_mv<T>(v);
    launch_eig_mv<T>(tasks_dev, item_task_dev, nitems_total, v, st, probe_y);  // warm
    cudaEventRecord(e0, st);
    for (int r = 0; r < 3; ++r) launch_eig_mv<T>(tasks_dev, item_task_dev, nitems_total, v, st, probe_y);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms / 3.0 < best.ms) {
      best.ms = ms / 3.0;
      best.mb = mb;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return best;
}

}  // namespace edgpu
