// Nodal batch: proposal, dS and accept for each vertex of a Jacobi batch.
//
// GSAP spends ~25 launches and two bb_segsorts of all E neighbour-block lists
// per batch (partition.hpp:456-662); each of its seven dS kernels has one
// thread walk a whole blockmodel row in a serial sorted merge with the
// vertex's sorted neighbour-block list (kernels.hpp:494-597, 1153-1726).
//
// Here a group of threads owns one vertex: 8, 16 or 32 lanes for vertices of
// up to 16, 32 or 64 neighbour entries (two entries a lane), a CTA of four
// warps for up to kWarpList entries a direction (or, up to kWideEntries in all
// and many to a batch, a warp), a larger CTA or a cluster for the few heavier
// ones (run on streams of their own next to the warp kernel).  The host sorts
// each batch's vertices into these lists once per job.
//   * proposal: Philox draws, an exact integer inverse-CDF pick of a
//     neighbour (out- then in-entries; with unit weights the drawn number is
//     the entry's index, else a prefix scan), then the per-block draws of the
//     batch (kernels.hpp:877-1032);
//   * neighbour blocks grouped per distinct block by comparing keys in shared
//     memory, or (heavy vertices) in a shared-memory hash table; GSAP sorts
//     all E entries every batch;
//   * dS: GSAP's seven terms rewritten as "changed cells + row degrees".
//     A row term  sum_c f(x_c)  with  f(x) = x (log2 x - log2 dcol[c] - L)
//     splits into  sum_c (x log2 x - x log2 dcol[c])  -  L * sum_c x ;
//     between the old and the new rows the first sums over unchanged columns
//     cancel, so only the columns the vertex touches and the four rows'
//     degree terms remain (see Acc below).  Counts come from the dense B x B
//     form (small B, O(1)) or by binary search in the CSR rows.
//     Quirks of the reference kept: old column degrees (Q2), one term per
//     list entry for blocks missing from the target row
//     (kernels.hpp:1648-1652, 1314-1318), the r/s in-weight corrections and
//     the conditional extra column term (kernels.hpp:1506-1510, 1573-1578,
//     1663-1669, 1718-1723), unsigned count arithmetic.
//   * accept iff dS < 0 (kernels.hpp:634-640), or by the general-mode rules
//     (exact MDL, Metropolis-Hastings) below; the new label goes to a side
//     buffer so every vertex of the batch sees the same old labels.
// All entropy arithmetic is FP64.
#include "common.cuh"
#include "kernels.h"
#include "multi.cuh"
#include "dense.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace sbp {

namespace {

constexpr int kNodalWarps = 4;
constexpr int kWarpList = 128;     // entries per direction a warp sorts in shared memory
constexpr int kHeavyThreads = 256;
constexpr int kHashSlots = 8192;  // of the heavy path's table

struct NodalArgs {
  const double* xlx;        // x log2 x table
  const int32_t *optr, *oidx, *iptr, *iidx;
  const uint32_t *ow, *iw, *kdo, *kdi;
  const int32_t* part;
  const int32_t *bop, *boe, *boc, *bip, *bie, *bic;
  const uint32_t *bon, *bin, *d_out, *d_in;
  const uint32_t *Md, *MTd;
  const double *ld_out, *ld_in;
  const int32_t* nbr_s;
  int32_t B;
  uint64_t seed;
  uint32_t seq;
  int32_t lo, count;
  const int32_t* verts;     // given mode
  const int32_t* props_in;  // given mode
  int32_t* newlab;
  double* rec;
  int32_t* props_out;
  double* dS_raw;
  const int32_t* heavy;     // batch indices handled by the CTA kernels, hubs first
  int32_t nheavy, nhub;
  const int32_t *small, *mid;  // batch indices of the warp kernel (NodalItems)
  int32_t nsmall, nmid;
  int32_t unit;                // every weight is 1
  int32_t nlarge, nwide, nmid64;  // mid vertices by path: a CTA, wide_vertex, 32 lanes, the others
  int32_t* err;             // error counter (hash table overflow)
  const int32_t* ctl;       // sweep control: gate, and seq += ctl[0] * seq_mul
  uint32_t seq_mul;
  // general-mode kernels only (ScoreMode)
  int32_t exact, mh;
  double beta;
  double* logH_raw;         // given mode: log Hastings ratio of each move
};

// g(x, a) = x log2 x - x a, zero for x == 0
__device__ __forceinline__ double gterm(const double* tab, uint32_t x, double a) {
  return x == 0u ? 0.0 : __fma_rn(-(double)x, a, xlx(tab, x));
}

// The four rows a move from r to s reads: out-rows r and s, in-rows r and s.
template <bool DENSE>
struct Rows;

template <>
struct Rows<false> {
  const int32_t *oc, *ic;
  const uint32_t *on, *inn;
  int32_t rO0, rO1, sO0, sO1, rI0, rI1, sI0, sI1;
  __device__ Rows(const NodalArgs& a, int r, int s)
      : oc(a.boc), ic(a.bic), on(a.bon), inn(a.bin), rO0(a.bop[r]), rO1(a.boe[r]),
        sO0(a.bop[s]), sO1(a.boe[s]), rI0(a.bip[r]), rI1(a.bie[r]), sI0(a.bip[s]),
        sI1(a.bie[s]) {}
  __device__ __forceinline__ uint32_t out_r(int c) const { return row_lookup(oc, on, rO0, rO1, c); }
  __device__ __forceinline__ uint32_t out_s(int c) const { return row_lookup(oc, on, sO0, sO1, c); }
  __device__ __forceinline__ uint32_t in_r(int c) const { return row_lookup(ic, inn, rI0, rI1, c); }
  __device__ __forceinline__ uint32_t in_s(int c) const { return row_lookup(ic, inn, sI0, sI1, c); }
  __device__ __forceinline__ uint32_t out_at(bool row_s, int c) const {
    return row_lookup(oc, on, row_s ? sO0 : rO0, row_s ? sO1 : rO1, c);
  }
};

template <>
struct Rows<true> {
  const uint32_t *orr, *ors, *irr, *irs;
  __device__ Rows(const NodalArgs& a, int r, int s)
      : orr(a.Md + (size_t)r * a.B), ors(a.Md + (size_t)s * a.B), irr(a.MTd + (size_t)r * a.B),
        irs(a.MTd + (size_t)s * a.B) {}
  __device__ __forceinline__ uint32_t out_r(int c) const { return orr[c]; }
  __device__ __forceinline__ uint32_t out_s(int c) const { return ors[c]; }
  __device__ __forceinline__ uint32_t in_r(int c) const { return irr[c]; }
  __device__ __forceinline__ uint32_t in_s(int c) const { return irs[c]; }
  __device__ __forceinline__ uint32_t out_at(bool row_s, int c) const {
    return (row_s ? ors : orr)[c];
  }
};

// Per-thread partial of a move's dS.  GSAP's seven terms (kernels.hpp:143-182,
// 494-597, 1153-1726) combine, after the per-block row sums cancel, into
//   dS = - sum_X d_X log2 d_X  +  sum_X L_X mass_X
//        - sum over changed cells (g(new) - g(old))  + corner cells
// where X runs over the old/new out- and in-rows of r and s, d_X the old row
// degree, L_X = log2 of the new row degree and mass_X the new row's total
// count; g(x, a) = x log2 x - x a with a = log2 of the old column degree (Q2).
// `acc` collects this thread's terms, m4..m7 the count changes of the new
// out-row r, out-row s, in-row r and in-row s.
struct Acc {
  double acc = 0.0;
  int m4 = 0, m5 = 0, m6 = 0, m7 = 0;
};

// One neighbour entry of v (block c, weight w) in direction `in` (false =
// out-edge, true = in-edge); `leader` marks one entry per distinct block of
// that direction and kc is v's total weight to/from c
// (kernels.hpp:1444-1726 for out, 1153-1362 for in).
template <bool DENSE>
__device__ __forceinline__ void entry(const NodalArgs& a, const Rows<DENSE>& R, int r, int s,
                                      uint32_t niS, bool in, int32_t c, uint32_t w, bool leader,
                                      uint32_t kc, Acc& q) {
  if (in && (c == r || c == s)) return;  // in-rows leave out blocks r and s
  const double ldc = in ? a.ld_out[c] : a.ld_in[c];
  const uint32_t Mt = in ? R.in_s(c) : R.out_s(c);
  int dmo = 0, dmt = 0;
  if (leader && c != r && c != s) {
    const uint32_t Mo = in ? R.in_r(c) : R.out_r(c);
    const uint32_t x = Mo - kc;
    q.acc -= gterm(a.xlx, x, ldc) - gterm(a.xlx, Mo, ldc);
    dmo = (int)((long long)x - (long long)Mo);
    if (Mt != 0u) {
      const uint32_t y = Mt + kc;
      q.acc -= gterm(a.xlx, y, ldc) - gterm(a.xlx, Mt, ldc);
      dmt = (int)((long long)y - (long long)Mt);
    }
  }
  if (Mt == 0u) {
    // block c absent from the target row: one term per list entry
    // (kernels.hpp:1648-1652, 1696-1713; 1314-1318, 1348-1358)
    const uint32_t y = in ? w : w - (c == r ? niS : 0u) + (c == s ? niS : 0u);
    q.acc -= gterm(a.xlx, y, ldc);
    dmt += (int)y;
  }
  if (in) {
    q.m6 += dmo;
    q.m7 += dmt;
  } else {
    q.m4 += dmo;
    q.m5 += dmt;
  }
}

// Group sums of the four direction weights v has to/from blocks r and s.
struct RsWeights {
  uint32_t koR, koS, niR, niS;
};

// What the corner cells (r,r), (r,s), (s,r), (s,s) of M and the row-degree
// terms of a move are made from.
struct Corner {
  uint32_t Mrr, Mrs, Msr, Mss;
  uint32_t dor, dos, dir, dis;  // old block degrees
  double ldo_r, ldo_s, ldi_r, ldi_s;
  uint32_t kO, kI;              // v's degrees
};

__device__ __forceinline__ void load_degrees(const NodalArgs& a, int v, int r, int s, Corner& q) {
  q.kO = a.kdo[v];
  q.kI = a.kdi[v];
  q.dor = a.d_out[r];
  q.dos = a.d_out[s];
  q.dir = a.d_in[r];
  q.dis = a.d_in[s];
  q.ldi_r = a.ld_in[r];
  q.ldi_s = a.ld_in[s];
  q.ldo_r = a.ld_out[r];
  q.ldo_s = a.ld_out[s];
}

// Term `k` (0..12) of a move's corner and degree terms, 0 for other k; m4..m7
// are the count changes of the new out-row r, out-row s, in-row r and in-row
// s away from the corners.  Terms 0-3: the old corner cells, + M log2 M; 4-7:
// the new corner cells, - g(x); 8-11: + L mass of the four new rows; 12: the
// old row degrees.  kernels.hpp:1506-1510, 1573-1578, 1663-1669, 1718-1723
// give the new corner counts.  Straight-line, no lane branches: every lane
// evaluates the cell form and the row form of its operands and keeps the one
// its k owns (CELLS / ROWS leave a form out where no lane of a call owns it).
template <bool CELLS, bool ROWS>
__device__ __forceinline__ double corner_term(const double* tab, const Corner& q,
                                              const RsWeights& w, int m4, int m5, int m6, int m7,
                                              int k) {
  const uint32_t xrr = q.Mrr - w.koR - w.niR;
  const uint32_t xrs = q.Mrs != 0u ? q.Mrs - w.koS + w.niR : w.niR;
  const uint32_t xsr = q.Msr + w.koR - w.niS;
  const uint32_t xss = q.Mss != 0u ? q.Mss + w.koS + w.niS : w.niS;
  const bool use_rs = q.Mrs != 0u || w.niR > 0u;                       // cell or extra term
  const bool use_ss = q.Mss != 0u || (w.koS == 0u && w.niS > 0u);
  const int j = k & 3;
  double t = 0.0;
  if (CELLS) {
    const uint32_t Mold = j == 0 ? q.Mrr : j == 1 ? q.Mrs : j == 2 ? q.Msr : q.Mss;
    const uint32_t xnew = j == 0 ? xrr : j == 1 ? xrs : j == 2 ? xsr : xss;
    const bool on = j == 0 ? q.Mrr != 0u : j == 1 ? use_rs : j == 2 ? q.Msr != 0u : use_ss;
    const double ld = (j & 1) ? q.ldi_s : q.ldi_r;
    const bool old_cell = k < 4;
    const uint32_t X = old_cell ? Mold : xnew;
    const bool cell_on = old_cell ? Mold != 0u : on;
    const double cell = old_cell ? xlx(tab, X) : -gterm(tab, X, ld);
    if (k < 8) t = cell_on ? cell : 0.0;
  }
  if (ROWS) {
    const long long l4 = m4 + (q.Mrr ? (long long)xrr - q.Mrr : 0) +
                         (use_rs ? (long long)xrs - (long long)q.Mrs : 0);
    const long long l5 = m5 + (q.Msr ? (long long)xsr - q.Msr : 0) +
                         (use_ss ? (long long)xss - (long long)q.Mss : 0);
    const long long mass4 = (long long)q.dor + l4;
    const long long mass5 = (long long)q.dos + l5;
    const long long mass6 = (long long)q.dir - (long long)q.Mrr - (long long)q.Msr + m6;
    const long long mass7 = (long long)q.dis - (long long)q.Mrs - (long long)q.Mss + m7;
    const long long mass = j == 0 ? mass4 : j == 1 ? mass5 : j == 2 ? mass6 : mass7;
    const uint32_t d =
        j == 0 ? q.dor - q.kO : j == 1 ? q.dos + q.kO : j == 2 ? q.dir - q.kI : q.dis + q.kI;
    const double row = mass != 0 ? l2x(tab, d) * (double)mass : 0.0;
    const double deg =
        -((q.dor ? (double)q.dor * q.ldo_r : 0.0) + (q.dos ? (double)q.dos * q.ldo_s : 0.0) +
          (q.dir ? (double)q.dir * q.ldi_r : 0.0) + (q.dis ? (double)q.dis * q.ldi_s : 0.0));
    if (k >= 8 && k < 12) t = row;
    else if (k == 12) t = deg;
  }
  return t;
}

// Adds the corner and degree terms to lanes 0..12 of the calling warp (after
// m4..m7 hold the group totals; call it from one warp of a CTA group).
template <bool DENSE>
__device__ __forceinline__ void corner_terms(const NodalArgs& a, const Rows<DENSE>& R, int v,
                                             int r, int s, const RsWeights& w, Acc& q, int lane) {
  // lane 0: M[r][r], 1: M[r][s], 2: M[s][r], 3: M[s][s]
  const uint32_t mm = lane < 4 ? R.out_at((lane & 2) != 0, (lane & 1) ? s : r) : 0u;
  Corner c;
  c.Mrr = __shfl_sync(kFull, mm, 0);
  c.Mrs = __shfl_sync(kFull, mm, 1);
  c.Msr = __shfl_sync(kFull, mm, 2);
  c.Mss = __shfl_sync(kFull, mm, 3);
  load_degrees(a, v, r, s, c);
  q.acc += corner_term<true, true>(a.xlx, c, w, q.m4, q.m5, q.m6, q.m7, lane);
}

// A thread group cooperating on one vertex: a warp (G = 32) or a CTA.
template <int G>
struct Group {
  double* red;  // G/32 doubles of shared scratch (CTA only)
  __device__ __forceinline__ int rank() const { return G == 32 ? (threadIdx.x & 31) : threadIdx.x; }
  __device__ __forceinline__ void sync() const {
    if (G == 32) __syncwarp();
    else __syncthreads();
  }
  __device__ double sum(double x) const {
    x = warp_sum(x);
    if (G == 32) return x;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < G / 32; ++i) t += red[i];
    __syncthreads();
    return t;
  }
  __device__ long long sum_ll(long long x) const {
    return (long long)sum((double)x);  // |x| < 2^53: exact
  }
};

// Lists of more than kWarpList entries: per-block totals from a shared-memory
// hash table, built in passes that each take the blocks of one hash class,
// so the table never holds more than a few thousand blocks.  Costs
// O(n * passes) with passes ~ n / 2048.
struct HashTab {
  int32_t* key;    // -1 = empty
  uint32_t* sum;
  int32_t* first;  // smallest entry index of the block
};

__device__ __forceinline__ uint32_t hslot(int32_t c) { return ((uint32_t)c * 2654435761u) >> 19; }
__device__ __forceinline__ uint32_t hclass(int32_t c, uint32_t P) {
  return ((uint32_t)c * 0x85EBCA6Bu ^ ((uint32_t)c >> 13)) % P;
}

// Inserts block c (entry k, weight w); false if the table is full.
__device__ bool hash_add(const HashTab& h, int32_t c, uint32_t w, int k) {
  uint32_t i = hslot(c);
  for (int probe = 0; probe < kHashSlots; ++probe, i = (i + 1) & (kHashSlots - 1)) {
    int32_t cur = atomicCAS(h.key + i, -1, c);
    if (cur == -1 || cur == c) {
      atomicAdd(h.sum + i, w);
      atomicMin(h.first + i, k);
      return true;
    }
  }
  return false;
}

__device__ int hash_find(const HashTab& h, int32_t c) {
  uint32_t i = hslot(c);
  for (int probe = 0; probe < kHashSlots; ++probe, i = (i + 1) & (kHashSlots - 1))
    if (h.key[i] == c) return (int)i;
  return -1;
}

// Neighbour of v whose running weight (out-entries, then in-entries) first
// exceeds t (choose_neighbored_node_block, kernels.hpp:877-939).
__device__ int32_t pick_neighbour(const NodalArgs& a, int v, uint64_t t, int lane) {
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  const int32_t i0 = a.iptr[v], ni = a.iptr[v + 1] - i0;
  const int n = no + ni;
  uint64_t acc = 0;
  for (int k0 = 0; k0 < n; k0 += 32) {
    int k = k0 + lane;
    uint32_t w = 0;
    int32_t u = 0;
    if (k < n) {
      if (k < no) { w = __ldg(a.ow + o0 + k); u = __ldg(a.oidx + o0 + k); }
      else { w = __ldg(a.iw + i0 + k - no); u = __ldg(a.iidx + i0 + k - no); }
    }
    uint64_t incl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    unsigned hit = __ballot_sync(kFull, k < n && acc + incl > t);
    if (hit) return __shfl_sync(kFull, u, __ffs(hit) - 1);
    acc += __shfl_sync(kFull, incl, 31);
  }
  return 0;
}

// Vertex and proposal of batch item i (computed by one warp).
// u2 = the vertex's third draw (the Metropolis-Hastings uniform).
template <bool GIVEN>
__device__ __forceinline__ void item(const NodalArgs& a, int i, int lane, int& v, int& s,
                                     uint32_t& u2) {
  if (GIVEN) {
    v = a.verts[i];
    s = a.props_in[i];
    u2 = 0u;
    return;
  }
  v = a.lo + i;
  P4 x = draw(a.seed, kRngNodalVertex, a.seq + ctl_itr(a.ctl) * a.seq_mul, (uint32_t)v);
  u2 = x.v[2];
  int rnd = (int)(x.v[0] % (uint32_t)a.B);
  uint64_t deg = (uint64_t)a.kdo[v] + a.kdi[v];
  if (deg == 0) {
    s = rnd;
  } else {
    int32_t un = pick_neighbour(a, v, scale_draw(x.v[1], deg), lane);
    int32_t u = a.part[un];
    s = a.nbr_s[u] < 0 ? rnd : a.nbr_s[u];
  }
}

__device__ __forceinline__ void write_result(const NodalArgs& a, bool given, int i, int r, int s,
                                             double d) {
  if (given) {
    a.dS_raw[i] = d;
  } else {
    bool acc = d < 0.0;
    a.newlab[i] = acc ? s : r;
    a.rec[i] = acc ? d : 0.0;
    if (a.props_out) a.props_out[i] = s;
  }
}

// Sum over a lane group of W lanes (32: the warp, 16: each half-warp).
template <int W>
__device__ __forceinline__ double group_sum(double x) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
  return x;
}

// ------------------------------------------------------------ general mode --
// Kernels instantiated with GEN = true score a move by the exact change of
// the MDL (exact = 1) or by GSAP's terms (exact = 0), and accept it by
// Metropolis-Hastings (mh = 1) or iff dS < 0.
//
// Exact dS.  S = model - data_S with
//   data_S = sum_cells M log2 M - sum_rows d_out log2 d_out - sum_cols d_in log2 d_in
// and the model term fixed while B is.  Moving v from r to s, with kout[c]
// and kin[c] v's weight to and from block c (self loops of weight `self`
// apart), moves kout[c] from cell (r,c) to (s,c) and kin[c] from (c,r) to
// (c,s) for every c other than r and s, changes the four corner cells as in
// corner_exact, and moves v's out- and in-degree between the rows and
// columns r and s; dS = -(change of data_S).  Only those cells and four
// degrees enter, each as x log2 x.
//
// Hastings ratio of GSAP's proposal (kernels.hpp:877-1032): v picks an
// incident edge with probability proportional to its weight, the edge's
// other end lies in block t, and s is proposed with probability
// (M_ts + M_st + 1) / (d_t + B), d_t = d_out[t] + d_in[t], so
//   p(r -> s) = sum_t k_t (M_ts + M_st + 1) / (d_t + B) / k_v
// with k_t v's weight to and from t (a self loop counts in both directions)
// and k_v the sum of the k_t.  The reverse move reads the blockmodel after
// the move, in which the self loops sit in block s.  A move is accepted when
//   u < 2^(-beta dS) p(s -> r) / p(r -> s)
// with u the vertex's third draw scaled to [0, 1).

struct Hast {
  double f = 0.0, b = 0.0;  // forward and reverse proposal weights (k_v times p)
};

// acc plus term `k` (0..15) of the corner cells and the four degrees of the
// exact dS, acc for other k: terms 0-3 the old cells (r,r), (r,s), (s,r), (s,s), 4-7 the
// same cells after the move, 8-11 the new degrees d_out[r], d_out[s], d_in[r],
// d_in[s], 12-15 the old ones.  koR..niS include the self loops (their other
// end is in r).  The rounding is spelled out, so that it does not hang on what
// the compiler contracts: beyond the table a product w log2 w joins the sum
// in one rounding, but for the old degrees.
__device__ __forceinline__ double corner_exact(const double* tab, const Corner& q,
                                               const RsWeights& w, uint32_t self, int k,
                                               double acc) {
  if (k >= 16) return acc;
  const int j = k & 3;
  uint32_t X;
  if (k < 8) {
    const uint32_t M = j == 0 ? q.Mrr : j == 1 ? q.Mrs : j == 2 ? q.Msr : q.Mss;
    // unsigned wrap-around in the middle is fine: the results are >= 0
    const uint32_t x = j == 0   ? M - w.koR - w.niR + self
                       : j == 1 ? M - w.koS + (w.niR - self)
                       : j == 2 ? M + (w.koR - self) - w.niS
                                : M + w.koS + w.niS + self;
    X = k < 4 ? M : x;
  } else {
    const uint32_t d0 = j == 0 ? q.dor : j == 1 ? q.dos : j == 2 ? q.dir : q.dis;
    const uint32_t d1 =
        j == 0 ? d0 - q.kO : j == 1 ? d0 + q.kO : j == 2 ? d0 - q.kI : d0 + q.kI;
    X = k < 12 ? d1 : d0;
  }
  const bool plus = k < 4 || (k >= 8 && k < 12);
  if (X >= kXlxTable && k < 12)
    return __fma_rn(plus ? (double)X : -(double)X, log2((double)X), acc);
  const double t = xlx(tab, X);
  return __dadd_rn(acc, plus ? t : -t);
}

// Exact change of - data_S in the off-corner cells of a neighbour block, once
// per block and direction (lead; c other than r and s).
__device__ __forceinline__ double exact_term(const double* tab, uint32_t Mo, uint32_t Mt,
                                             uint32_t kc) {
  return __dsub_rn(__dadd_rn(__dsub_rn(xlx(tab, Mo), xlx(tab, Mo - kc)), xlx(tab, Mt)),
                   xlx(tab, Mt + kc));
}

// Proposal weights of a neighbour block t other than r and s, kt = v's
// weight to and from t.
template <bool DENSE>
__device__ __forceinline__ void hast_block(const NodalArgs& a, const Rows<DENSE>& R, int32_t t,
                                           uint32_t kt, Hast& h) {
  const double D = (double)a.d_out[t] + (double)a.d_in[t] + (double)a.B;
  const double k = (double)kt;
  h.f += k * ((double)R.in_s(t) + (double)R.out_s(t) + 1.0) / D;
  h.b += k * ((double)R.in_r(t) + (double)R.out_r(t) - k + 1.0) / D;
}

// Proposal weights of blocks r and s (one thread of the group).
template <bool DENSE>
__device__ __forceinline__ void hast_rs(const NodalArgs& a, const Rows<DENSE>& R, int v, int r,
                                        int s, const RsWeights& w, uint32_t self, Hast& h) {
  const uint32_t Mrr = R.out_at(false, r), Mrs = R.out_at(false, s);
  const uint32_t Msr = R.out_at(true, r), Mss = R.out_at(true, s);
  const uint32_t xrr = Mrr - w.koR - w.niR + self;
  const uint32_t xrs = Mrs - w.koS + (w.niR - self);
  const uint32_t xsr = Msr + (w.koR - self) - w.niS;
  const double kv = (double)a.kdo[v] + (double)a.kdi[v], Bd = (double)a.B;
  const double Dr = (double)a.d_out[r] + (double)a.d_in[r];
  const double Ds = (double)a.d_out[s] + (double)a.d_in[s];
  const double kr = (double)w.koR + (double)w.niR, ks = (double)w.koS + (double)w.niS;
  const double sl = 2.0 * (double)self;
  h.f += kr * ((double)Mrs + (double)Msr + 1.0) / (Dr + Bd);
  h.f += ks * ((double)Mss + (double)Mss + 1.0) / (Ds + Bd);
  h.b += (kr - sl) * ((double)xrr + (double)xrr + 1.0) / (Dr - kv + Bd);
  h.b += (ks + sl) * ((double)xsr + (double)xrs + 1.0) / (Ds + kv + Bd);
}

// Corner counts and degrees for corner_term, on a full warp.
template <bool DENSE>
__device__ __forceinline__ Corner load_corner(const NodalArgs& a, int v, int r, int s, int lane) {
  const uint32_t mm =
      lane < 4 ? Rows<DENSE>(a, r, s).out_at((lane & 2) != 0, (lane & 1) ? s : r) : 0u;
  Corner q{};
  load_degrees(a, v, r, s, q);
  q.Mrr = __shfl_sync(kFull, mm, 0);
  q.Mrs = __shfl_sync(kFull, mm, 1);
  q.Msr = __shfl_sync(kFull, mm, 2);
  q.Mss = __shfl_sync(kFull, mm, 3);
  return q;
}

constexpr double kLn2 = 0.6931471805599453;

// Accept test of a general-mode move (r != s).
__device__ __forceinline__ bool accept_move(const NodalArgs& a, double d, double logH,
                                            uint32_t u) {
  if (!a.mh) return d < 0.0;
  // -beta * dS * ln 2 + logH, rounded step by step (no contraction)
  const double x = __dadd_rn(__dmul_rn(__dmul_rn(-a.beta, d), kLn2), logH);
  if (x >= 0.0) return true;
  return log((double)u * 2.3283064365386963e-10) < x;
}

__device__ __forceinline__ void write_result_gen(const NodalArgs& a, bool given, int i, int r,
                                                 int s, double d, double logH, uint32_t u) {
  if (given) {
    a.dS_raw[i] = d;
    if (a.logH_raw) a.logH_raw[i] = logH;
    return;
  }
  const bool acc = r != s && accept_move(a, d, logH, u);
  a.newlab[i] = acc ? s : r;
  a.rec[i] = acc ? d : 0.0;
  if (a.props_out) a.props_out[i] = s;
}

// ------------------------------------------------------------- warp paths --
// A move's dS is a sum of per-entry terms and 13 corner and degree terms.
// The entries are dealt to lanes in a fixed order and each lane subtracts its
// entries' terms one after the other (the rounding of the sum is part of the
// result, since a move is accepted iff dS < 0), so what may be arranged
// freely is everything before the subtraction: the loads, the grouping of
// equal blocks and the terms themselves.
//
// What bounds these kernels is the chain of dependent loads of a vertex (its
// rows, its entries, their blocks, the proposal's block draw, the counts of
// the proposed block's rows, the x log2 x table) and, on large batches, the
// instructions issued per vertex.  So a group holds two entries a lane (the
// same sums: a butterfly over 2L lanes starts by adding lanes l and l + L),
// equal blocks are found by comparing against the group's keys in shared
// memory (__reduce_add_sync over __match_any_sync's groups runs once per
// distinct mask), the count changes of the four rows come in closed form
// from v's degrees instead of four more group sums, and everything that does
// not depend on the proposal is loaded before it is known.

// Counts M[row][c] (out-entries) or M[c][row] (in-entries) of E entries; 0
// where not wanted.  In the CSR form the binary searches advance together.
template <bool DENSE, int E>
__device__ __forceinline__ void row_counts(const NodalArgs& a, int row, const bool* in,
                                           const int32_t* c, const bool* want, uint32_t* m) {
  if constexpr (DENSE) {
#pragma unroll
    for (int j = 0; j < E; ++j)
      m[j] = want[j] ? (in[j] ? a.MTd : a.Md)[(size_t)row * a.B + c[j]] : 0u;
  } else {
    int32_t lo[E], hi[E], end[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
      lo[j] = want[j] ? (in[j] ? a.bip : a.bop)[row] : 0;
      hi[j] = end[j] = want[j] ? (in[j] ? a.bie : a.boe)[row] : 0;
    }
    bool go = true;
    while (go) {
      go = false;
      int32_t x[E];
#pragma unroll
      for (int j = 0; j < E; ++j)
        x[j] = lo[j] < hi[j] ? (in[j] ? a.bic : a.boc)[(lo[j] + hi[j]) >> 1] : 0;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if (lo[j] >= hi[j]) continue;
        const int32_t mid = (lo[j] + hi[j]) >> 1;
        if (x[j] < c[j]) lo[j] = mid + 1;
        else hi[j] = mid;
        go = go || lo[j] < hi[j];
      }
    }
#pragma unroll
    for (int j = 0; j < E; ++j)
      m[j] = lo[j] < end[j] && (in[j] ? a.bic : a.boc)[lo[j]] == c[j]
                 ? (in[j] ? a.bin : a.bon)[lo[j]]
                 : 0u;
  }
}

// What a neighbour entry (block c, weight w) subtracts from its lane's sum:
// t1 for the changed cell of row r, then t2 for the one of row s
// (kernels.hpp:1444-1726 for out, 1153-1362 for in).  lead marks one entry
// per distinct block of the direction, kc is v's total weight to/from c, Mo
// and Mt the counts in rows r and s, ld the log2 of c's degree.  A block
// absent from the target row gives one term per list entry
// (kernels.hpp:1648-1652, 1696-1713; 1314-1318, 1348-1358); in-rows leave out
// blocks r and s.
__device__ __forceinline__ void entry_terms(const double* tab, bool ok, bool in, int32_t c,
                                            uint32_t w, bool lead, uint32_t kc, uint32_t Mo,
                                            uint32_t Mt, double ld, int r, int s, uint32_t niS,
                                            double& t1, double& t2) {
  const bool rs = c == r || c == s;
  const bool cell = ok && lead && !rs;
  const uint32_t y = Mt != 0u ? Mt + kc : in ? w : w - (c == r ? niS : 0u) + (c == s ? niS : 0u);
  t1 = cell ? gterm(tab, Mo - kc, ld) - gterm(tab, Mo, ld) : 0.0;
  t2 = cell || (ok && Mt == 0u && !(in && rs)) ? gterm(tab, y, ld) - gterm(tab, Mt, ld) : 0.0;
}

// Count changes of the new out-row r, out-row s, in-row r and in-row s away
// from the corners.  Every block c other than r and s loses v's weight kc
// from row r's cell and gains it in row s's, so the changes are v's degrees
// less its weights to r and s; where M[s][r] or M[s][s] is 0, the entries in
// that block add their own terms' counts (entry_terms): nR and nS of them.
// All modulo 2^32, as the entry-wise sums are.
struct RowChange {
  int m4, m5, m6, m7;
};
__device__ __forceinline__ RowChange row_change(const Corner& q, const RsWeights& w, uint32_t nR,
                                                uint32_t nS) {
  const uint32_t o = q.kO - w.koR - w.koS, i = q.kI - w.niR - w.niS;
  return RowChange{(int)(0u - o),
                   (int)(o + (q.Msr == 0u ? w.koR - nR * w.niS : 0u) +
                         (q.Mss == 0u ? w.koS + nS * w.niS : 0u)),
                   (int)(0u - i), (int)i};
}

// Block proposed by a vertex whose drawn neighbour lies in block cu
// (kernels.hpp:1000-1032): nbr_s holds the block's second-hop draw, or -1
// where its proposals are uniform.
__device__ __forceinline__ int proposed(const NodalArgs& a, int cu, int rnd) {
  const int nb = a.nbr_s[cu];
  return nb < 0 ? rnd : nb;
}

// Sum of the weights ws[b] over the set bits b of m.
template <class Mask>
__device__ __forceinline__ uint32_t mask_weight(const uint32_t* ws, Mask m) {
  uint32_t t = 0u;
  for (; m; m &= m - 1) t += ws[sizeof(Mask) == 8 ? __ffsll(m) - 1 : __ffs((unsigned)m) - 1];
  return t;
}

// One vertex (batch index i) on a group of L lanes with two entries a lane:
// L = 8 for at most 16 entries (four vertices a warp), L = 16 for at most 32
// (two), L = 32 for at most 64.  Entry k (out-entries, then in-entries) sits
// in slot k / L of lane k % L; a full warp whose directions both fit a lane
// each holds out-entry l and in-entry l in lane l.  buf: 128 words of the
// warp's shared memory.  Groups without a vertex of their own (active =
// false) repeat another's and write nothing.  GEN: the general mode (L = 8 or
// 16).
template <bool GIVEN, bool DENSE, bool GEN, int L>
__device__ __forceinline__ void group_vertex(const NodalArgs& a, int i, bool active, int lane,
                                             uint32_t* buf) {
  using Mask = typename std::conditional<L == 32, unsigned long long, uint32_t>::type;
  const int hl = lane & (L - 1), hb = lane & (32 - L);
  const int v = GIVEN ? a.verts[i] : a.lo + i;
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  const int32_t i0 = a.iptr[v], ni = a.iptr[v + 1] - i0;
  const bool split = L == 32 && no <= 32 && ni <= 32;  // a direction per slot
  int32_t c[2];
  uint32_t w[2], key[2];
  bool in[2], ok[2], loop[2];  // loop: an out-entry to v itself
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int k = hl + L * j;
    in[j] = split ? j == 1 : k >= no;
    const int e = split ? hl : in[j] ? k - no : k;
    ok[j] = e < (in[j] ? ni : no);
    c[j] = -1;  // the neighbour, then its block
    w[j] = 0u;
    if (ok[j]) {
      c[j] = __ldg((in[j] ? a.iidx + i0 : a.oidx + o0) + e);
      w[j] = a.unit ? 1u : __ldg((in[j] ? a.iw + i0 : a.ow + o0) + e);
    }
    loop[j] = GEN && !in[j] && c[j] == v;
  }
  const uint64_t deg = (uint64_t)a.kdo[v] + a.kdi[v];
  wait_kernel();
  if (ctl_stopped(a.ctl)) return;
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (ok[j]) c[j] = a.part[c[j]];
  const int r = a.part[v];
  P4 x{};
  if (!GIVEN) x = draw(a.seed, kRngNodalVertex, a.seq + ctl_itr(a.ctl) * a.seq_mul, (uint32_t)v);
  uint32_t* skey = buf + 2 * hb;
  uint32_t* sw = skey + 64;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    // direction in the top bit; idle slots match no entry
    key[j] = ok[j] ? (uint32_t)c[j] | (in[j] ? 0x80000000u : 0u) : 0xffffffffu;
    skey[hl + L * j] = key[j];
    sw[hl + L * j] = w[j];
  }
  const bool unit = __all_sync(kFull, w[0] <= 1u && w[1] <= 1u);
  __syncwarp();
  // the neighbour whose running weight first exceeds t
  // (choose_neighbored_node_block, kernels.hpp:877-939): with unit weights
  // it is entry t
  int s;
  if (GIVEN) {
    s = a.props_in[i];
  } else {
    const int rnd = (int)(x.v[0] % (uint32_t)a.B);
    const uint64_t t = scale_draw(x.v[1], deg);
    int at = -1;
    if (unit) {
      if (deg != 0) at = split && (int)t >= no ? 32 + (int)t - no : (int)t;
    } else {
      uint64_t incl[2] = {w[0], w[1]};
#pragma unroll
      for (int o = 1; o < L; o <<= 1) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint64_t y = __shfl_up_sync(kFull, incl[j], o);
          if (hl >= o) incl[j] += y;
        }
      }
      incl[1] += __shfl_sync(kFull, incl[0], hb + L - 1);
      const unsigned gm = L == 32 ? kFull : ((1u << (L & 31)) - 1u) << hb;
      const unsigned h0 = __ballot_sync(kFull, ok[0] && incl[0] > t) & gm;
      const unsigned h1 = __ballot_sync(kFull, ok[1] && incl[1] > t) & gm;
      at = h0 ? __ffs(h0) - 1 - hb : h1 ? L + __ffs(h1) - 1 - hb : -1;
    }
    s = rnd;
    if (deg != 0)
      s = proposed(a, at >= 0 ? (int)(skey[at] & 0x7fffffffu) : a.part[0], rnd);
  }
  double d = 0.0, logH = 0.0;
  if (__any_sync(kFull, r != s)) {
    // row r's counts and the column degrees need no proposal
    uint32_t Mo[2], Mt[2];
    double ld[2];
    bool want[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      want[j] = ok[j] && c[j] != r;
      ld[j] = ok[j] ? (in[j] ? a.ld_out : a.ld_in)[c[j]] : 0.0;
    }
    row_counts<DENSE, 2>(a, r, in, c, want, Mo);
    row_counts<DENSE, 2>(a, s, in, c, ok, Mt);
    const uint32_t mm =
        hl < 4 ? Rows<DENSE>(a, r, s).out_at((hl & 2) != 0, (hl & 1) ? s : r) : 0u;
    Corner q;
    load_degrees(a, v, r, s, q);
    // the entries of each block: bit k of eq[j] for entry k
    // (general mode: anyd, over both directions)
    Mask eq[2] = {0, 0}, anyd[2] = {0, 0};
    const int bound = split ? 32 + ni : no + ni;
    const int nm = L == 32 ? bound : __reduce_max_sync(kFull, bound);
#pragma unroll
    for (int b = 0; b < 2 * L; b += 4) {
      if (b >= nm) break;
      const uint4 g = *reinterpret_cast<const uint4*>(skey + b);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (g.x == key[j]) eq[j] |= (Mask)1 << b;
        if (g.y == key[j]) eq[j] |= (Mask)1 << (b + 1);
        if (g.z == key[j]) eq[j] |= (Mask)1 << (b + 2);
        if (g.w == key[j]) eq[j] |= (Mask)1 << (b + 3);
        if constexpr (GEN) {
          if (((g.x ^ key[j]) << 1) == 0u) anyd[j] |= (Mask)1 << b;
          if (((g.y ^ key[j]) << 1) == 0u) anyd[j] |= (Mask)1 << (b + 1);
          if (((g.z ^ key[j]) << 1) == 0u) anyd[j] |= (Mask)1 << (b + 2);
          if (((g.w ^ key[j]) << 1) == 0u) anyd[j] |= (Mask)1 << (b + 3);
        }
      }
    }
    // the entries in blocks r and s, per direction, and the self loops
    Mask inR = 0, inS = 0, selfs = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned bR = __ballot_sync(kFull, c[j] == r), bS = __ballot_sync(kFull, c[j] == s);
      const unsigned lm = L == 32 ? kFull : (1u << (L & 31)) - 1u;
      inR |= (Mask)((bR >> hb) & lm) << (L * j);
      inS |= (Mask)((bS >> hb) & lm) << (L * j);
      if constexpr (GEN) selfs |= (Mask)((__ballot_sync(kFull, loop[j]) >> hb) & lm) << (L * j);
    }
    const int nout = split ? 32 : no;
    const Mask out = nout >= 2 * L ? ~(Mask)0 : ((Mask)1 << nout) - 1;
    auto count = [](Mask m) {
      return (uint32_t)(sizeof(Mask) == 8 ? __popcll(m) : __popc((unsigned)m));
    };
    const uint32_t nR = count(inR & out), nS = count(inS & out);
    RsWeights rw{nR, nS, count(inR & ~out), count(inS & ~out)};
    uint32_t kc[2] = {count(eq[0]), count(eq[1])};
    if (!unit) {
      rw = RsWeights{mask_weight(sw, inR & out), mask_weight(sw, inS & out),
                     mask_weight(sw, inR & ~out), mask_weight(sw, inS & ~out)};
#pragma unroll
      for (int j = 0; j < 2; ++j) kc[j] = ok[j] ? mask_weight(sw, eq[j]) : 0u;
    }
    q.Mrr = __shfl_sync(kFull, mm, hb);
    q.Mrs = __shfl_sync(kFull, mm, hb + 1);
    q.Msr = __shfl_sync(kFull, mm, hb + 2);
    q.Mss = __shfl_sync(kFull, mm, hb + 3);
    const RowChange m = row_change(q, rw, nR, nS);
    double t1[2], t2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const Mask below = ((Mask)1 << (hl + L * j)) - 1;
      const bool lead = (eq[j] & below) == 0;
      if (GEN && a.exact) {
        t1[j] = ok[j] && lead && c[j] != r && c[j] != s
                    ? -exact_term(a.xlx, Mo[j], Mt[j], kc[j])
                    : 0.0;
        t2[j] = 0.0;
      } else {
        entry_terms(a.xlx, ok[j], in[j], c[j], w[j], lead, kc[j], Mo[j], Mt[j], ld[j], r, s,
                    rw.niS, t1[j], t2[j]);
      }
    }
    double acc = 0.0 - t1[0];
    acc -= t2[0];
    if constexpr (L == 32) {
      acc -= t1[1];
      acc -= t2[1];
      acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, hl);
    } else {
      double acc1 = 0.0 - t1[1];
      acc1 -= t2[1];
      uint32_t self = 0u;
      if constexpr (GEN) self = unit ? count(selfs) : mask_weight(sw, selfs);
      if (GEN && a.exact) {
        acc = corner_exact(a.xlx, q, rw, self, hl, acc);
        if constexpr (L == 8) acc1 = corner_exact(a.xlx, q, rw, self, hl + 8, acc1);
      } else if constexpr (L == 16) {
        acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, hl);
      } else {
        acc += corner_term<true, false>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, hl);
        acc1 += corner_term<false, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, hl + 8);
      }
      acc += acc1;
      if (GEN && a.mh) {
        // proposal weights once per block over both directions, then r and s
        Hast h[2];
        const Rows<DENSE> R(a, r, s);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const bool lead = (anyd[j] & (((Mask)1 << (hl + L * j)) - 1)) == 0;
          if (ok[j] && lead && c[j] != r && c[j] != s)
            hast_block<DENSE>(a, R, c[j], unit ? count(anyd[j]) : mask_weight(sw, anyd[j]), h[j]);
        }
        if (hl == 0) hast_rs<DENSE>(a, R, v, r, s, rw, self, h[0]);
        const double f = group_sum<L>(h[0].f + h[1].f), bk = group_sum<L>(h[0].b + h[1].b);
        if (no + ni != 0) logH = log(bk) - log(f);
      }
    }
    d = group_sum<L>(acc);
  }
  if (hl == 0 && active) {
    d = r != s ? d : 0.0;
    if constexpr (GEN) write_result_gen(a, GIVEN, i, r, s, d, r != s ? logH : 0.0, x.v[2]);
    else write_result(a, GIVEN, i, r, s, d);
  }
  __syncwarp();
}

// A vertex of more than kGroupEntries entries (at most kWarpList a
// direction) on the CTA, an entry (of up to 256) a thread and slot: on one
// warp such a vertex, the longest chain of a batch, set the launch time of
// graphs whose batches fit the GPU at once (20k HH: 34 us a launch, 14 with
// this path and group_vertex).  The terms are computed by entry and
// subtracted by warp 0 in the order the warp's lanes would: by entry index up
// to kWarpList entries, else by rank in the direction's (block, weight)
// order.  GEN: the general mode, always by rank, and with T = 32 on one warp
// for vertices of up to 64 entries.
template <int T, bool GEN>
struct LargeBuf {
  uint32_t key[2 * T], w[2 * T];
  double t1[2 * T], t2[2 * T];
  double f[GEN ? 2 * T : 1], b[GEN ? 2 * T : 1];  // proposal weights
  uint32_t ord[2 * T];  // (direction, block, entry), in one word
  uint32_t cnt[7];  // koR, koS, niR, niS, out-entries in r, in s, self loops
};
constexpr int kOrdBlocks = 1 << 22;  // blocks whose entries' order fits a word

// First index in the ascending key[lo, hi) whose key exceeds x.
__device__ __forceinline__ int upper_bound(const uint32_t* key, int lo, int hi, uint32_t x) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (key[mid] > x) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

template <bool GIVEN, bool DENSE, bool GEN, int T>
__device__ void large_vertex(const NodalArgs& a, int i, LargeBuf<T, GEN>& sm) {
  static_assert(T == 32 || (T == kNodalWarps * 32 && T == kWarpList), "a warp or the CTA");
  const int tid = T == 32 ? threadIdx.x & 31 : threadIdx.x, lane = tid & 31;
  auto sync = [] {
    if (T == 32) __syncwarp();
    else __syncthreads();
  };
  const int v = GIVEN ? a.verts[i] : a.lo + i;
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  const int32_t i0 = a.iptr[v], ni = a.iptr[v + 1] - i0;
  const int n = no + ni;
  int32_t c[2];
  uint32_t w[2], key[2], ord[2];
  bool in[2], ok[2];
  uint32_t selfp = 0u;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int k = tid + T * j;
    ok[j] = k < n;
    in[j] = k >= no;
    const int e = in[j] ? k - no : k;
    c[j] = -1;  // the neighbour, then its block
    w[j] = 0u;
    if (ok[j]) {
      c[j] = __ldg((in[j] ? a.iidx + i0 : a.oidx + o0) + e);
      w[j] = a.unit ? 1u : __ldg((in[j] ? a.iw + i0 : a.ow + o0) + e);
      if (GEN && !in[j] && c[j] == v) selfp += w[j];
    }
  }
  wait_kernel();
  if (ctl_stopped(a.ctl)) return;  // the same in every thread
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int k = tid + T * j;
    if (ok[j]) c[j] = a.part[c[j]];
    key[j] = ok[j] ? (uint32_t)c[j] | (in[j] ? 0x80000000u : 0u) : 0xffffffffu;
    ord[j] = ok[j] ? (in[j] ? 1u << 30 : 0u) | (uint32_t)c[j] << 8 | (uint32_t)k : 0xffffffffu;
    sm.key[k] = key[j];
    sm.w[k] = w[j];
    sm.ord[k] = ord[j];
  }
  const int r = a.part[v];
  if (tid < 7) sm.cnt[tid] = 0u;
  const bool light = w[0] <= 1u && w[1] <= 1u;
  bool unit;
  if (T == 32) {
    unit = __all_sync(kFull, light);
    __syncwarp();
  } else {
    unit = __syncthreads_and(light);
  }
  uint32_t u2 = 0u;
  int s;
  if (GIVEN) {
    s = a.props_in[i];
  } else {
    const P4 x = draw(a.seed, kRngNodalVertex, a.seq + ctl_itr(a.ctl) * a.seq_mul, (uint32_t)v);
    u2 = x.v[2];
    const int rnd = (int)(x.v[0] % (uint32_t)a.B);
    const uint64_t t = scale_draw(x.v[1], (uint64_t)a.kdo[v] + a.kdi[v]);
    int at = (int)t;
    if (!unit) {  // the first entry whose running weight exceeds t
      at = -1;
      uint64_t acc = 0;
      for (int k0 = 0; k0 < n && at < 0; k0 += 32) {
        uint64_t incl = sm.w[k0 + lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint64_t y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        const unsigned hit = __ballot_sync(kFull, k0 + lane < n && acc + incl > t);
        if (hit) at = k0 + __ffs(hit) - 1;
        acc += __shfl_sync(kFull, incl, 31);
      }
    }
    s = proposed(a, at >= 0 ? (int)(sm.key[at] & 0x7fffffffu) : a.part[0], rnd);
  }
  if (r == s) {  // the same in every thread
    if (tid == 0) {
      if constexpr (GEN) write_result_gen(a, GIVEN, i, r, s, 0.0, 0.0, u2);
      else write_result(a, GIVEN, i, r, s, 0.0);
    }
    sync();
    return;
  }
  uint32_t Mo[2], Mt[2];
  double ld[2];
  bool want[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    want[j] = ok[j] && c[j] != r;
    ld[j] = ok[j] ? (in[j] ? a.ld_out : a.ld_in)[c[j]] : 0.0;
    if (c[j] == r) {
      atomicAdd(sm.cnt + (in[j] ? 2 : 0), w[j]);
      if (!in[j]) atomicAdd(sm.cnt + 4, 1u);
    }
    if (c[j] == s) {
      atomicAdd(sm.cnt + (in[j] ? 3 : 1), w[j]);
      if (!in[j]) atomicAdd(sm.cnt + 5, 1u);
    }
  }
  if (GEN && selfp) atomicAdd(sm.cnt + 6, selfp);
  row_counts<DENSE, 2>(a, r, in, c, want, Mo);
  row_counts<DENSE, 2>(a, s, in, c, ok, Mt);
  Corner q{};
  if (tid < 32) q = load_corner<DENSE>(a, v, r, s, lane);
  // each entry's block total, whether an entry of its block comes before it
  // in the summing order, and its place in that order
  // (general mode: also the block's total over both directions, and whether
  // it has an out-entry)
  uint32_t kc[2] = {0u, 0u}, kany[2] = {0u, 0u};
  int pos[2];
  bool lead[2], outside[2] = {false, false};
  const bool by_index = !GEN && n <= kWarpList;
  if (by_index) {
    bool before = false;
    for (int b = 0; b < n; b += 4) {  // idle slots match no entry
      const uint4 g = *reinterpret_cast<const uint4*>(sm.key + b);
      const uint4 u = *reinterpret_cast<const uint4*>(sm.w + b);
      kc[0] += (g.x == key[0] ? u.x : 0u) + (g.y == key[0] ? u.y : 0u) +
               (g.z == key[0] ? u.z : 0u) + (g.w == key[0] ? u.w : 0u);
      before = before || (b < tid && g.x == key[0]) || (b + 1 < tid && g.y == key[0]) ||
               (b + 2 < tid && g.z == key[0]) || (b + 3 < tid && g.w == key[0]);
    }
    lead[0] = !before;
    lead[1] = false;
    pos[0] = tid;
    pos[1] = tid + T;
  } else if (a.B <= kOrdBlocks) {
    // the order by (direction, block, entry) is that of one word per entry; in
    // it a block's entries are a run.  With equal weights it is the order
    // wanted, and a block's total the length of its run; otherwise its run is
    // walked for the total and for the entries of less weight.  (The loop over
    // pairs with weights, below, set the launch time: 20k HH partitions 43.4 ms
    // with it, 37.8 this way; a weighted sweep of 30k vertices of 150 entries
    // 0.93 and 0.58 ms.)
    int rank[2] = {0, 0};
#pragma unroll 4
    for (int b = 0; b < n; b += 4) {  // idle slots come last
      const uint4 g = *reinterpret_cast<const uint4*>(sm.ord + b);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        rank[j] += (g.x < ord[j] ? 1 : 0) + (g.y < ord[j] ? 1 : 0) + (g.z < ord[j] ? 1 : 0) +
                   (g.w < ord[j] ? 1 : 0);
    }
    // the keys in order, then the weights (unless all are 1), where the terms
    // will go
    uint32_t* const run = reinterpret_cast<uint32_t*>(sm.t1);
    uint32_t* const runw = run + 2 * T;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (!ok[j]) continue;
      run[rank[j]] = key[j];
      if (!unit) runw[rank[j]] = w[j];
    }
    sync();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      lead[j] = ok[j] && (rank[j] == 0 || run[rank[j] - 1] != key[j]);
      pos[j] = rank[j];
      if (unit) {
        if (lead[j]) kc[j] = (uint32_t)(upper_bound(run, rank[j], n, key[j]) - rank[j]);
      } else if (ok[j]) {
        int lo = rank[j], less = 0;
        while (lo > 0 && run[lo - 1] == key[j]) --lo;
        for (int q = lo; q < n && run[q] == key[j]; ++q) {
          const uint32_t u = runw[q];
          kc[j] += u;
          less += u < w[j] || (u == w[j] && q < rank[j]) ? 1 : 0;
        }
        lead[j] = less == 0;
        pos[j] = lo + less;
      }
      if constexpr (GEN) {
        if (a.mh && lead[j]) {
          const uint32_t other = key[j] ^ 0x80000000u;
          const int lo = in[j] ? 0 : no, hi = in[j] ? no : n;
          const int k1 = upper_bound(run, lo, hi, other);
          const int k0 = other == 0u ? lo : upper_bound(run, lo, hi, other - 1u);
          kany[j] = kc[j] + (uint32_t)(k1 - k0);
          if (!unit) {
            kany[j] = kc[j];
            for (int q = k0; q < k1; ++q) kany[j] += runw[q];
          }
          outside[j] = in[j] && k1 > k0;
        }
      }
    }
  } else {
    int rank[2] = {0, 0}, same[2] = {0, 0};
    for (int b = 0; b < n; ++b) {
      const uint32_t g = sm.key[b], u = sm.w[b];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bool e = g == key[j];
        kc[j] += e ? u : 0u;
        const bool first = e && (u < w[j] || (u == w[j] && b < tid + T * j));
        same[j] += first ? 1 : 0;
        rank[j] += first || g < key[j] ? 1 : 0;
        if constexpr (GEN) {
          const bool same_block = ((g ^ key[j]) << 1) == 0u;
          kany[j] += same_block ? u : 0u;
          outside[j] = outside[j] || (same_block && b < no);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      lead[j] = same[j] == 0;
      pos[j] = rank[j];  // out-entries' keys rank before every in-entry's
    }
  }
  sync();
  const RsWeights rw{sm.cnt[0], sm.cnt[1], sm.cnt[2], sm.cnt[3]};
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (!ok[j]) continue;
    if (GEN && a.exact) {
      sm.t1[pos[j]] = lead[j] && c[j] != r && c[j] != s
                          ? -exact_term(a.xlx, Mo[j], Mt[j], kc[j])
                          : 0.0;
      sm.t2[pos[j]] = 0.0;
    } else {
      entry_terms(a.xlx, true, in[j], c[j], w[j], lead[j], kc[j], Mo[j], Mt[j], ld[j], r, s,
                  rw.niS, sm.t1[pos[j]], sm.t2[pos[j]]);
    }
    if constexpr (GEN) {
      // a block on both lists is counted with the out-list
      Hast h;
      if (a.mh && lead[j] && c[j] != r && c[j] != s && !(in[j] && outside[j]))
        hast_block<DENSE>(a, Rows<DENSE>(a, r, s), c[j], kany[j], h);
      sm.f[pos[j]] = h.f;
      sm.b[pos[j]] = h.b;
    }
  }
  sync();
  if (tid < 32) {
    double acc = 0.0;
    Hast h;
    const int n0 = by_index ? n : no;
    for (int lo = 0, hi = n0; lo < n; lo = hi, hi = n)
      for (int p = lo + lane; p < hi; p += 32) {
        acc -= sm.t1[p];
        acc -= sm.t2[p];
        if constexpr (GEN) {
          h.f += sm.f[p];
          h.b += sm.b[p];
        }
      }
    if (GEN && a.exact) {
      acc = corner_exact(a.xlx, q, rw, sm.cnt[6], lane, acc);
    } else {
      const RowChange m = row_change(q, rw, sm.cnt[4], sm.cnt[5]);
      acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, lane);
    }
    const double d = warp_sum(acc);
    if constexpr (GEN) {
      double logH = 0.0;
      if (a.mh) {
        if (lane == 0) hast_rs<DENSE>(a, Rows<DENSE>(a, r, s), v, r, s, rw, sm.cnt[6], h);
        const double f = warp_sum(h.f), b = warp_sum(h.b);
        logH = log(b) - log(f);
      }
      if (lane == 0) write_result_gen(a, GIVEN, i, r, s, d, logH, u2);
    } else if (lane == 0) {
      write_result(a, GIVEN, i, r, s, d);
    }
  }
  sync();  // the next vertex reuses the buffer
}

// exact_term of an entry added to q where it leads its block.
template <bool DENSE>
__device__ __forceinline__ void entry_exact(const NodalArgs& a, const Rows<DENSE>& R, int r, int s,
                                            bool in, int32_t c, bool leader, uint32_t kc,
                                            Acc& q) {
  if (!leader || c == r || c == s) return;
  q.acc += exact_term(a.xlx, in ? R.in_r(c) : R.out_r(c), in ? R.in_s(c) : R.out_s(c), kc);
}

// v's self-loop weight (group sum over its out-list).
template <int G>
__device__ uint32_t self_weight(const NodalArgs& a, int v, const Group<G>& grp) {
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  uint32_t t = 0u;
  for (int k = grp.rank(); k < no; k += G)
    if (__ldg(a.oidx + o0 + k) == v) t += __ldg(a.ow + o0 + k);
  return (uint32_t)grp.sum_ll(t);
}

// Group totals, then the corner terms (exact or GSAP's) on warp 0, then the
// sums of dS and of the proposal weights.
template <bool DENSE, int G>
__device__ double finish_gen(const NodalArgs& a, const Rows<DENSE>& R, int v, int r, int s,
                             const RsWeights& w, uint32_t self, Acc q, Hast h,
                             const Group<G>& grp, double& logH) {
  if (a.exact) {
    if (G == 32 || threadIdx.x < 32)
      q.acc = corner_exact(a.xlx, load_corner<DENSE>(a, v, r, s, threadIdx.x & 31), w, self,
                           threadIdx.x & 31, q.acc);
  } else {
    q.m4 = (int)grp.sum_ll(q.m4);
    q.m5 = (int)grp.sum_ll(q.m5);
    q.m6 = (int)grp.sum_ll(q.m6);
    q.m7 = (int)grp.sum_ll(q.m7);
    if (G == 32 || threadIdx.x < 32)
      corner_terms<DENSE>(a, R, v, r, s, w, q, threadIdx.x & 31);
  }
  logH = 0.0;
  if (a.mh) {
    const double f = grp.sum(h.f), b = grp.sum(h.b);
    if ((uint64_t)a.kdo[v] + a.kdi[v] != 0u) logH = log(b) - log(f);
  }
  return grp.sum(q.acc);
}

template <bool DENSE, int G>
__device__ double delta_hashed_gen(const NodalArgs& a, int v, int r, int s, HashTab h, int* flag,
                                   const Group<G>& grp, double& logH) {
  const int t = grp.rank();
  const Rows<DENSE> R(a, r, s);
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  const int32_t i0 = a.iptr[v], ni = a.iptr[v + 1] - i0;
  logH = 0.0;
  uint32_t koR = 0, koS = 0, niR = 0, niS = 0;
  for (int k = t; k < no; k += G) {
    int32_t c = a.part[__ldg(a.oidx + o0 + k)];
    uint32_t w = __ldg(a.ow + o0 + k);
    koR += c == r ? w : 0u;
    koS += c == s ? w : 0u;
  }
  for (int k = t; k < ni; k += G) {
    int32_t c = a.part[__ldg(a.iidx + i0 + k)];
    uint32_t w = __ldg(a.iw + i0 + k);
    niR += c == r ? w : 0u;
    niS += c == s ? w : 0u;
  }
  const RsWeights rw{(uint32_t)grp.sum_ll(koR), (uint32_t)grp.sum_ll(koS),
                     (uint32_t)grp.sum_ll(niR), (uint32_t)grp.sum_ll(niS)};
  const uint32_t self = self_weight<G>(a, v, grp);
  Acc q;
  Hast hs;
  // dS: per direction, one hash class of blocks per pass
  for (int dir = 0; dir < 2; ++dir) {
    const int32_t base = dir == 0 ? o0 : i0, n = dir == 0 ? no : ni;
    const int32_t* idx = dir == 0 ? a.oidx : a.iidx;
    const uint32_t* wt = dir == 0 ? a.ow : a.iw;
    const uint32_t P = (uint32_t)((n + kHashSlots / 4 - 1) / (kHashSlots / 4));
    for (uint32_t pass = 0; pass < P; ++pass) {
      for (int i = t; i < kHashSlots; i += G) {
        h.key[i] = -1;
        h.sum[i] = 0u;
        h.first[i] = 0x7fffffff;
      }
      if (t == 0) *flag = 0;
      grp.sync();
      for (int k = t; k < n; k += G) {
        int32_t c = a.part[__ldg(idx + base + k)];
        if (hclass(c, P) == pass && !hash_add(h, c, __ldg(wt + base + k), k)) *flag = 1;
      }
      grp.sync();
      if (*flag) return __longlong_as_double(0x7ff8000000000000ll);  // table overflow
      for (int k = t; k < n; k += G) {
        int32_t c = a.part[__ldg(idx + base + k)];
        if (hclass(c, P) != pass) continue;
        const int slot = hash_find(h, c);
        const bool leader = h.first[slot] == k;
        const uint32_t kc = h.sum[slot];
        if (a.exact) entry_exact<DENSE>(a, R, r, s, dir == 1, c, leader, kc, q);
        else entry<DENSE>(a, R, r, s, rw.niS, dir == 1, c, __ldg(wt + base + k), leader, kc, q);
      }
      grp.sync();
    }
  }
  if (a.mh) {
    // proposal weights: per block over both directions, one hash class per pass
    const int n = no + ni;
    const uint32_t P = (uint32_t)((n + kHashSlots / 4 - 1) / (kHashSlots / 4));
    for (uint32_t pass = 0; pass < P; ++pass) {
      for (int i = t; i < kHashSlots; i += G) {
        h.key[i] = -1;
        h.sum[i] = 0u;
        h.first[i] = 0x7fffffff;
      }
      if (t == 0) *flag = 0;
      grp.sync();
      for (int k = t; k < n; k += G) {
        const bool in = k >= no;
        const int j = in ? k - no : k;
        const int32_t c = a.part[__ldg((in ? a.iidx + i0 : a.oidx + o0) + j)];
        if (c == r || c == s || hclass(c, P) != pass) continue;
        if (!hash_add(h, c, __ldg((in ? a.iw + i0 : a.ow + o0) + j), k)) *flag = 1;
      }
      grp.sync();
      if (*flag) return __longlong_as_double(0x7ff8000000000000ll);
      for (int i = t; i < kHashSlots; i += G)
        if (h.key[i] != -1) hast_block<DENSE>(a, R, h.key[i], h.sum[i], hs);
      grp.sync();
    }
    if (t == 0) hast_rs<DENSE>(a, R, v, r, s, rw, self, hs);
  }
  return finish_gen<DENSE, G>(a, R, v, r, s, rw, self, q, hs, grp, logH);
}

// A vertex of kGroupEntries to kWideEntries entries on a warp, four entries a
// lane: the terms and sums of large_vertex (by index), with fewer instructions
// and a longer chain.  A batch of more such vertices than the GPU holds CTAs is
// bound by instructions, one of fewer by the chain.  buf: 512 words of the
// warp's shared memory.
template <bool GIVEN, bool DENSE>
__device__ void wide_vertex(const NodalArgs& a, int i, int lane, uint32_t* buf) {
  constexpr int S = kWideEntries / 32;
  const int v = GIVEN ? a.verts[i] : a.lo + i;
  const int32_t o0 = a.optr[v], no = a.optr[v + 1] - o0;
  const int32_t i0 = a.iptr[v], ni = a.iptr[v + 1] - i0;
  const int n = no + ni;
  int32_t c[S];
  uint32_t w[S];
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const int k = lane + 32 * j;
    const bool in = k >= no;
    const int e = in ? k - no : k;
    c[j] = -1;  // the neighbour, then its block
    w[j] = 0u;
    if (k < n) {
      c[j] = __ldg((in ? a.iidx + i0 : a.oidx + o0) + e);
      w[j] = a.unit ? 1u : __ldg((in ? a.iw + i0 : a.ow + o0) + e);
    }
  }
  const uint64_t deg = (uint64_t)a.kdo[v] + a.kdi[v];
  wait_kernel();
  if (ctl_stopped(a.ctl)) return;
  uint32_t* const skey = buf;
  uint32_t* const sw = buf + kWideEntries;
  bool light = true;
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const int k = lane + 32 * j;
    if (k < n) c[j] = a.part[c[j]];
    // direction in the top bit; idle slots match no entry
    skey[k] = k < n ? (uint32_t)c[j] | (k >= no ? 0x80000000u : 0u) : 0xffffffffu;
    sw[k] = w[j];
    light = light && w[j] <= 1u;
  }
  const int r = a.part[v];
  const bool unit = __all_sync(kFull, light);
  __syncwarp();
  int s;
  if (GIVEN) {
    s = a.props_in[i];
  } else {
    const P4 x = draw(a.seed, kRngNodalVertex, a.seq + ctl_itr(a.ctl) * a.seq_mul, (uint32_t)v);
    const int rnd = (int)(x.v[0] % (uint32_t)a.B);
    const uint64_t t = scale_draw(x.v[1], deg);
    int at = (int)t;
    if (!unit) {  // the first entry whose running weight exceeds t
      at = -1;
      uint64_t acc = 0;
      for (int k0 = 0; k0 < n && at < 0; k0 += 32) {
        uint64_t incl = sw[k0 + lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint64_t y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        const unsigned hit = __ballot_sync(kFull, k0 + lane < n && acc + incl > t);
        if (hit) at = k0 + __ffs(hit) - 1;
        acc += __shfl_sync(kFull, incl, 31);
      }
    }
    s = proposed(a, at >= 0 ? (int)(skey[at] & 0x7fffffffu) : a.part[0], rnd);
  }
  double d = 0.0;
  if (r != s) {  // the same in every lane
    // the counts first: the table below is built while they are on their way
    uint32_t Mo[S], Mt[S];
    bool in[S], ok[S], want[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int k = lane + 32 * j;
      in[j] = k >= no;
      ok[j] = k < n;
      want[j] = ok[j] && c[j] != r;
    }
    row_counts<DENSE, S>(a, r, in, c, want, Mo);
    row_counts<DENSE, S>(a, s, in, c, ok, Mt);
    const uint32_t mm =
        lane < 4 ? Rows<DENSE>(a, r, s).out_at((lane & 2) != 0, (lane & 1) ? s : r) : 0u;
    // v's weights to and from r and s, and its out-entries there
    uint32_t oR = 0u, oS = 0u, iR = 0u, iS = 0u, nR = 0u, nS = 0u;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const bool in = lane + 32 * j >= no, hr = c[j] == r, hs = c[j] == s;
      oR += hr && !in ? w[j] : 0u;
      oS += hs && !in ? w[j] : 0u;
      iR += hr && in ? w[j] : 0u;
      iS += hs && in ? w[j] : 0u;
      nR += hr && !in ? 1u : 0u;
      nS += hs && !in ? 1u : 0u;
    }
    const RsWeights rw{__reduce_add_sync(kFull, oR), __reduce_add_sync(kFull, oS),
                       __reduce_add_sync(kFull, iR), __reduce_add_sync(kFull, iS)};
    nR = __reduce_add_sync(kFull, nR);
    nS = __reduce_add_sync(kFull, nS);
    // each entry's block by a table from key to one of its entries, and there
    // the block's total and first entry
    uint32_t* const tab = buf + 2 * kWideEntries;
    auto fill = [&](uint32_t x, uint32_t y) {
      *reinterpret_cast<uint4*>(tab + 4 * lane) = make_uint4(x, x, x, x);
      *reinterpret_cast<uint4*>(tab + kWideEntries + 4 * lane) = make_uint4(y, y, y, y);
      __syncwarp();
    };
    fill(~0u, ~0u);
    int own[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int k = lane + 32 * j;
      own[j] = k;
      if (k >= n) continue;
      const uint32_t key = skey[k];
      for (uint32_t q = key * 2654435761u >> 24;; q = (q + 1) & (2 * kWideEntries - 1)) {
        const uint32_t cur = atomicCAS(tab + q, ~0u, (uint32_t)k);
        if (cur != ~0u) own[j] = (int)cur;
        if (cur == ~0u || skey[cur] == key) break;  // at most half the slots fill
        own[j] = k;
      }
    }
    __syncwarp();
    fill(0u, ~0u);
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int k = lane + 32 * j;
      if (k >= n) continue;
      atomicAdd(tab + own[j], w[j]);
      atomicMin(tab + kWideEntries + own[j], (uint32_t)k);
    }
    __syncwarp();
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      if (32 * j >= n) break;
      const bool lead = tab[kWideEntries + own[j]] == (uint32_t)(lane + 32 * j);
      const double ld = ok[j] ? (in[j] ? a.ld_out : a.ld_in)[c[j]] : 0.0;
      double t1, t2;
      entry_terms(a.xlx, ok[j], in[j], c[j], w[j], lead, tab[own[j]], Mo[j], Mt[j], ld, r, s,
                  rw.niS, t1, t2);
      acc -= t1;
      acc -= t2;
    }
    Corner q;
    load_degrees(a, v, r, s, q);
    q.Mrr = __shfl_sync(kFull, mm, 0);
    q.Mrs = __shfl_sync(kFull, mm, 1);
    q.Msr = __shfl_sync(kFull, mm, 2);
    q.Mss = __shfl_sync(kFull, mm, 3);
    const RowChange m = row_change(q, rw, nR, nS);
    acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, lane);
    d = warp_sum(acc);
  }
  if (lane == 0) write_result(a, GIVEN, i, r, s, d);
  __syncwarp();
}

// Work items of the warp kernel, larger vertices first (as the host lists
// them: a longest-first schedule): a CTA per large vertex, then a warp per
// vertex that wide_vertex takes and per vertex of up to 64 entries, per two of
// up to 32 and per four small ones.
struct NodalItems {
  int large, wide, mid64, mid32, small;  // large in CTAs, the others in warps
  __host__ __device__ NodalItems(const NodalArgs& a)
      : large(a.nlarge), wide(a.nwide), mid64(a.nmid64),
        mid32((a.nmid - a.nlarge - a.nwide - a.nmid64 + 1) / 2), small((a.nsmall + 3) / 4) {}
  __host__ __device__ int ctas() const {
    return large + (wide + mid64 + mid32 + small + kNodalWarps - 1) / kNodalWarps;
  }
};

template <bool GIVEN, bool DENSE, bool GEN>
struct NodalBody {
  using Args = NodalArgs;
  static constexpr int kThreads = kNodalWarps * 32;
  static constexpr int kMinBlocks = GEN ? 5 : 8;
  static constexpr bool kEarly = true;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    using Large = LargeBuf<kThreads, GEN>;
    // per warp: the keys and weights of wide_vertex and group_vertex, or
    // (general mode) a 33-64-entry vertex's LargeBuf
    using Mid = LargeBuf<32, GEN>;
    constexpr size_t kWarpBytes =
        GEN ? (sizeof(Mid) + 15) / 16 * 16 : 4 * kWideEntries * sizeof(uint32_t);
    constexpr size_t kBytes =
        sizeof(Large) > kNodalWarps * kWarpBytes ? sizeof(Large) : kNodalWarps * kWarpBytes;
    __shared__ __align__(16) unsigned char raw[kBytes];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* const own = raw + kWarpBytes * wid;
    uint32_t* const buf = reinterpret_cast<uint32_t*>(own);
    const NodalItems n(a);
    const int nmid32 = a.nmid - a.nlarge - a.nwide - a.nmid64;
    const int32_t *wide = a.mid + a.nlarge, *mid64 = wide + a.nwide, *mid32 = mid64 + a.nmid64;
    for (int blk = vb; blk < n.ctas(); blk += vg) {
      if (blk < n.large) {
        large_vertex<GIVEN, DENSE, GEN, kThreads>(a, a.mid[blk], *reinterpret_cast<Large*>(raw));
        continue;
      }
      int it = (blk - n.large) * kNodalWarps + wid;
      if constexpr (!GEN) {  // general mode has none
        if (it < n.wide) {
          wide_vertex<GIVEN, DENSE>(a, wide[it], lane, buf);
          continue;
        }
        it -= n.wide;
      }
      if (it < n.mid64) {
        if constexpr (GEN)
          large_vertex<GIVEN, DENSE, GEN, 32>(a, mid64[it], *reinterpret_cast<Mid*>(own));
        else
          group_vertex<GIVEN, DENSE, GEN, 32>(a, mid64[it], true, lane, buf);
        continue;
      }
      it -= n.mid64;
      if (it < n.mid32) {
        const int q = 2 * it + (lane >> 4);
        group_vertex<GIVEN, DENSE, GEN, 16>(a, mid32[min(q, nmid32 - 1)], q < nmid32, lane, buf);
        continue;
      }
      it -= n.mid32;
      if (it < n.small) {
        const int q = 4 * it + (lane >> 3);
        group_vertex<GIVEN, DENSE, GEN, 8>(a, a.small[min(q, a.nsmall - 1)], q < a.nsmall, lane,
                                           buf);
      }
    }
  }
};

// What the CTA paths of heavy vertices share: a vertex's entries (out-entries,
// then in-entries) as direction-tagged keys, and a shared-memory table from
// key to the key's total weight and first entry (open addressing).
struct HeavyEntries {
  const NodalArgs& a;
  int32_t o0, i0;
  int no, n;
  bool unit;  // every weight is 1
  __device__ HeavyEntries(const NodalArgs& args, int v)
      : a(args), o0(args.optr[v]), i0(args.iptr[v]), no(args.optr[v + 1] - o0),
        n(no + args.iptr[v + 1] - i0) {
    // weights are at least 1
    unit = (uint64_t)args.kdo[v] + args.kdi[v] == (uint64_t)n;
  }
  __device__ __forceinline__ uint32_t key(int k) const {
    return k < no ? (uint32_t)a.part[__ldg(a.oidx + o0 + k)]
                  : (uint32_t)a.part[__ldg(a.iidx + i0 + k - no)] | 0x80000000u;
  }
  __device__ __forceinline__ uint32_t w(int k) const {
    return unit ? 1u : k < no ? __ldg(a.ow + o0 + k) : __ldg(a.iw + i0 + k - no);
  }
};

struct HeavyTab {
  int32_t* key;  // -1 = empty (blocks lie below 2^31 - 1, so no key is -1)
  uint32_t* sum;
  int32_t* first;
  int slots;  // a power of two
  __device__ __forceinline__ void clear() const {
    for (int k = threadIdx.x; k < slots; k += kHeavyThreads) {
      key[k] = -1;
      sum[k] = 0u;
      first[k] = 0x7fffffff;
    }
  }
  __device__ __forceinline__ uint32_t slot(uint32_t x) const {
    return (x * 2654435761u) >> 16 & (uint32_t)(slots - 1);
  }
  // entry k of key x and weight w; false when the table is full
  __device__ __forceinline__ bool add(uint32_t x, uint32_t w, int k) const {
    uint32_t q = slot(x);
    for (int probe = 0; probe < slots; ++probe, q = (q + 1) & (uint32_t)(slots - 1)) {
      int32_t cur = *(volatile int32_t*)(key + q);
      if (cur == -1) cur = atomicCAS(key + q, -1, (int32_t)x);
      if (cur == -1 || cur == (int32_t)x) {
        atomicAdd(sum + q, w);
        atomicMin(first + q, k);
        return true;
      }
    }
    return false;
  }
  __device__ __forceinline__ uint32_t find(uint32_t x) const {
    uint32_t q = slot(x);
    for (int probe = 0; probe < slots && key[q] != (int32_t)x; ++probe)
      q = (q + 1) & (uint32_t)(slots - 1);
    return q;
  }
};

// The block that v proposes (the same in every thread of the CTA); wsum and
// at are the CTA's shared scratch, get(k) an entry's key.
template <bool GIVEN, class Get>
__device__ __forceinline__ int heavy_proposal(const NodalArgs& a, int i, int v,
                                              const HeavyEntries& e, unsigned long long* wsum,
                                              int* at, Get get) {
  if (GIVEN) return a.props_in[i];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const P4 x = draw(a.seed, kRngNodalVertex, a.seq + ctl_itr(a.ctl) * a.seq_mul, (uint32_t)v);
  const int rnd = (int)(x.v[0] % (uint32_t)a.B);
  const uint64_t target = scale_draw(x.v[1], (uint64_t)a.kdo[v] + a.kdi[v]);
  int k = (int)target;
  if (!e.unit) {
    // the first entry whose running weight exceeds the target: the thread
    // whose run of consecutive entries holds it
    if (t == 0) *at = -1;
    const int per = (e.n + kHeavyThreads - 1) / kHeavyThreads;
    const int k0 = min(e.n, t * per), k1 = min(e.n, k0 + per);
    uint64_t own = 0;
    for (int q = k0; q < k1; ++q) own += e.w(q);
    uint64_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    for (int q = 0; q < wid; ++q) incl += wsum[q];
    uint64_t run = incl - own;
    if (run <= target && target < incl)
      for (int q = k0; q < k1; ++q) {
        run += e.w(q);
        if (run > target) {
          *at = q;
          break;
        }
      }
    __syncthreads();
    k = *at;
  }
  return proposed(a, k >= 0 ? (int)(get(k) & 0x7fffffffu) : a.part[0], rnd);
}

// koR, koS, niR, niS, out-entries in r, in s of one entry into cnt[0..5].
__device__ __forceinline__ void add_rs(uint32_t* cnt, bool in, int c, int r, int s, uint32_t w) {
  if (c == r) {
    atomicAdd(cnt + (in ? 2 : 0), w);
    if (!in) atomicAdd(cnt + 4, 1u);
  }
  if (c == s) {
    atomicAdd(cnt + (in ? 3 : 1), w);
    if (!in) atomicAdd(cnt + 5, 1u);
  }
}

// A vertex of more than kWarpList entries in a direction, at most
// kHubEntries in all, on a CTA: its threads take the entries of each
// direction strided by kHeavyThreads and subtract their terms in that order.
// Up to four entries a thread are in flight at a time.  The table and the
// keys take 28 KB of shared memory, so that the SM keeps its L1 for these
// CTAs and the warp kernel's beside them (with the hubs' 112 KB here, the
// terms of a 500-entry vertex alone took 5.6 us, all of it L2 latency).  13 us
// a launch at 200k HH.
constexpr size_t kHeavySmem = (3 * 2 * kHubEntries + kHubEntries) * sizeof(int32_t);

template <bool GIVEN, bool DENSE>
__device__ void heavy_vertex(const NodalArgs& a, int i, const Group<kHeavyThreads>& grp) {
  constexpr int T = kHeavyThreads, U = 4;
  extern __shared__ unsigned long long hsm[];
  __shared__ unsigned long long wsum[T / 32];
  __shared__ uint32_t cnt[6];
  __shared__ int s_at;
  const int t = threadIdx.x, lane = t & 31;
  const int v = GIVEN ? a.verts[i] : a.lo + i;
  const HeavyEntries e(a, v);
  const int n = e.n, no = e.no;
  int slots = 512;
  while (slots < 2 * n) slots <<= 1;
  const HeavyTab tab{(int32_t*)hsm, (uint32_t*)hsm + 2 * kHubEntries,
                     (int32_t*)hsm + 4 * kHubEntries, slots};
  uint32_t* const stage = (uint32_t*)hsm + 6 * kHubEntries;
#pragma unroll 4
  for (int k = t; k < n; k += T) stage[k] = e.key(k);
  const int r = a.part[v];
  tab.clear();
  if (t < 6) cnt[t] = 0u;
  __syncthreads();
  const int s =
      heavy_proposal<GIVEN>(a, i, v, e, wsum, &s_at, [&](int k) { return stage[k]; });
  if (r == s) {  // the same in every thread
    if (t == 0) write_result(a, GIVEN, i, r, s, 0.0);
    __syncthreads();
    return;
  }
  Corner q{};
  if (t < 32) q = load_corner<DENSE>(a, v, r, s, lane);
  for (int k = t; k < n; k += T) {
    const uint32_t key = stage[k], w = e.w(k);
    add_rs(cnt, k >= no, (int)(key & 0x7fffffffu), r, s, w);
    tab.add(key, w, k);  // at most half full
  }
  __syncthreads();
  const RsWeights rw{cnt[0], cnt[1], cnt[2], cnt[3]};
  double acc = 0.0;
  for (int dir = 0; dir < 2; ++dir) {
    const int hi = dir ? n : no;
    for (int k = (dir ? no : 0) + t; k < hi; k += U * T) {
      bool in[U], ok[U], want[U], lead[U];
      int32_t c[U];
      uint32_t w[U], kc[U], Mo[U], Mt[U];
      double ld[U], t1[U], t2[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int at = k + u * T;
        ok[u] = at < hi;
        in[u] = dir == 1;
        const uint32_t key = ok[u] ? stage[at] : 0u;
        c[u] = (int32_t)(key & 0x7fffffffu);
        w[u] = ok[u] ? e.w(at) : 0u;
        const uint32_t sl = ok[u] ? tab.find(key) : 0u;
        lead[u] = tab.first[sl] == at;
        kc[u] = tab.sum[sl];
        want[u] = ok[u] && c[u] != r;
        ld[u] = ok[u] ? (dir ? a.ld_out : a.ld_in)[c[u]] : 0.0;
      }
      row_counts<DENSE, U>(a, r, in, c, want, Mo);
      row_counts<DENSE, U>(a, s, in, c, ok, Mt);
#pragma unroll
      for (int u = 0; u < U; ++u)
        entry_terms(a.xlx, ok[u], in[u], c[u], w[u], lead[u], kc[u], Mo[u], Mt[u], ld[u], r, s,
                    rw.niS, t1[u], t2[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        acc -= t1[u];
        acc -= t2[u];
      }
    }
  }
  if (t < 32) {
    const RowChange m = row_change(q, rw, cnt[4], cnt[5]);
    acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, lane);
  }
  const double d = grp.sum(acc);
  if (t == 0) write_result(a, GIVEN, i, r, s, d);
  __syncthreads();  // the CTA's next vertex reuses the shared memory
}

// A hub, more than kHubEntries entries, on a cluster of eight CTAs.  The sum
// it must give is that of 256 threads that take the entries of a direction
// strided by 256, each subtracting its entries' terms in the order of P hash
// classes of blocks (P = entries / 2048; the order of a table that holds one
// class at a time), then of the index, summed by warps.  CTA q does warp q's
// part, eight lanes a thread: they compute the terms of its next eight
// entries together and subtract them in order.  Every CTA fills its own
// table of all entries, one of both directions' blocks where they are sure to
// fit (n entries, or 2 B blocks, at most half the slots), else one per class.
// One CTA took 119 us for a hub of 5,400 entries at B = 600 and 233 at B =
// 20k, the longest chain of every batch of such a graph; a launch of this
// kernel over its three hubs a batch takes 26 us in the median.
constexpr int kHubCluster = 8;
constexpr int kHubList = 64;  // a thread's entries in order, up to 256 * kHubList entries
constexpr size_t kHubSmem = (3 * kHashSlots + 32 * kHubList) * sizeof(int32_t);
static_assert(kHeavyThreads == 32 * kHubCluster, "a virtual warp per CTA");

template <bool GIVEN, bool DENSE>
__device__ void hub_vertex(const NodalArgs& a, int i, int& parity) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int T = kHeavyThreads, G = 8;
  extern __shared__ unsigned long long hsm[];
  __shared__ unsigned long long wsum[T / 32];
  __shared__ double accs[32], red[2][kHubCluster];
  __shared__ uint32_t cnt[6];
  __shared__ int s_at, overflow;
  const int t = threadIdx.x, lane = t & 31, rank = (int)cl.block_rank();
  const int v = GIVEN ? a.verts[i] : a.lo + i;
  const HeavyEntries e(a, v);
  const int n = e.n, no = e.no;
  const bool fits = n <= kHashSlots / 2 || 2LL * a.B <= kHashSlots / 2;
  int slots = 512;
  while (slots < kHashSlots && (!fits || slots < 2 * min(n, 2 * a.B))) slots <<= 1;
  const HeavyTab tab{(int32_t*)hsm, (uint32_t*)hsm + kHashSlots, (int32_t*)hsm + 2 * kHashSlots,
                     slots};
  int32_t* const list = (int32_t*)hsm + 3 * kHashSlots;  // of each virtual thread
  const int r = a.part[v];
  tab.clear();
  if (t < 6) cnt[t] = 0u;
  if (t == 0) overflow = 0;
  __syncthreads();
  const int s = heavy_proposal<GIVEN>(a, i, v, e, wsum, &s_at, [&](int k) { return e.key(k); });
  if (r == s) {  // the same in every thread of the cluster
    if (rank == 0 && t == 0) write_result(a, GIVEN, i, r, s, 0.0);
    __syncthreads();
    return;
  }
#pragma unroll 4
  for (int k = t; k < n; k += T) {
    const uint32_t key = e.key(k), w = e.w(k);
    add_rs(cnt, k >= no, (int)(key & 0x7fffffffu), r, s, w);
    if (fits && !tab.add(key, w, k)) overflow = 1;
  }
  __syncthreads();
  const RsWeights rw{cnt[0], cnt[1], cnt[2], cnt[3]};
  const int vt = t >> 3, h = t & (G - 1), hb = lane & 24;  // virtual thread of the warp, helper
  const int first = 32 * rank + vt;
  double acc = 0.0;
  for (int dir = 0; dir < 2; ++dir) {
    const int lo = dir ? no : 0, hi = dir ? n : no;
    const uint32_t P = (uint32_t)((hi - lo + kHashSlots / 4 - 1) / (kHashSlots / 4));
    const int len = hi - lo > first ? (hi - lo - first + T - 1) / T : 0;
    const bool listed = hi - lo <= T * kHubList;
    int32_t* const mine = list + vt * kHubList;
    if (listed && P > 1) {
      // the thread's entries by class, then index
      int at = 0;
      for (uint32_t pass = 0; pass < P; ++pass)
        for (int j0 = 0; j0 < kHubList; j0 += G) {
          const int j = j0 + h;
          const int k = lo + first + j * T;
          const bool m = j < len && hclass((int32_t)(e.key(k) & 0x7fffffffu), P) == pass;
          const unsigned mm = __ballot_sync(kFull, m) >> hb & 0xffu;
          if (m) mine[at + __popc(mm & ((1u << h) - 1u))] = k;
          at += __popc(mm);
        }
    } else if (listed) {
      for (int j = h; j < len; j += G) mine[j] = lo + first + j * T;
    }
    __syncwarp();
    // one sweep over the list, or (a class's own table, or no list) one per
    // class that leaves out the other classes' entries
    const uint32_t sweeps = fits && listed ? (P ? 1 : 0) : P;
    for (uint32_t pass = 0; pass < sweeps; ++pass) {
      if (!fits) {
        __syncthreads();
        tab.clear();
        __syncthreads();
#pragma unroll 4
        for (int k = lo + t; k < hi; k += T) {
          const uint32_t key = e.key(k);
          if (hclass((int32_t)(key & 0x7fffffffu), P) == pass && !tab.add(key, e.w(k), k))
            overflow = 1;
        }
        __syncthreads();
      }
      const int most = (hi - lo + T - 1) / T;  // of any virtual thread: uniform
      for (int j0 = 0; j0 < most; j0 += G) {
        const int j = j0 + h;
        const int k = j >= len ? lo : listed ? mine[j] : lo + first + j * T;
        const uint32_t key = j < len ? e.key(k) : 0u;
        const int32_t c = (int32_t)(key & 0x7fffffffu);
        const bool in = dir == 1;
        const bool ok = j < len && (sweeps == 1 || hclass(c, P) == pass);
        const uint32_t w = ok ? e.w(k) : 0u;
        const uint32_t sl = ok ? tab.find(key) : 0u;
        const bool want = ok && c != r;
        const double ld = ok ? (in ? a.ld_out : a.ld_in)[c] : 0.0;
        uint32_t Mo, Mt;
        row_counts<DENSE, 1>(a, r, &in, &c, &want, &Mo);
        row_counts<DENSE, 1>(a, s, &in, &c, &ok, &Mt);
        double t1, t2;
        entry_terms(a.xlx, ok, in, c, w, tab.first[sl] == k, tab.sum[sl], Mo, Mt, ld, r, s,
                    rw.niS, t1, t2);
#pragma unroll
        for (int u = 0; u < G; ++u) {
          acc -= __shfl_sync(kFull, t1, hb + u);
          acc -= __shfl_sync(kFull, t2, hb + u);
        }
      }
    }
    __syncwarp();
  }
  if (h == 0) accs[vt] = acc;
  __syncthreads();
  if (t < 32) {
    acc = accs[lane];
    if (rank == 0) {
      const Corner q = load_corner<DENSE>(a, v, r, s, lane);
      const RowChange m = row_change(q, rw, cnt[4], cnt[5]);
      acc += corner_term<true, true>(a.xlx, q, rw, m.m4, m.m5, m.m6, m.m7, lane);
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      cl.map_shared_rank(&red[0][0], 0)[parity * kHubCluster + rank] = acc;
      if (overflow) atomicAdd(a.err, 1);
    }
  }
  cl.sync();
  if (rank == 0 && t == 0) {
    double d = 0.0;
    for (int q = 0; q < kHubCluster; ++q) d += red[parity][q];
    write_result(a, GIVEN, i, r, s, d);
  }
  // the next hub's sums go to the other half: it ends with a cluster barrier
  // that this one's reader reaches first
  parity ^= 1;
  __syncthreads();
}

// Heavy vertices but the hubs: one CTA each.
template <bool GIVEN, bool DENSE, bool GEN>
struct NodalHeavyBody {
  using Args = NodalArgs;
  static constexpr int kThreads = kHeavyThreads, kMinBlocks = 2;
  static constexpr size_t kSmem = kHeavySmem;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    __shared__ double red[kHeavyThreads / 32];
    const Group<kHeavyThreads> grp{red};
    for (int h = a.nhub + vb; h < a.nheavy; h += vg)
      heavy_vertex<GIVEN, DENSE>(a, a.heavy[h], grp);
  }
};

// Hubs: one cluster each.
template <bool GIVEN, bool DENSE>
struct NodalHubBody {
  using Args = NodalArgs;
  static constexpr int kThreads = kHeavyThreads, kMinBlocks = 1, kCluster = kHubCluster;
  static constexpr size_t kSmem = kHubSmem;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;  // the same in every thread of the cluster
    // every CTA of the cluster has started before one stores into another's
    // shared memory
    cooperative_groups::this_cluster().sync();
    int parity = 0;
    for (int h = vb / kHubCluster; h < a.nhub; h += vg / kHubCluster)
      hub_vertex<GIVEN, DENSE>(a, a.heavy[h], parity);
  }
};

// General mode: every heavy vertex on a CTA.
template <bool GIVEN, bool DENSE>
struct NodalHeavyBody<GIVEN, DENSE, true> {
  using Args = NodalArgs;
  static constexpr int kThreads = kHeavyThreads, kMinBlocks = 2;
  static constexpr size_t kSmem = 3 * kHashSlots * sizeof(int32_t);
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    extern __shared__ unsigned long long hsm[];
    __shared__ double red[kHeavyThreads / 32];
    __shared__ int flag, sh_v, sh_s;
    __shared__ uint32_t sh_u2;
    Group<kHeavyThreads> grp{red};
    HashTab ht{(int32_t*)hsm, (uint32_t*)hsm + kHashSlots, (int32_t*)hsm + 2 * kHashSlots};
    for (int h = vb; h < a.nheavy; h += vg) {
      const int i = a.heavy[h];
      if (threadIdx.x < 32) {
        int v, s;
        uint32_t u2;
        item<GIVEN>(a, i, threadIdx.x, v, s, u2);
        if (threadIdx.x == 0) {
          sh_v = v;
          sh_s = s;
          sh_u2 = u2;
        }
      }
      __syncthreads();
      const int v = sh_v, s = sh_s;
      const int r = a.part[v];
      double d = 0.0, lh = 0.0;
      if (r != s) {
        d = delta_hashed_gen<DENSE, kHeavyThreads>(a, v, r, s, ht, &flag, grp, lh);
        if (threadIdx.x == 0 && d != d) atomicAdd(a.err, 1);
      }
      if (threadIdx.x == 0) write_result_gen(a, GIVEN, i, r, s, d, lh, sh_u2);
      __syncthreads();
    }
  }
};

// Applies the batch's labels and sums its recorded dS.  Each CTA sums a fixed
// slice (one vertex a thread) in a fixed order into its own partial; the
// last CTA to finish (a ticket, no waiting) adds the partials with one warp
// in a fixed order, so the result does not depend on scheduling.  In dense
// mode the CTAs also refresh the log2 of the block degrees that
// dense_update changed, and the virtual blocks past `ncommit` (if any) make
// the next batch's per-block draws: they read only M, its chunk sums and the
// block degrees, all final once dense_update has run, so the draws need no
// launch of their own.
constexpr int kCommitThreads = 256;

struct CommitArgs {
  int32_t* part;
  const int32_t* newlab;
  const double* rec;
  double* slot_sum;
  long long* slot_acc;
  const uint32_t *d_out, *d_in;  // dense mode: refresh ld_out / ld_in
  double *ld_out, *ld_in;
  double* part_sum;
  long long* part_cnt;
  unsigned* ticket;
  const int32_t* ctl;  // sweep control: gate, and slots advance ctl[0] * slot_mul
  // dense mode, draws for the next batch (RNG sequence draw_seq + ctl[0] *
  // draw_seq_mul) by the virtual blocks past ncommit
  const uint32_t *Md, *MTd, *Sd;
  int32_t* nbr_s;
  uint64_t seed;
  uint32_t draw_seq, draw_seq_mul;
  int32_t lo, count, B, slot_mul;
  int32_t ncommit, pad;
  int32_t* mark;  // the sweep's last batch: the job's sweep control, handed on (add_commit)
};

struct CommitBody {
  using Args = CommitArgs;
  static constexpr int kThreads = kCommitThreads, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (a.mark && vb == 0 && tid == 0) {
      a.mark[2] = a.mark[0] + 1;
      a.mark[3] = a.mark[1];
    }
    if (ctl_stopped(a.ctl)) return;
    if (vb >= a.ncommit) {
      const uint32_t seq = a.draw_seq + ctl_itr(a.ctl) * a.draw_seq_mul;
      const int nw = ((vg - a.ncommit) * kCommitThreads) >> 5;
      for (int b = ((vb - a.ncommit) * kCommitThreads + tid) >> 5; b < a.B; b += nw)
        dense_block_draw(a.Md, a.MTd, a.Sd, a.d_out, a.d_in, a.B, a.seed, seq, b, lane,
                         a.nbr_s);
      return;
    }
    const int nc = a.ncommit;
    __shared__ double sh[kCommitThreads / 32];
    __shared__ long long shc[kCommitThreads / 32];
    __shared__ bool last;
    double s = 0.0;
    long long c = 0;
    for (int i = vb * kCommitThreads + tid; i < a.count; i += nc * kCommitThreads) {
      const int32_t nl = a.newlab[i];
      const int32_t old = a.part[a.lo + i];
      const double x = a.rec[i];
      if (old != nl) {
        a.part[a.lo + i] = nl;
        ++c;
      }
      s += x;
    }
    if (a.ld_out)
      for (int b = vb * kCommitThreads + tid; b < a.B; b += nc * kCommitThreads) {
        a.ld_out[b] = log2((double)a.d_out[b]);
        a.ld_in[b] = log2((double)a.d_in[b]);
      }
    s = warp_sum(s);
    c = warp_sum_ll(c);
    if (lane == 0) {
      sh[wid] = s;
      shc[wid] = c;
    }
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      long long n = 0;
      for (int k = 0; k < kCommitThreads / 32; ++k) {
        t += sh[k];
        n += shc[k];
      }
      a.part_sum[vb] = t;
      a.part_cnt[vb] = n;
      __threadfence();
      last = atomicAdd(a.ticket, 1u) == (unsigned)nc - 1u;
    }
    __syncthreads();
    if (last && wid == 0) {
      __threadfence();
      double t = 0.0;
      long long n = 0;
      for (int k = lane; k < nc; k += 32) {
        t += ((volatile double*)a.part_sum)[k];
        n += ((volatile long long*)a.part_cnt)[k];
      }
      t = warp_sum(t);
      n = warp_sum_ll(n);
      if (lane == 0) {
        const int k = (int)ctl_itr(a.ctl) * a.slot_mul;
        a.slot_sum[k] += t;
        a.slot_acc[k] += n;
        *a.ticket = 0u;
      }
    }
  }
};

// CTAs of one commit: a function of the batch size only.
int32_t vg_commit(int32_t count) {
  return std::max(1, std::min(kCommitCtas, ceil_div(count, kCommitThreads)));
}

CommitArgs commit_args(int32_t* part, int32_t lo, int32_t count, const int32_t* newlab,
                       const double* rec, double* slot_sum, long long* slot_acc,
                       const DevBM* dense_m, int32_t B, const CommitScratch& cs) {
  CommitArgs a{};
  a.part = part;
  a.newlab = newlab;
  a.rec = rec;
  a.slot_sum = slot_sum;
  a.slot_acc = slot_acc;
  if (dense_m) {
    a.d_out = dense_m->d_out;
    a.d_in = dense_m->d_in;
    a.ld_out = dense_m->ld_out;
    a.ld_in = dense_m->ld_in;
    a.B = B;
  }
  a.part_sum = cs.part_sum;
  a.part_cnt = cs.part_cnt;
  a.ticket = cs.ticket;
  a.lo = lo;
  a.count = count;
  a.ncommit = vg_commit(count);
  return a;
}

// Vertices of kGroupEntries to kWideEntries entries go to wide_vertex where a
// batch has more than kWideMin of them, the CTAs that the GPU holds at once.
// Dense sweeps of four batches of vertices of 80 entries, B = 1000, a CTA each /
// this way: 1000 a batch 0.096 / 0.117 ms, 2000 0.123 / 0.120, 4000 0.170 /
// 0.125, 16000 0.452 / 0.267.
constexpr int32_t kWideMin = 8 * 148;

NodalArgs make_args(const DevGraph& g, const int32_t* part, const DevBM& m, int32_t B,
                    const NodalAux& aux, const ScoreMode& md) {
  NodalArgs a{};
  a.exact = md.exact;
  a.mh = md.mh;
  a.beta = md.beta;
  a.xlx = m.xlx;
  a.optr = g.optr; a.oidx = g.oidx; a.iptr = g.iptr; a.iidx = g.iidx;
  a.ow = g.ow; a.iw = g.iw; a.kdo = g.kdo; a.kdi = g.kdi;
  a.part = part;
  a.bop = m.optr; a.boe = m.oend; a.boc = m.ocol;
  a.bip = m.iptr; a.bie = m.iend; a.bic = m.icol;
  a.bon = m.ocnt; a.bin = m.icnt; a.d_out = m.d_out; a.d_in = m.d_in;
  a.Md = m.Md; a.MTd = m.MTd;
  a.ld_out = m.ld_out; a.ld_in = m.ld_in;
  a.nbr_s = m.nbr_s;
  a.B = B;
  a.unit = g.unit;
  a.heavy = aux.heavy;
  a.nheavy = aux.nheavy;
  a.nhub = aux.nhub;
  a.small = aux.small;
  a.nsmall = aux.nsmall;
  a.mid = aux.mid;
  a.nmid = aux.nmid;
  a.nwide = !md.general() && aux.nlarge - aux.nlong > kWideMin ? aux.nlarge - aux.nlong : 0;
  a.nlarge = aux.nlarge - a.nwide;
  a.nmid64 = aux.nmid64;
  a.err = aux.err;
  return a;
}

// CTAs of the warp kernel.
int32_t nodal_ctas(const NodalArgs& a) {
  return NodalItems(a).ctas();
}

template <bool GIVEN, bool DENSE, bool GEN>
void launch_pair(const NodalArgs& a, const NodalAux& aux, cudaStream_t st) {
  const int nhub = GEN ? 0 : a.nhub;
  if (a.nheavy > 0) {
    // heavy vertices on the side stream, next to the warp kernel
    cudaEventRecord(aux.fork, st);
    cudaStreamWaitEvent(aux.side, aux.fork, 0);
    if (nhub > 0)
      launch_single<NodalHubBody<GIVEN, DENSE>>(a, kHubCluster * std::min(nhub, 18), aux.side);
    launch_single<NodalHeavyBody<GIVEN, DENSE, GEN>>(a, std::min(a.nheavy - nhub, 4 * 148),
                                                     aux.side);
    cudaEventRecord(aux.join, aux.side);
  }
  launch_single<NodalBody<GIVEN, DENSE, GEN>>(a, nodal_ctas(a), st);
  if (a.nheavy > 0) cudaStreamWaitEvent(st, aux.join, 0);
}

template <bool GIVEN, bool DENSE>
void launch_mode(const NodalArgs& a, const NodalAux& aux, cudaStream_t st, bool gen) {
  if (gen) launch_pair<GIVEN, DENSE, true>(a, aux, st);
  else launch_pair<GIVEN, DENSE, false>(a, aux, st);
}

// indexed by ScoreMode::slot(dense)
const MultiKernel kmNodal[4] = {
    multi_kernel_desc<NodalBody<false, false, false>>("nodal_csr"),
    multi_kernel_desc<NodalBody<false, true, false>>("nodal_dense"),
    multi_kernel_desc<NodalBody<false, false, true>>("nodal_gen_csr"),
    multi_kernel_desc<NodalBody<false, true, true>>("nodal_gen_dense")};
const MultiKernel kmNodalHeavy[4] = {
    multi_kernel_desc<NodalHeavyBody<false, false, false>>("nodal_heavy_csr"),
    multi_kernel_desc<NodalHeavyBody<false, true, false>>("nodal_heavy_dense"),
    multi_kernel_desc<NodalHeavyBody<false, false, true>>("nodal_heavy_gen_csr"),
    multi_kernel_desc<NodalHeavyBody<false, true, true>>("nodal_heavy_gen_dense")};

const MultiKernel kmNodalHub[2] = {multi_kernel_desc<NodalHubBody<false, false>>("nodal_hub_csr"),
                                   multi_kernel_desc<NodalHubBody<false, true>>("nodal_hub_dense")};

const MultiKernel kmCommit = multi_kernel_desc<CommitBody>("commit");

}  // namespace

template <class... Bodies>
cudaError_t allow_smem_all() {
  cudaError_t e = cudaSuccess;
  for (cudaError_t x : {allow_smem<Bodies>()...})
    if (x != cudaSuccess) e = x;
  return e;
}

cudaError_t init_nodal_attributes() {
  const cudaError_t e =
      allow_smem_all<NodalHeavyBody<false, false, true>, NodalHeavyBody<false, true, true>,
                     NodalHeavyBody<true, false, true>, NodalHeavyBody<true, true, true>>();
  const cudaError_t e2 =
      allow_smem_all<NodalHubBody<false, false>, NodalHubBody<false, true>,
                     NodalHubBody<true, false>, NodalHubBody<true, true>>();
  return e != cudaSuccess ? e : e2;
}

int nodal_heavy_threshold() { return kWarpList; }

void nodal_batch_sample(const DevGraph& g, const int32_t* part, const DevBM& m, int32_t B,
                        bool dense, uint64_t seed, uint32_t seq, int32_t lo, int32_t count,
                        int32_t* newlab, double* rec, int32_t* props, const NodalAux& aux,
                        cudaStream_t st, const ScoreMode& md) {
  NodalArgs a = make_args(g, part, m, B, aux, md);
  a.seed = seed;
  a.seq = seq;
  a.lo = lo;
  a.count = count;
  a.newlab = newlab;
  a.rec = rec;
  a.props_out = props;
  if (count <= 0) return;
  if (dense) launch_mode<false, true>(a, aux, st, md.general());
  else launch_mode<false, false>(a, aux, st, md.general());
}

void nodal_delta_given(const DevGraph& g, const int32_t* part, const DevBM& m, int32_t B,
                       bool dense, int32_t nv, const int32_t* verts, const int32_t* props,
                       double* dS, const NodalAux& aux, cudaStream_t st, const ScoreMode& md,
                       double* logH) {
  NodalArgs a = make_args(g, part, m, B, aux, md);
  a.count = nv;
  a.verts = verts;
  a.props_in = props;
  a.dS_raw = dS;
  a.logH_raw = logH;
  if (nv <= 0) return;
  if (dense) launch_mode<true, true>(a, aux, st, md.general());
  else launch_mode<true, false>(a, aux, st, md.general());
}

void nodal_commit(int32_t* part, int32_t lo, int32_t count, const int32_t* newlab,
                  const double* rec, double* slot_sum, long long* slot_acc, const DevBM* dense_m,
                  int32_t B, const CommitScratch& cs, cudaStream_t st) {
  launch_single<CommitBody>(
      commit_args(part, lo, count, newlab, rec, slot_sum, slot_acc, dense_m, B, cs),
      vg_commit(count), st);
}

void add_nodal(Slot& warp, Slot& heavy, Slot& hub, bool dense, const ScoreMode& md, const DevGraph& g,
               const int32_t* part,
               const DevBM& m, int32_t B, uint64_t seed, uint32_t seq, int32_t lo, int32_t count,
               int32_t* newlab, double* rec, int32_t* props, const NodalAux& aux,
               const int32_t* ctl, uint32_t seq_mul) {
  if (count <= 0) return;
  NodalArgs a = make_args(g, part, m, B, aux, md);
  a.seed = seed;
  a.seq = seq;
  a.lo = lo;
  a.count = count;
  a.newlab = newlab;
  a.rec = rec;
  a.props_out = props;
  a.ctl = ctl;
  a.seq_mul = seq_mul;
  slot_push(slot_bind(warp, kmNodal[md.slot(dense)]), a, nodal_ctas(a));
  const int32_t nhub = md.general() ? 0 : aux.nhub;
  slot_push(slot_bind(heavy, kmNodalHeavy[md.slot(dense)]), a, aux.nheavy - nhub);
  if (nhub > 0) slot_push(slot_bind(hub, kmNodalHub[dense ? 1 : 0]), a, kHubCluster * nhub);
}

void add_commit(Slot& s, int32_t* part, int32_t lo, int32_t count, const int32_t* newlab,
                const double* rec, double* slot_sum, long long* slot_acc, const DevBM* dense_m,
                int32_t B, const CommitScratch& cs, int32_t* ctl, int32_t slot_mul, bool mark,
                bool draw_next, uint64_t seed, uint32_t draw_seq, uint32_t draw_seq_mul) {
  CommitArgs a = commit_args(part, lo, count, newlab, rec, slot_sum, slot_acc, dense_m, B, cs);
  a.ctl = ctl;
  a.slot_mul = slot_mul;
  if (mark) a.mark = ctl;
  int32_t vg = a.ncommit;
  if (draw_next && dense_m) {
    a.Md = dense_m->Md;
    a.MTd = dense_m->MTd;
    a.Sd = dense_m->Sd;
    a.nbr_s = dense_m->nbr_s;
    a.seed = seed;
    a.draw_seq = draw_seq;
    a.draw_seq_mul = draw_seq_mul;
    // a warp per block, as the block-terms kernel
    vg += std::max(1, std::min(8192, ceil_div((long long)B * 32, kCommitThreads)));
  }
  slot_push(slot_bind(s, kmCommit), a, vg);
}

}  // namespace sbp
