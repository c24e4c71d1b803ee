// Blockmodel rebuild, per-block terms and the MDL sum.
//
// GSAP rebuilds M after every merge step and every nodal batch with
// thrust::sort_by_key over vertices, four thrust scans, a scatter of
// neighbour blocks, bb_segsort over block segments, six memsets, two
// remove_if compactions with a host read-back and mgpu::segreduce
// (calculate_new_csr, partition.hpp:707-849; about 30 launches and ten hidden
// allocations or synchronisations per call).  Here it is six launches with no
// host round trip, both directions (out rows / in rows) in each:
//
//   count    per vertex: entries of its row segment, slot inside the segment
//   scan     segment offsets, where the rows stay
//   scatter  per graph entry: (neighbour block, weight) into its segment
//   tile     short segments: a thread per entry, ranked by comparison
//   rank     longer ones: a warp each, ranked through a bitmap of columns
//   big      the longest: a CTA or a cluster of eight CTAs each
//
// The result is exact integer work and identical to the oracle's builder.
#include "common.cuh"
#include "kernels.h"
#include "multi.cuh"
#include "dense.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

namespace sbp {

thread_local long long g_launches = 0;

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

// Exclusive scan across the CTA (any blockDim multiple of 32 up to 1024).
// `sh` needs 33 ints.  Returns the exclusive prefix; *total gets the sum.
__device__ __forceinline__ int cta_excl_scan(int x, int* sh, int* total) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sh[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int v = lane < nw ? sh[lane] : 0;
    int vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(kFull, vi, o);
      if (lane >= o) vi += y;
    }
    if (lane < nw) sh[lane] = vi - v;
    if (lane == 31) sh[32] = vi;
  }
  __syncthreads();
  int res = incl - x + sh[wid];
  *total = sh[32];
  __syncthreads();
  return res;
}

// Scan of one array in three steps when it spans more than one CTA's tiles:
// per-tile sums, a one-CTA scan of those sums, then each tile applies its
// offset.  Short arrays take the one-CTA scan directly.
struct ScanArgs {
  const int32_t* in;
  int32_t* out;
  int32_t* tile;  // tile sums (tile body), offsets (apply body)
  const int32_t* ctl;
  int32_t n, pad;
};

struct ScanTileBody {
  using Args = ScanArgs;
  static constexpr int kThreads = kScanThreads, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    if (ctl_stopped(a.ctl)) return;
    __shared__ int sh[33];
    int base = vb * kScanTile + threadIdx.x * kScanItems;
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (base + k < a.n) s += a.in[base + k];
    int tot;
    cta_excl_scan(s, sh, &tot);
    if (threadIdx.x == 0) a.tile[vb] = tot;
  }
};

// Exclusive scan of `n` values (in place allowed), one CTA, tile by tile with
// a carry; out[n] = total.
struct ScanSingleBody {
  using Args = ScanArgs;
  static constexpr int kThreads = kScanThreads, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int, int) {
    if (ctl_stopped(a.ctl)) return;
    __shared__ int sh[33];
    int carry = 0;
    for (int t0 = 0; t0 < a.n; t0 += kScanTile) {
      int base = t0 + threadIdx.x * kScanItems;
      int v[kScanItems];
      int s = 0;
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < a.n ? a.in[base + k] : 0;
        s += v[k];
      }
      int tot;
      int pre = cta_excl_scan(s, sh, &tot) + carry;
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        if (base + k < a.n) a.out[base + k] = pre;
        pre += v[k];
      }
      carry += tot;
    }
    if (threadIdx.x == 0) a.out[a.n] = carry;
  }
};

struct ScanApplyBody {
  using Args = ScanArgs;
  static constexpr int kThreads = kScanThreads, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    __shared__ int sh[33];
    int base = vb * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = base + k < a.n ? a.in[base + k] : 0;
      s += v[k];
    }
    int tot;
    int pre = cta_excl_scan(s, sh, &tot) + a.tile[vb];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < a.n) a.out[base + k] = pre;
      pre += v[k];
    }
    if (vb == vg - 1 && threadIdx.x == blockDim.x - 1) a.out[a.n] = pre;
  }
};

constexpr int kScanSingleMax = 8 * kScanTile;

// ------------------------------------------------------------ rebuild ------
// M's rows are left at their segments' offsets: row b occupies
// [ptr[b], end[b]) of the segment [ptr[b], ptr[b+1]) of the entries its
// edges made, with unused entries after it.  A compact CSR needs the rows'
// unique counts before their offsets, so it costs another scan and a copy of
// every entry (200k HH, E = 2M: 80 us of a 430 us rebuild); nothing that
// reads M needs its rows back to back.
struct RbSide {
  const int32_t* gptr;
  const int32_t* gidx;
  const uint32_t* gw;
  const int32_t* gsrc;
  int32_t* cnt;
  int32_t* vofs;
  int32_t* tcol;
  uint32_t* tw;
  int32_t *mid, *big, *giant;  // longer segments by kernel path
  int32_t* nlist;              // their counts
  int32_t* bptr;
  int32_t* bend;
  int32_t* bcol;
  uint32_t* bcnt;
  uint32_t* bcum;
  uint32_t* bdeg;
  double* bld;
};

struct RbArgs {
  RbSide s[2];
  const int32_t* part;
  const int32_t* ctl;
  const double* xlx;
  int32_t* nnz;
  int32_t N, E, B;
  int32_t tile_cap;   // longest segment ranked by comparison (RbTileBody)
  int32_t warp_max;   // longest segment ranked by a warp (RbRankBody)
  int32_t tile_rows;  // rows of a tile
  int32_t unit;       // every weight is 1: tw is neither written nor read
  int32_t pad;
};

// The rebuild bodies work on both directions: virtual block vb serves
// direction vb & 1 with the direction's own virtual block vb >> 1.

// Per vertex: its entries form one run inside its block's segment.
struct RbCountBody {
  using Args = RbArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
  if (ctl_stopped(a.ctl)) return;
  const RbSide& d = a.s[vb & 1];
  int v = (vb >> 1) * blockDim.x + threadIdx.x;
  const bool live = v < a.N;
  const unsigned active = __ballot_sync(kFull, live);
  if (!live) return;
  int b = a.part[v];
  int len = d.gptr[v + 1] - d.gptr[v];
  // warp-aggregated: lanes with the same block reserve one range together
  unsigned peers = __match_any_sync(active, b);
  int lane = threadIdx.x & 31;
  int leader = __ffs(peers) - 1;
  int pre = 0, tot = 0;
  for (unsigned m = peers; m; m &= m - 1) {
    int j = __ffs(m) - 1;
    int x = __shfl_sync(peers, len, j);
    tot += x;
    if (j < lane) pre += x;
  }
  int base = 0;
  if (lane == leader) base = atomicAdd(d.cnt + b, tot);
  base = __shfl_sync(peers, base, leader);
  d.vofs[v] = base + pre;
  }
};

// Per graph entry: (block of the neighbour, weight) into the owner's run.
struct RbScatterBody {
  using Args = RbArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    if (ctl_stopped(a.ctl)) return;
    const RbSide& d = a.s[vb & 1];
    int j = (vb >> 1) * blockDim.x + threadIdx.x;
    if (j >= a.E) return;
    int v = __ldg(d.gsrc + j);
    int b = a.part[v];
    int pos = d.bptr[b] + d.vofs[v] + (j - __ldg(d.gptr + v));
    d.tcol[pos] = a.part[__ldg(d.gidx + j)];
    if (!a.unit) d.tw[pos] = __ldg(d.gw + j);
  }
};

// End, degree and its log2 of row b with u unique entries and weight sum deg.
__device__ __forceinline__ void row_done(const RbArgs& a, const RbSide& d, int b, int base, int u,
                                         uint32_t deg) {
  d.bend[b] = base + u;
  d.bdeg[b] = deg;
  d.bld[b] = l2x(a.xlx, deg);
}

constexpr int kBigCap = 12288;  // longest segment a CTA takes; longer ones go to a cluster

// Short segments: a CTA takes tile_rows consecutive rows and gives every
// entry a thread, which counts its segment's entries before it in (column,
// index) order, its place in the sorted segment; eight lanes a row then walk
// the sorted entries and write each run of a column once.  What bounds it is
// the comparisons, so column and index share a word (up to kTileBlocks
// blocks) and are compared four at a time: 86 us a rebuild of the 200k HH
// graph comparing columns and weights one by one, 72 this way, 141 for a warp
// per segment (a match over its lanes, or a bitonic sort).  Longer segments
// are listed for the kernels below.
constexpr int kTileEntries = 2048, kTileMaxCap = 128;
// (column, index) in a word: 7 bits of index, and no such word is the padding
constexpr int kTileBlocks = (1 << 25) - 1;
struct RbTileBody {
  using Args = RbArgs;
  static constexpr int kThreads = 256, kMinBlocks = 6;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    if (ctl_stopped(a.ctl)) return;
    // a segment starts at a multiple of four entries, padded with ~0
    __shared__ __align__(16) uint32_t key[kTileEntries];
    __shared__ uint32_t w[kTileEntries];
    __shared__ uint8_t owner[kTileEntries], sorted[kTileEntries];  // row; index by place
    __shared__ int off[kThreads + 1], src[kThreads];
    __shared__ uint8_t slen[kThreads];
    __shared__ int sh[33];
    __shared__ int s_nnz;
    const RbSide& d = a.s[vb & 1];
    const int tid = threadIdx.x, lane = tid & 31;
    const int b0 = (vb >> 1) * a.tile_rows, nr = min(a.tile_rows, a.B - b0);
    const bool packed = a.B <= kTileBlocks;
    int len = 0;
    if (tid < nr) {
      const int b = b0 + tid, base = d.bptr[b];
      len = d.bptr[b + 1] - base;
      src[tid] = base;
      if (len > a.tile_cap) {
        const int k = len <= a.warp_max ? 0 : len <= kBigCap ? 1 : 2;
        (k == 0 ? d.mid : k == 1 ? d.big : d.giant)[atomicAdd(d.nlist + k, 1)] = b;
        len = 0;
      } else if (len == 0) {
        row_done(a, d, b, base, 0, 0u);
      }
    }
    slen[tid] = (uint8_t)len;
    if (tid == 0) s_nnz = 0;
    const int plen = (len + 3) & ~3;
    int total;
    const int at = cta_excl_scan(plen, sh, &total);
    off[tid] = at;
    if (tid == 0) off[kThreads] = total;
    __syncthreads();
    // rounds of rows whose offsets lie in a window, so that their entries fit;
    // the next round's window starts at its first row, so that a round writes
    // all the entries it ranks
    const int win = kTileEntries - kTileMaxCap;
    const int g = tid >> 3, gl = tid & 7;
    int nnz = 0;
    for (int q0 = 0, end; q0 < total; q0 += end) {
      for (int r = g; r < nr; r += kThreads / 8) {
        const int o = off[r] - q0, n = slen[r];
        if (n == 0 || o < 0 || o >= win) continue;
        for (int i = gl; i < ((n + 3) & ~3); i += 8) {
          uint32_t x = 0xffffffffu;
          if (i < n) {
            x = (uint32_t)d.tcol[src[r] + i];
            if (packed) x = x << 7 | (uint32_t)i;
            if (!a.unit) w[o + i] = d.tw[src[r] + i];
          }
          key[o + i] = x;
          owner[o + i] = (uint8_t)r;
        }
      }
      __syncthreads();
      // the round's entries end where the next round's first row starts
      end = total - q0;
      if (end > win) {
        const bool mine = tid < nr && len > 0 && at - q0 >= 0 && at - q0 < win;
        end = mine ? at - q0 + plen : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) end = max(end, __shfl_xor_sync(kFull, end, o));
        if (lane == 0) sh[tid >> 5] = end;
        __syncthreads();
        end = 0;
        for (int i = 0; i < kThreads / 32; ++i) end = max(end, sh[i]);
      }
      for (int e = tid; e < end; e += kThreads) {
        const uint32_t k = key[e];
        if (k == 0xffffffffu) continue;
        const int r = owner[e], s0 = off[r] - q0, s1 = s0 + ((slen[r] + 3) & ~3);
        int lt = 0;
        if (packed) {
          for (int j = s0; j < s1; j += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(key + j);
            lt += (x.x < k ? 1 : 0) + (x.y < k ? 1 : 0) + (x.z < k ? 1 : 0) + (x.w < k ? 1 : 0);
          }
        } else {
          for (int j = s0; j < s1; ++j) lt += key[j] < k || (key[j] == k && j < e) ? 1 : 0;
        }
        sorted[s0 + lt] = (uint8_t)(e - s0);
      }
      __syncthreads();
      for (int r0 = 0; r0 < nr; r0 += kThreads / 8) {
        const int r = r0 + g;
        const int o = r < nr ? off[r] - q0 : -1, n = r < nr ? slen[r] : 0;
        const bool live = n > 0 && o >= 0 && o < win;
        const int steps = live ? (n + 7) >> 3 : 0;
        auto column = [&](int p) {
          const uint32_t x = key[o + sorted[o + p]];
          return packed ? x >> 7 : x;
        };
        int u = 0;
        uint32_t deg = 0u;  // the count so far
        const int most = __reduce_max_sync(kFull, steps);
        for (int i = 0; i < most; ++i) {
          const int p = 8 * i + gl;
          uint32_t c = 0u, x = 0u;
          if (live && p < n) {
            x = column(p);
            if (p == 0 || column(p - 1) != x) {  // the first of its column's run
              int q = p;
              do c += a.unit ? 1u : w[o + sorted[o + q]];
              while (++q < n && column(q) == x);
            }
          }
          const unsigned m = __ballot_sync(kFull, c != 0u) >> (lane & 24) & 0xffu;
          uint32_t incl = c;
#pragma unroll
          for (int z = 1; z < 8; z <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, incl, z, 8);
            if (gl >= z) incl += y;
          }
          if (c) {
            const int z = src[r] + u + __popc(m & ((1u << gl) - 1u));
            d.bcol[z] = (int32_t)x;
            d.bcnt[z] = c;
            d.bcum[z] = deg + incl;
          }
          deg += __shfl_sync(kFull, incl, 7, 8);
          u += __popc(m);
        }
        if (live && gl == 0) {
          row_done(a, d, b0 + r, src[r], u, deg);
          nnz += u;
        }
      }
      __syncthreads();
    }
    if (vb & 1) return;  // the two directions have the same entries
    if (nnz) atomicAdd(&s_nnz, nnz);
    __syncthreads();
    if (tid == 0 && s_nnz) atomicAdd(a.nnz, s_nnz);
  }
};

// Longer segments by a bitmap of their columns: a column's place among the
// distinct ones is the number of bits below it (the words before it, then
// its own word), so no sort is needed; its total is added at that place.
// Columns are taken in windows of the bitmap's size.  A warp's shared memory:
// a window's bitmap and running counts, and the totals.
constexpr int kRankMax = 1024;       // longest segment a warp takes
constexpr int kRankWords = 512;      // bitmap words of a window
constexpr int kRankWarps = 8;
constexpr size_t kRankWarpBytes = kRankWords * 6 + kRankMax * 4;
struct RbRankBody {
  using Args = RbArgs;
  static constexpr int kThreads = kRankWarps * 32, kMinBlocks = 1;
  static constexpr size_t kSmem = kRankWarps * kRankWarpBytes;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    extern __shared__ __align__(16) unsigned char rank_sm[];
    const RbSide& d = a.s[vb & 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t* cnt = (uint32_t*)(rank_sm + wid * kRankWarpBytes);
    uint32_t* bm = cnt + kRankMax;
    uint16_t* pre = (uint16_t*)(bm + kRankWords);
    const int nmid = d.nlist[0];
    int nnz = 0;
    for (int idx = (vb >> 1) * kRankWarps + wid; idx < nmid; idx += (vg >> 1) * kRankWarps) {
      const int b = d.mid[idx], base = d.bptr[b], n = d.bptr[b + 1] - base;
      for (int i = lane; i < n; i += 32) cnt[i] = 0u;
      int u = 0;
      for (int w0 = 0; w0 < a.B; w0 += 32 * kRankWords) {
        const int cols = min(32 * kRankWords, a.B - w0);
        for (int x = 4 * lane; x < kRankWords; x += 128)
          *reinterpret_cast<uint4*>(bm + x) = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
#pragma unroll 4
        for (int i = lane; i < n; i += 32) {
          const int c = d.tcol[base + i] - w0;
          if ((unsigned)c < (unsigned)cols) atomicOr(bm + (c >> 5), 1u << (c & 31));
        }
        __syncwarp();
        // each lane counts sixteen consecutive words (in an order of four
        // that spreads the lanes over the banks)
        constexpr int kPer = kRankWords / 32;
        int own[kPer / 4], local = 0;
#pragma unroll
        for (int k = 0; k < kPer / 4; ++k) {
          const int x = lane * kPer + 4 * ((k + (lane >> 1)) & (kPer / 4 - 1));
          const uint4 g = *reinterpret_cast<const uint4*>(bm + x);
          const int p0 = __popc(g.x), p1 = p0 + __popc(g.y), p2 = p1 + __popc(g.z);
          own[k] = p2 + __popc(g.w);
          // within the four, to be offset below
          *reinterpret_cast<ushort4*>(pre + x) = make_ushort4(0, p0, p1, p2);
          local += own[k];
        }
        const int incl = (int)warp_incl_scan_u((unsigned)local, lane);
        const int run = __shfl_sync(kFull, incl, 31);
        {
          // the four's places in ascending order of words
          int at[kPer / 4];
          int before = incl - local;
#pragma unroll
          for (int z = 0; z < kPer / 4; ++z) {
            const int k = (z - (lane >> 1)) & (kPer / 4 - 1);  // the one that holds words 4z
            int c = 0;
#pragma unroll
            for (int y = 0; y < kPer / 4; ++y) c = k == y ? own[y] : c;
            at[z] = before;
            before += c;
          }
#pragma unroll
          for (int z = 0; z < kPer / 4; ++z) {
            ushort4* q = reinterpret_cast<ushort4*>(pre + lane * kPer + 4 * z);
            ushort4 v = *q;
            v.x += at[z];
            v.y += at[z];
            v.z += at[z];
            v.w += at[z];
            *q = v;
          }
        }
        __syncwarp();
#pragma unroll 4
        for (int i = lane; i < n; i += 32) {
          const int c = d.tcol[base + i] - w0;
          if ((unsigned)c >= (unsigned)cols) continue;
          const int at = u + pre[c >> 5] + __popc(bm[c >> 5] & ((1u << (c & 31)) - 1u));
          atomicAdd(cnt + at, a.unit ? 1u : d.tw[base + i]);
          d.bcol[base + at] = c + w0;
        }
        u += run;
        __syncwarp();
      }
      uint32_t deg = 0u;
      for (int i0 = 0; i0 < u; i0 += 32) {
        const int i = i0 + lane;
        const uint32_t c = i < u ? cnt[i] : 0u;
        const uint32_t incl = warp_incl_scan_u(c, lane);
        if (i < u) {
          d.bcnt[base + i] = c;
          d.bcum[base + i] = deg + incl;
        }
        deg += __shfl_sync(kFull, incl, 31);
      }
      if (lane == 0) row_done(a, d, b, base, u, deg);
      nnz += u;
      __syncwarp();
    }
    if (!(vb & 1) && lane == 0 && nnz) atomicAdd(a.nnz, nnz);
  }
};

// The longest segments, the same way: up to kBigCap entries by a CTA, longer
// ones (a block that many merged into: 50k-500k entries of the 200k HH graph)
// by a cluster of eight CTAs, each with an eighth of the entries.  Each CTA
// marks its entries' columns, merges an eighth of the eight bitmaps through
// distributed shared memory and hands the merged words and their running
// counts to all; the totals are then added in place, or (few columns) in
// shared memory first.  One CTA for such a segment took 157 us of every
// rebuild of the 200k HH graph, and up to 1.1 ms; the cluster 17 us (at most
// 48).
// Where many segments are that long the clusters take their turns, and a CTA
// each is faster as long as none of them takes much more than its share of the
// whole; a CTA can where the columns' totals fit its shared memory (at most
// kBigCap blocks).  A rebuild of 200k vertices of degree 10 in B even blocks,
// clusters only with all totals in place / now: B = 150 212 / 115 us, B = 71
// 174 / 106, B = 50 127 / 99 (share 768 / 1024), B = 32 146 / 106, B = 2 550 / 196.
constexpr int kBigThreads = 512, kBigCluster = 8;
constexpr int kBigWords = 4096;  // bitmap words of a window (131072 columns)
constexpr size_t kBigSmem = (size_t)(2 * kBigWords + kBigCap) * 4;
static_assert(kBigCap >= kBigWords, "the giant path's third array of words");
constexpr int kCtaShare = 1024;
struct RbBigBody {
  using Args = RbArgs;
  static constexpr int kThreads = kBigThreads, kMinBlocks = 2, kCluster = kBigCluster;
  static constexpr size_t kSmem = kBigSmem;

  // The columns of a bitmap word from place `at` on.
  static __device__ __forceinline__ void write_columns(uint32_t m, int col0, int32_t* bcol,
                                                       int at) {
    for (; m; m &= m - 1) bcol[at++] = col0 + __ffs((int)m) - 1;
  }

  static __device__ void big_row(const RbArgs& a, const RbSide& d, int b, uint32_t* bm,
                                 uint32_t* pre, uint32_t* cnt, int* sh, int& nnz) {
    constexpr int T = kBigThreads, kPer = kBigWords / T;
    const int tid = threadIdx.x;
    const int base = d.bptr[b], n = d.bptr[b + 1] - base;
    for (int i = tid; i < min(n, a.B); i += T) cnt[i] = 0u;
    int u = 0;
    for (int w0 = 0; w0 < a.B; w0 += 32 * kBigWords) {
      const int cols = min(32 * kBigWords, a.B - w0), nw = (cols + 31) >> 5;
      for (int x = tid; x < nw; x += T) bm[x] = 0u;
      __syncthreads();
#pragma unroll 4
      for (int i = tid; i < n; i += T) {
        const int c = d.tcol[base + i] - w0;
        if ((unsigned)c < (unsigned)cols) atomicOr(bm + (c >> 5), 1u << (c & 31));
      }
      __syncthreads();
      int nz = 0;
      const int per = (nw + T - 1) / T;
      for (int j = 0; j < per && j < kPer; ++j) {
        const int x = tid * per + j;
        nz += x < nw ? __popc(bm[x]) : 0;
      }
      int tot;
      int run = cta_excl_scan(nz, sh, &tot);
      // columns from the bitmap where the entries are many to a column
      const bool many = n > 4LL * tot;
      for (int j = 0; j < per && j < kPer; ++j) {
        const int x = tid * per + j;
        if (x >= nw) break;
        pre[x] = (uint32_t)run;
        if (many) write_columns(bm[x], w0 + 32 * x, d.bcol + base + u, run);
        run += __popc(bm[x]);
      }
      __syncthreads();
      auto add = [&](auto by_entry) {
#pragma unroll 4
        for (int i = tid; i < n; i += T) {
          const int c = d.tcol[base + i] - w0;
          if ((unsigned)c >= (unsigned)cols) continue;
          const int at = u + (int)pre[c >> 5] + __popc(bm[c >> 5] & ((1u << (c & 31)) - 1u));
          atomicAdd(cnt + at, a.unit ? 1u : d.tw[base + i]);
          if (by_entry) d.bcol[base + at] = c + w0;
        }
      };
      if (many) add(std::false_type{});
      else add(std::true_type{});
      u += tot;
      __syncthreads();
    }
    uint32_t deg = 0u;
    for (int i0 = 0; i0 < u; i0 += T) {
      const int i = i0 + tid;
      const uint32_t c = i < u ? cnt[i] : 0u;
      int tot;
      const uint32_t ex = (uint32_t)cta_excl_scan((int)c, sh, &tot);
      if (i < u) {
        d.bcnt[base + i] = c;
        d.bcum[base + i] = deg + ex + c;
      }
      deg += (uint32_t)tot;
    }
    if (tid == 0) row_done(a, d, b, base, u, deg);
    nnz += u;
    __syncthreads();
  }

  static __device__ void giant_row(const RbArgs& a, const RbSide& d, int b, uint32_t* part,
                                   uint32_t* merged, uint32_t* pre, uint32_t* tots, int* sh,
                                   int& nnz) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int T = kBigThreads, C = kBigCluster;
    const int tid = threadIdx.x, q = (int)cl.block_rank();
    const int base = d.bptr[b], n = d.bptr[b + 1] - base;
    const int e0 = (int)((long long)n * q / C), e1 = (int)((long long)n * (q + 1) / C);
    for (int i = e0 + tid; i < e1; i += T) d.bcnt[base + i] = 0u;
    int u = 0;
    for (int w0 = 0; w0 < a.B; w0 += 32 * kBigWords) {
      const int cols = min(32 * kBigWords, a.B - w0), nw = (cols + 31) >> 5;
      const int seg = (nw + C - 1) / C;  // words a CTA merges: at most T
      for (int x = tid; x < nw; x += T) part[x] = 0u;
      __syncthreads();
#pragma unroll 4
      for (int i = e0 + tid; i < e1; i += T) {
        const int c = d.tcol[base + i] - w0;
        if ((unsigned)c < (unsigned)cols) atomicOr(part + (c >> 5), 1u << (c & 31));
      }
      cl.sync();
      const int x = q * seg + tid;
      uint32_t m = 0u;
      const bool mine = tid < seg && x < nw;
      if (mine)
        for (int p = 0; p < C; ++p) m |= cl.map_shared_rank(part, p)[x];
      int tot;
      const int ex = cta_excl_scan(__popc(m), sh, &tot);
      if (mine)
        for (int p = 0; p < C; ++p) {
          cl.map_shared_rank(merged, p)[x] = m;
          cl.map_shared_rank(pre, p)[x] = (uint32_t)ex;
        }
      if (tid < C) cl.map_shared_rank(tots, tid)[q] = (uint32_t)tot;
      cl.sync();
      uint32_t first[C];  // distinct columns before each segment of words
      uint32_t run = (uint32_t)u, own = 0u;
#pragma unroll
      for (int p = 0; p < C; ++p) {
        first[p] = run;
        if (p == q) own = run;
        run += tots[p];
      }
      // the totals of a window's few distinct columns are added up in shared
      // memory first, and the columns written from the bitmap: the entries of
      // a row of few columns, all of them done in place, queue at the same few
      // words
      const int distinct = (int)run - u;
      const bool local = distinct <= kBigCap - kBigWords;
      uint32_t* const sum = pre + kBigWords;
      auto add = [&](auto in_shared) {
#pragma unroll 4
        for (int i = e0 + tid; i < e1; i += T) {
          const int c = d.tcol[base + i] - w0;
          if ((unsigned)c >= (unsigned)cols) continue;
          const int word = c >> 5, sg = word / seg;
          uint32_t f = first[0];
#pragma unroll
          for (int p = 1; p < C; ++p) f = sg == p ? first[p] : f;
          const int at = (int)(f + pre[word]) + __popc(merged[word] & ((1u << (c & 31)) - 1u));
          const uint32_t w = a.unit ? 1u : d.tw[base + i];
          if (in_shared) {
            atomicAdd(sum + at - u, w);
          } else {
            atomicAdd(d.bcnt + base + at, w);
            d.bcol[base + at] = c + w0;
          }
        }
      };
      if (local) {
        if (mine) write_columns(m, w0 + 32 * x, d.bcol + base, (int)own + ex);
        for (int i = tid; i < distinct; i += T) sum[i] = 0u;
        __syncthreads();
        add(std::true_type{});
        __syncthreads();
        for (int i = tid; i < distinct; i += T)
          if (sum[i]) atomicAdd(d.bcnt + base + u + i, sum[i]);
      } else {
        add(std::false_type{});
      }
      u = (int)run;
    }
    __threadfence();
    cl.sync();
    // running counts: each CTA an eighth of the distinct columns
    const int u0 = (int)((long long)u * q / C), u1 = (int)((long long)u * (q + 1) / C);
    uint32_t own = 0u;
    for (int i = u0 + tid; i < u1; i += T) own += __ldcg(d.bcnt + base + i);
    int tot;
    cta_excl_scan((int)own, sh, &tot);
    if (tid < C) cl.map_shared_rank(tots, tid)[C + q] = (uint32_t)tot;
    cl.sync();
    uint32_t run = 0u, deg = 0u;
#pragma unroll
    for (int p = 0; p < C; ++p) {
      if (p == q) run = deg;
      deg += tots[C + p];
    }
    for (int i0 = u0; i0 < u1; i0 += T) {
      const int i = i0 + tid;
      const uint32_t c = i < u1 ? __ldcg(d.bcnt + base + i) : 0u;
      const uint32_t ex = (uint32_t)cta_excl_scan((int)c, sh, &tot);
      if (i < u1) d.bcum[base + i] = run + ex + c;
      run += (uint32_t)tot;
    }
    if (q == 0) {
      if (tid == 0) row_done(a, d, b, base, u, deg);
      nnz += u;
    }
  }

  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    extern __shared__ __align__(16) unsigned char big_raw[];
    __shared__ int sh[33];
    __shared__ uint32_t tots[2 * kBigCluster];
    uint32_t* const w1 = (uint32_t*)big_raw;
    uint32_t* const w2 = w1 + kBigWords;
    uint32_t* const w3 = w2 + kBigWords;
    // clusters take directions in turn; a cluster's CTAs are consecutive
    const int cluster = vb / kBigCluster, rank = vb % kBigCluster, nc = vg / kBigCluster / 2;
    const int dir = cluster & 1, ci = cluster >> 1;
    const RbSide& d = a.s[dir];
    const int nbig = d.nlist[1], ngiant = d.nlist[2];
    if (nbig + ngiant == 0) return;  // the same in every thread of the cluster
    // giants a CTA takes: of up to kCtaShare entries a giant there is
    const int cta_max = a.B <= kBigCap ? kCtaShare * ngiant : 0;
    const auto len = [&](int b) { return d.bptr[b + 1] - d.bptr[b]; };
    int nnz = 0;
    for (int k = ci; k < ngiant; k += nc)
      if (len(d.giant[k]) > cta_max) giant_row(a, d, d.giant[k], w1, w2, w3, tots, sh, nnz);
    for (int k = ci * kBigCluster + rank; k < ngiant; k += nc * kBigCluster)
      if (len(d.giant[k]) <= cta_max) big_row(a, d, d.giant[k], w1, w2, w3, sh, nnz);
    for (int k = ci * kBigCluster + rank; k < nbig; k += nc * kBigCluster)
      big_row(a, d, d.big[k], w1, w2, w3, sh, nnz);
    if (dir == 0 && threadIdx.x == 0 && nnz) atomicAdd(a.nnz, nnz);
  }
};

// A compact copy of one direction's rows (sbp_build_blockmodel hands the
// rows out back to back): lengths, and after their scan the entries.
struct RbCompactArgs {
  const int32_t *bptr, *bend, *bcol;
  const uint32_t* bcnt;
  int32_t* len;
  const int32_t* ptr;
  int32_t* col;
  uint32_t* cnt;
  int32_t B, fill;  // fill 0: lengths, 1: entries
};

struct RbCompactBody {
  using Args = RbCompactArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    const int lane = threadIdx.x & 31;
    for (int b = (vb * kThreads + threadIdx.x) >> 5; b < a.B; b += (vg * kThreads) >> 5) {
      const int src = a.bptr[b], u = a.bend[b] - src;
      if (!a.fill) {
        if (lane == 0) a.len[b] = u;
        continue;
      }
      const int dst = a.ptr[b];
      for (int i = lane; i < u; i += 32) {
        a.col[dst + i] = a.bcol[src + i];
        a.cnt[dst + i] = a.bcnt[src + i];
      }
    }
  }
};

// ------------------------------------------------------------ block terms --
struct BtArgs {
  const double* xlx;
  const int32_t *optr, *oend, *ocol, *iptr, *iend, *icol;
  const uint32_t *ocnt, *icnt, *ocum, *icum, *d_out, *d_in;
  const double *ld_out, *ld_in;
  double *dSout, *ambout, *ambin, *sinfull;
  int32_t* nbr_s;
  const int32_t* ctl;  // sweep control: gate, and seq += ctl[0] * seq_mul
  int32_t B, pad;
  uint64_t seed;
  uint32_t seq, seq_mul;
};

// One cell's share of a row sum, x log2 x - x * ld, with one rounding order
// (a fused multiply-add) wherever the per-block sums are formed, so the CSR
// and the dense form give the same bits.
__device__ __forceinline__ double cell_term(const double* tab, uint32_t m, double ld) {
  return __fma_rn(-(double)m, ld, xlx(tab, m));
}

// Row sum minus its degree term; d == 0 leaves the sum (log2 0 = -inf).
__device__ __forceinline__ double row_total(double s, uint32_t d, double ld) {
  return d ? __dsub_rn(s, __dmul_rn((double)d, ld)) : s;
}

// The draws of a nodal batch from the CSR rows (as dense_block_draw): eight
// lanes a block search the first entry of out-row ++ in-row whose running
// count exceeds the drawn number, eight ways a step; the block's out-degree
// tells the row.  A warp summing along every row took 91 us a batch of the
// 200k HH graph, up to 700 where a block had 50k entries; this takes 9.
struct BlockDrawBody {
  using Args = BtArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    const uint32_t seq = a.seq + ctl_itr(a.ctl) * a.seq_mul;
    const int lane = threadIdx.x & 31, gl = lane & 7, hb = lane & 24;
    const int ng = (vg * kThreads) >> 3;
    for (int b0 = (vb * kThreads + threadIdx.x) >> 3; b0 - (hb >> 3) < a.B; b0 += ng) {
      const int b = min(b0, a.B - 1);  // idle groups repeat the last block
      const P4 x = draw(a.seed, kRngNodalBlock, seq, (uint32_t)b);
      const uint32_t dout = a.d_out[b];
      const uint64_t deg = (uint64_t)dout + a.d_in[b];
      const uint64_t t64 = scale_draw(x.v[1], deg);
      const bool in = t64 >= dout;
      const uint32_t t = (uint32_t)(in ? t64 - dout : t64);  // below the row's sum
      const int lo = (in ? a.iptr : a.optr)[b];
      const uint32_t* cum = (in ? a.icum : a.ocum) + lo;
      // the entry is one of [first, first + len)
      int first = 0, len = deg ? (in ? a.iend : a.oend)[b] - lo : 0;
      while (__any_sync(kFull, len > 1)) {
        const bool go = len > 1;
        const int step = (len + 7) >> 3;
        const int at = first + min((gl + 1) * step, len) - 1;
        const unsigned m = __ballot_sync(kFull, go && cum[at] > t) >> hb & 0xffu;
        if (go) {
          const int j = __ffs(m) - 1;
          first += j * step;
          len = min(step, len - j * step);
        }
      }
      if (gl == 0 && b0 < a.B) {
        const int nb = len > 0 ? (in ? a.icol : a.ocol)[lo + first] : 0;
        a.nbr_s[b] = accept_random(x.v[0], deg, (uint64_t)a.B) ? -1 : nb;
      }
    }
  }
};

struct BlockTermsBody {
  using Args = BtArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
  if (ctl_stopped(a.ctl)) return;
  int lane = threadIdx.x & 31;
  int w = (vb * blockDim.x + threadIdx.x) >> 5;
  int nw = (vg * blockDim.x) >> 5;
  for (int b = w; b < a.B; b += nw) {
    double acc = 0.0;
    // the row's k-th nonzero is added by lane k % 32, in order of k
    // (unrolled so that several entries' loads are in flight at once)
#pragma unroll 4
    for (int i = a.optr[b] + lane; i < a.oend[b]; i += 32)
      acc += cell_term(a.xlx, a.ocnt[i], a.ld_in[a.ocol[i]]);
    double ao = warp_sum(acc);
    acc = 0.0;
#pragma unroll 4
    for (int i = a.iptr[b] + lane; i < a.iend[b]; i += 32)
      acc += cell_term(a.xlx, a.icnt[i], a.ld_out[a.icol[i]]);
    double ai = warp_sum(acc);
    if (lane == 0) {
      a.ambout[b] = ao;
      a.dSout[b] = row_total(ao, a.d_out[b], a.ld_out[b]);
      a.ambin[b] = ai;
      a.sinfull[b] = row_total(ai, a.d_in[b], a.ld_in[b]);
    }
  }
  }
};


// ------------------------------------------------------------ dense form --
// For small B the blockmodel is kept as two B x B count matrices (rows and
// columns of M both contiguous).  Built once per merge step / golden-section
// restore; after each nodal batch only the edges of the moved vertices are
// applied, with integer atomics (exact, order-independent).

struct DenseArgs {
  const int32_t *osrc, *optr, *oidx, *iptr, *iidx;
  const uint32_t *ow, *iw, *kdo, *kdi;
  const int32_t* part;
  const int32_t* newlab;  // update: new labels of vertices lo..lo+count-1
  uint32_t *Md, *MTd, *Sd, *d_out, *d_in;
  double *ld_out, *ld_in;
  const int32_t* ctl;
  // update: the batch's heavy vertices (more than heavy_min entries in a
  // direction), and the vertices a warp covers
  const int32_t* heavy;
  int32_t N, E, B, lo, count, nheavy, heavy_min, per_warp;
  int32_t unit, combine;  // combine: chunk sums over a warp's lanes first (dense_move_apply)
};

// Chunk sums of a dense cell (r, c): out-row r's chunk of column c and
// in-row c's chunk of row r (DevBM::Sd).
__device__ __forceinline__ uint32_t* sd_out(uint32_t* Sd, int K, int r, int c) {
  return Sd + (size_t)r * 2 * K + (c >> 5);
}
__device__ __forceinline__ uint32_t* sd_in(uint32_t* Sd, int K, int r, int c) {
  return Sd + (size_t)c * 2 * K + K + (r >> 5);
}

// Build step 1: every edge adds its weight to M[r][c] (and the transpose).
struct DenseEdgesBody {
  using Args = DenseArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    int j = vb * blockDim.x + threadIdx.x;
    if (j >= a.E) return;
    int r = a.part[__ldg(a.osrc + j)], c = a.part[__ldg(a.oidx + j)];
    uint32_t w = a.unit ? 1u : __ldg(a.ow + j);
    const int K = (a.B + 31) >> 5;
    atomicAdd(a.Md + (size_t)r * a.B + c, w);
    atomicAdd(a.MTd + (size_t)c * a.B + r, w);
    atomicAdd(sd_out(a.Sd, K, r, c), w);
    atomicAdd(sd_in(a.Sd, K, r, c), w);
  }
};

// Build step 2: block degrees from vertex degrees.
struct DenseDegreesBody {
  using Args = DenseArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    int v = vb * blockDim.x + threadIdx.x;
    if (v >= a.N) return;
    int b = a.part[v];
    atomicAdd(a.d_out + b, a.kdo[v]);
    atomicAdd(a.d_in + b, a.kdi[v]);
  }
};

// Build step 1 after a merge step: the dense form of the merged labels from
// the CSR blockmodel of the labels before it (rebuilt for the merge) and the
// merge map: entry (r, c, count) adds count at (map[r], map[c]).  The same
// integer sums as adding every edge (the counts are the edges' weight sums),
// from nnz entries instead of E edges; a warp per old block row.
struct DenseMapArgs {
  const int32_t *bop, *boe, *boc;
  const uint32_t* bon;
  const int32_t* map;
  uint32_t *Md, *MTd, *Sd;
  int32_t B_old, B;
};

struct DenseFromCsrBody {
  using Args = DenseMapArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    const int lane = threadIdx.x & 31;
    const int K = (a.B + 31) >> 5;
    for (int r = (vb * kThreads + threadIdx.x) >> 5; r < a.B_old; r += (vg * kThreads) >> 5) {
      const int R = a.map[r];
      for (int i = a.bop[r] + lane; i < a.boe[r]; i += 32) {
        const int C = a.map[a.boc[i]];
        const uint32_t w = a.bon[i];
        atomicAdd(a.Md + (size_t)R * a.B + C, w);
        atomicAdd(a.MTd + (size_t)C * a.B + R, w);
        atomicAdd(sd_out(a.Sd, K, R, C), w);
        atomicAdd(sd_in(a.Sd, K, R, C), w);
      }
    }
  }
};

// The CSR blockmodel from a dense form that holds the current labels' M (a
// merge step after sweeps that left the labels as they were): a warp per
// row of M (the out CSR) and of M^T (the in CSR) counts the row's nonzero
// cells, and after the scan writes them in column order with their counts:
// the arrays the rebuild from the edges builds.  Degrees and their log2 are
// the dense form's own.
struct DenseCsrArgs {
  const uint32_t *Md, *MTd;
  int32_t *cnt_o, *cnt_i;  // per row: nonzero cells (the scan's input)
  const int32_t *optr, *iptr;
  int32_t *oend, *iend;
  int32_t *ocol, *icol;
  uint32_t *ocnt, *icnt, *ocum, *icum;
  int32_t* nnz;
  int32_t B, fill;  // fill 0: count, 1: write the rows
};

struct DenseCsrBody {
  using Args = DenseCsrArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int B = a.B;
    for (int t = (vb * kThreads + threadIdx.x) >> 5; t < 2 * B; t += (vg * kThreads) >> 5) {
      const bool in = t >= B;
      const int b = in ? t - B : t;
      const uint32_t* row = (in ? a.MTd : a.Md) + (size_t)b * B;
      int k = 0;
      int32_t* col = nullptr;
      uint32_t *cnt = nullptr, *cum = nullptr;
      if (a.fill) {
        k = (in ? a.iptr : a.optr)[b];
        col = in ? a.icol : a.ocol;
        cnt = in ? a.icnt : a.ocnt;
        cum = in ? a.icum : a.ocum;
      }
      int n = 0;
      uint32_t run = 0u;
      // four chunks of columns in flight at a time
      for (int c0 = 0; c0 < B; c0 += 128) {
        uint32_t m[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + 32 * u + lane;
          m[u] = c < B ? row[c] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const unsigned nz = __ballot_sync(kFull, m[u] != 0u);
          if (a.fill && nz) {
            const uint32_t incl = warp_incl_scan_u(m[u], lane);
            if (m[u]) {
              const int pos = k + n + __popc(nz & lt);
              col[pos] = c0 + 32 * u + lane;
              cnt[pos] = m[u];
              cum[pos] = run + incl;
            }
            run += __shfl_sync(kFull, incl, 31);
          }
          n += __popc(nz);
        }
      }
      if (lane != 0) continue;
      if (!a.fill) {
        (in ? a.cnt_i : a.cnt_o)[b] = n;
      } else {
        (in ? a.iend : a.oend)[b] = k + n;
        if (t == B - 1) *a.nnz = k + n;
      }
    }
  }
};

// Build step 3: log2 of the block degrees.
struct DenseLogsBody {
  using Args = DenseArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int) {
    int b = vb * blockDim.x + threadIdx.x;
    if (b >= a.B) return;
    a.ld_out[b] = log2((double)a.d_out[b]);
    a.ld_in[b] = log2((double)a.d_in[b]);
  }
};

// The moved vertices of a batch: its out-edges move from (r, old block of
// w) to (s, new block of w); its in-edges from unmoved sources move from
// (b(u), r) to (b(u), s).  Edges between two moved vertices are handled
// once, from the source's out-edges.
//
// What bounds a launch is the latency of its longest warp.  A warp covers a
// few batch vertices (one for batches of a few thousand, up to eight, so that
// every SM has some 16 warps): a lane each finds the moved ones and loads
// their row bounds, then the warp strides over all their entries together,
// whatever vertex they belong to.  Heavy vertices, listed, have a CTA each.
// A warp that took eight vertices' moved ones, and their two directions, one
// after the other took 7.5 us a launch at 20k HH in the median and up to 86
// where a heavy vertex moved (13 and 230 at 200k); this 5.3, at most 24.
constexpr int kDuVerts = 8;
struct DenseMove {
  int32_t r, s, o0, no, i0, ni;
};

// What entry e (out-entries, then in-entries) of a moved vertex does: its
// weight moves from cell (r0, c0) to (r1, c1).  Loaded apart from being
// applied, so that the loads of several entries are in flight together (none
// may pass an atomic).
struct DenseCells {
  int32_t r0, c0, r1, c1;
  uint32_t w;  // 0: nothing to do
  bool in;
};
__device__ __forceinline__ DenseCells dense_move_load(const DenseArgs& a, const DenseMove& v,
                                                      int e) {
  const int32_t lo = a.lo, count = a.count;
  const bool in = e >= v.no;
  const int j = in ? v.i0 + e - v.no : v.o0 + e;
  const int x = __ldg((in ? a.iidx : a.oidx) + j);
  const uint32_t wt = a.unit ? 1u : __ldg((in ? a.iw : a.ow) + j);
  const int bo = a.part[x];
  const int bn = x >= lo && x < lo + count ? a.newlab[x - lo] : bo;
  // an in-edge of a moved source is the source's
  return DenseCells{in ? bo : v.r, in ? v.r : bo, in ? bo : v.s, in ? v.s : bn,
                    in && bn != bo ? 0u : wt, in};
}

// The whole warp calls it.  In few blocks the chunk sums are few words that
// every entry of every moved vertex adds to, and that is what a launch takes:
// there the sums at the vertex's own blocks r and s are added up over the
// warp's lanes first, and those at the entry's block, whose change is 0 where r
// and s lie in one chunk, left out.  A launch over 16000 vertices of 24 entries
// that all move, entry by entry / this way: B = 20 319 / 72 us, 50 229 / 84, 130
// 90 / 62, 300 38 / 34, 1000 26 / 26 (and 18 / 20 with fewer moves).  It lengthens
// the chain of a small batch, where nothing queues: weighted 5k partitions 43 /
// 46 ms, so batches of a few thousand vertices go entry by entry.
constexpr int kDuCombine = 512;
template <bool COMBINE>
__device__ __forceinline__ void dense_move_apply(const DenseArgs& a, const DenseCells& m) {
  const int32_t B = a.B;
  const int K = (B + 31) >> 5;
  const bool on = m.w != 0u;
  const unsigned act = COMBINE ? __ballot_sync(kFull, on) : 0u;
  if (!on) return;
  atomicSub(a.Md + (size_t)m.r0 * B + m.c0, m.w);
  atomicSub(a.MTd + (size_t)m.c0 * B + m.r0, m.w);
  atomicAdd(a.Md + (size_t)m.r1 * B + m.c1, m.w);
  atomicAdd(a.MTd + (size_t)m.c1 * B + m.r1, m.w);
  uint32_t *const o0 = sd_out(a.Sd, K, m.r0, m.c0), *const i0 = sd_in(a.Sd, K, m.r0, m.c0);
  uint32_t *const o1 = sd_out(a.Sd, K, m.r1, m.c1), *const i1 = sd_in(a.Sd, K, m.r1, m.c1);
  if constexpr (COMBINE) {
    uint32_t *const e0 = m.in ? o0 : i0, *const e1 = m.in ? o1 : i1;
    if (e0 != e1) {
      atomicSub(e0, m.w);
      atomicAdd(e1, m.w);
    }
    const int lane = threadIdx.x & 31;
    auto add = [&](uint32_t* p, bool minus) {
      const unsigned peers = __match_any_sync(act, (unsigned)(p - a.Sd));
      const uint32_t w = a.unit ? (uint32_t)__popc(peers) : __reduce_add_sync(peers, m.w);
      if (__ffs(peers) - 1 == lane) atomicAdd(p, minus ? 0u - w : w);
    };
    add(m.in ? i0 : o0, true);
    add(m.in ? i1 : o1, false);
  } else {
    atomicSub(o0, m.w);
    atomicSub(i0, m.w);
    atomicAdd(o1, m.w);
    atomicAdd(i1, m.w);
  }
}

template <int U>
__device__ __forceinline__ void dense_move_apply_all(const DenseArgs& a, const DenseCells* c) {
  if (a.combine) {
#pragma unroll
    for (int u = 0; u < U; ++u) dense_move_apply<true>(a, c[u]);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) dense_move_apply<false>(a, c[u]);
  }
}

__device__ __forceinline__ void dense_move_degrees(const DenseArgs& a, int v, int r, int s) {
  const uint32_t o = a.kdo[v], i = a.kdi[v];
  atomicSub(a.d_out + r, o);
  atomicAdd(a.d_out + s, o);
  atomicSub(a.d_in + r, i);
  atomicAdd(a.d_in + s, i);
}

// Four CTAs an SM (64 registers, no spills): at the 90 that the multi-job kernel
// takes otherwise, two, 24 served requests took 195 ms, this way 186.
struct DenseUpdateBody {
  using Args = DenseArgs;
  static constexpr int kThreads = 256, kMinBlocks = 4;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    const int lane = threadIdx.x & 31;
    if (vb < a.nheavy) {
      const int i = a.heavy[vb], v = a.lo + i;
      DenseMove m{a.part[v], a.newlab[i], a.optr[v], 0, a.iptr[v], 0};
      m.no = a.optr[v + 1] - m.o0;
      m.ni = a.iptr[v + 1] - m.i0;
      if (m.r == m.s) return;
      if (threadIdx.x == 0) dense_move_degrees(a, v, m.r, m.s);
      constexpr int U = 4;
      const int n = m.no + m.ni;
      for (int e0 = threadIdx.x & ~31; e0 < n; e0 += U * kThreads) {
        DenseCells c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = e0 + lane + u * kThreads;
          c[u].w = 0u;
          if (e < n) c[u] = dense_move_load(a, m, e);
        }
        dense_move_apply_all<U>(a, c);
      }
      return;
    }
    const int per = a.per_warp;
    const int w0 = (((vb - a.nheavy) * kThreads + threadIdx.x) >> 5) * per;
    const int i = w0 + lane;
    DenseMove m{0, 0, 0, 0, 0, 0};
    if (lane < per && i < a.count) {
      const int v = a.lo + i;
      m.r = a.part[v];
      m.s = a.newlab[i];
      if (m.r != m.s) {
        m.o0 = a.optr[v];
        m.no = a.optr[v + 1] - m.o0;
        m.i0 = a.iptr[v];
        m.ni = a.iptr[v + 1] - m.i0;
        if (m.no > a.heavy_min || m.ni > a.heavy_min) m.no = m.ni = 0;  // listed
        else dense_move_degrees(a, v, m.r, m.s);
      }
    }
    int incl = m.no + m.ni;
#pragma unroll
    for (int o = 1; o < kDuVerts; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(kFull, incl, kDuVerts - 1);
    for (int e0 = 0; e0 < total; e0 += 64) {
      DenseCells c[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = e0 + 32 * h + lane;
        // the vertex of entry e: the first whose running count exceeds it
        int j = 0;
#pragma unroll
        for (int q = 0; q < kDuVerts; ++q) j += __shfl_sync(kFull, incl, q) <= e ? 1 : 0;
        j = min(j, kDuVerts - 1);
        DenseMove u;
        u.r = __shfl_sync(kFull, m.r, j);
        u.s = __shfl_sync(kFull, m.s, j);
        u.o0 = __shfl_sync(kFull, m.o0, j);
        u.no = __shfl_sync(kFull, m.no, j);
        u.i0 = __shfl_sync(kFull, m.i0, j);
        u.ni = __shfl_sync(kFull, m.ni, j);
        const int first = __shfl_sync(kFull, incl, j) - u.no - u.ni;
        c[h].w = 0u;
        if (e < total) c[h] = dense_move_load(a, u, e - first);
      }
      dense_move_apply_all<2>(a, c);
    }
  }
};

// Sum of cell_term over a dense row with the CSR loop's order: each chunk of
// 32 columns hands its nonzeros, by their rank in the row, to lanes
// (rank % 32) through a 32-slot shared buffer of the warp, so every lane adds
// the same terms in the same order as over the row's CSR entries.
// Four chunks at a time: their counts, degrees and cell terms are loaded and
// computed first (independent loads in flight together), then handed out
// chunk by chunk in the same order as one chunk at a time.
__device__ __forceinline__ double dense_row_sum(const double* tab, const uint32_t* row,
                                                const double* ld, int B, int lane,
                                                double* buf) {
  constexpr int U = 4;
  double acc = 0.0;
  int k = 0;  // nonzeros before this chunk
  const unsigned lt = (1u << lane) - 1u;
  for (int c0 = 0; c0 < B; c0 += 32 * U) {
    uint32_t m[U];
    double t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + 32 * u + lane;
      m[u] = c < B ? row[c] : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + 32 * u + lane;
      t[u] = m[u] ? cell_term(tab, m[u], ld[c]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned nz = __ballot_sync(kFull, m[u] != 0u);
      if (nz == 0u) continue;
      const int n = __popc(nz);
      if (m[u]) buf[(k + __popc(nz & lt)) & 31] = t[u];
      __syncwarp();
      if (((lane - k) & 31) < n) acc += buf[lane];
      __syncwarp();
      k += n;
    }
  }
  return acc;
}

struct BtDenseArgs {
  const double* xlx;
  const uint32_t *Md, *MTd, *Sd, *d_out, *d_in;
  const double *ld_out, *ld_in;
  double *dSout, *ambout, *ambin, *sinfull;
  int32_t* nbr_s;
  const int32_t* ctl;  // sweep control: gate, and seq += ctl[0] * seq_mul
  int32_t B;
  int draws;
  uint64_t seed;
  uint32_t seq, seq_mul;
};

struct BlockTermsDenseBody {
  using Args = BtDenseArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
  if (ctl_stopped(a.ctl)) return;
  __shared__ double tbuf[kThreads / 32][32];
  const uint32_t seq = a.seq + ctl_itr(a.ctl) * a.seq_mul;
  int lane = threadIdx.x & 31;
  int w = (vb * blockDim.x + threadIdx.x) >> 5;
  int nw = (vg * blockDim.x) >> 5;
  const int B = a.B;
  for (int b = w; b < B; b += nw) {
    const uint32_t* orow = a.Md + (size_t)b * B;
    const uint32_t* irow = a.MTd + (size_t)b * B;
    if (a.draws != 1) {
    double* buf = tbuf[threadIdx.x >> 5];
    double ao = warp_sum(dense_row_sum(a.xlx, orow, a.ld_in, B, lane, buf));
    double ai = warp_sum(dense_row_sum(a.xlx, irow, a.ld_out, B, lane, buf));
    if (lane == 0) {
      a.ambout[b] = ao;
      a.dSout[b] = row_total(ao, a.d_out[b], a.ld_out[b]);
      a.ambin[b] = ai;
      a.sinfull[b] = row_total(ai, a.d_in[b], a.ld_in[b]);
    }
    }
    if (a.draws)
      dense_block_draw(a.Md, a.MTd, a.Sd, a.d_out, a.d_in, B, a.seed, seq, b, lane, a.nbr_s);
  }
  }
};

__global__ void fill_xlx_kernel(double* tab) {
  uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x < kXlxTable) {
    tab[x] = xlog2x(x);
    tab[kXlxTable + x] = log2((double)x);
  }
}

struct MdlArgs {
  const double* dSout;
  double* out;  // written at out[ctl[0]] under sweep control
  const int32_t* ctl;
  int32_t B, pad;
};

// data_S = sum of dSout over the blocks, one CTA per job, fixed order.
struct MdlSumBody {
  using Args = MdlArgs;
  static constexpr int kThreads = 512, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int, int) {
    if (ctl_stopped(a.ctl)) return;
    __shared__ double sh[kThreads];
    double s = 0.0;
    for (int b = threadIdx.x; b < a.B; b += kThreads) s += a.dSout[b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) a.out[ctl_itr(a.ctl)] = sh[0];
  }
};

// The stop test of a queued sweep (partition.hpp:920-934), one thread per
// job, after the sweep's MDL: ctl[0] = sweeps done so far including this
// one; ctl[1] = 1 once the moving-average dS test or the sweep limit ends
// the outer step.  The arithmetic is the host's, operation for operation.
struct SweepCtlArgs {
  int32_t* ctl;
  const double* dsum;   // per sweep of the outer step
  const double* dataS;  // per sweep of the outer step
  double model_S;       // E(1+x)ln(1+x) - x ln x + N ln B of the step's B
  double thr;           // threshold1 or threshold2 by the bracket's state
  int32_t window;       // 0: no stop test (a fixed number of sweeps)
  int32_t max_itr;
};

struct SweepCtlBody {
  using Args = SweepCtlArgs;
  static constexpr int kThreads = 32, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int, int) {
    if (threadIdx.x != 0 || a.ctl[1] != 0) return;
    const int itr = a.ctl[0];
    bool stop = false;
    if (a.window > 0 && itr >= a.window - 1) {
      double mean = 0.0;
      for (int i = itr - a.window + 1; i < itr; ++i) mean += a.dsum[i];
      mean /= (double)(a.window - 1);
      const double S = a.model_S - a.dataS[itr];
      stop = -mean < a.thr * S;
    }
    a.ctl[0] = itr + 1;
    if (stop || itr + 1 >= a.max_itr) a.ctl[1] = 1;
  }
};

// Small utility bodies of the multi-job engine.
struct WordsArgs {
  uint32_t* dst;
  const uint32_t* src;  // copy source (copy body)
  long long n;          // 32-bit words
  const int32_t* ctl;
};

struct ZeroBody {
  using Args = WordsArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    for (long long i = (long long)vb * kThreads + threadIdx.x; i < a.n;
         i += (long long)vg * kThreads)
      a.dst[i] = 0u;
  }
};

struct CopyBody {
  using Args = WordsArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    for (long long i = (long long)vb * kThreads + threadIdx.x; i < a.n;
         i += (long long)vg * kThreads)
      a.dst[i] = a.src[i];
  }
};

struct IotaBody {
  using Args = WordsArgs;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  static constexpr size_t kSmem = 0;
  static __device__ void run(const Args& a, int vb, int vg) {
    if (ctl_stopped(a.ctl)) return;
    for (long long i = (long long)vb * kThreads + threadIdx.x; i < a.n;
         i += (long long)vg * kThreads)
      a.dst[i] = (uint32_t)i;
  }
};

int grid_for(long long items, int per_block, int cap) {
  long long g = (items + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

RbArgs rb_args(const DevGraph& g, const int32_t* part, int32_t B, DevBM& m, RebuildScratch& rs,
               const RebuildTune& t) {
  RbArgs a{};
  a.tile_cap = std::max(32, std::min(kTileMaxCap, t.warp_cap));
  a.warp_max = std::max(256, std::min(kRankMax, t.big_entries));
  // about half a tile's entries, so that most tiles take one round
  a.tile_rows = (int32_t)std::max<long long>(
      8, std::min<long long>(RbTileBody::kThreads,
                             (long long)kTileEntries / 2 * B / std::max(g.E, 1)));
  a.unit = g.unit;
  a.part = part;
  a.xlx = m.xlx;
  a.nnz = m.nnz;
  a.N = g.N;
  a.E = g.E;
  a.B = B;
  for (int dir = 0; dir < 2; ++dir) {
    RbSide& s = a.s[dir];
    const RebuildDir& r = rs.d[dir];
    s.gptr = dir == 0 ? g.optr : g.iptr;
    s.gidx = dir == 0 ? g.oidx : g.iidx;
    s.gw = dir == 0 ? g.ow : g.iw;
    s.gsrc = dir == 0 ? g.osrc : g.isrc;
    s.cnt = r.cnt;
    s.vofs = r.vofs;
    s.tcol = r.tcol;
    s.tw = r.tw;
    s.mid = r.mid;
    s.big = r.big;
    s.giant = r.giant;
    s.nlist = rs.nlist + 3 * dir;
    s.bptr = dir == 0 ? m.optr : m.iptr;
    s.bend = dir == 0 ? m.oend : m.iend;
    s.bcol = dir == 0 ? m.ocol : m.icol;
    s.bcnt = dir == 0 ? m.ocnt : m.icnt;
    s.bcum = dir == 0 ? m.ocum : m.icum;
    s.bdeg = dir == 0 ? m.d_out : m.d_in;
    s.bld = dir == 0 ? m.ld_out : m.ld_in;
  }
  return a;
}

// Virtual grids: functions of one job's sizes only.
int32_t vg_count(const RbArgs& a) { return 2 * ceil_div(a.N, 256); }
int32_t vg_scatter(const RbArgs& a) { return a.E > 0 ? 2 * ceil_div(a.E, 256) : 0; }
int32_t vg_tile(const RbArgs& a) { return 2 * ceil_div(a.B, a.tile_rows); }
// segments longer than tile_cap entries number at most E / tile_cap
int32_t vg_rank(const RbArgs& a) {
  return 2 * grid_for(a.E / (a.tile_cap + 1), kRankWarps, 148 * 2);
}
int32_t vg_big(const RbArgs& a) {
  return 2 * kBigCluster * grid_for(a.E / (a.warp_max + 1), kBigCluster, 16);
}
int32_t vg_words(long long n) {
  return n <= 0 ? 0 : (int32_t)std::min<long long>(4096, (n + 2047) / 2048);
}

BtArgs bt_args(DevBM& m, int32_t B, uint64_t seed, uint32_t seq) {
  BtArgs a{};
  a.xlx = m.xlx;
  a.optr = m.optr; a.oend = m.oend; a.ocol = m.ocol;
  a.iptr = m.iptr; a.iend = m.iend; a.icol = m.icol;
  a.ocnt = m.ocnt; a.icnt = m.icnt; a.ocum = m.ocum; a.icum = m.icum;
  a.d_out = m.d_out; a.d_in = m.d_in;
  a.ld_out = m.ld_out; a.ld_in = m.ld_in;
  a.dSout = m.dSout; a.ambout = m.ambout; a.ambin = m.ambin; a.sinfull = m.sinfull;
  a.nbr_s = m.nbr_s;
  a.B = B; a.seed = seed; a.seq = seq;
  return a;
}

BtDenseArgs bt_dense_args(DevBM& m, int32_t B, int draws, uint64_t seed, uint32_t seq) {
  BtDenseArgs a{};
  a.xlx = m.xlx;
  a.Md = m.Md; a.MTd = m.MTd; a.Sd = m.Sd; a.d_out = m.d_out; a.d_in = m.d_in;
  a.ld_out = m.ld_out; a.ld_in = m.ld_in;
  a.dSout = m.dSout; a.ambout = m.ambout; a.ambin = m.ambin; a.sinfull = m.sinfull;
  a.nbr_s = m.nbr_s;
  a.B = B; a.draws = draws; a.seed = seed; a.seq = seq;
  return a;
}

DenseArgs dense_args(const DevGraph& g, const int32_t* part, int32_t B, DevBM& m) {
  DenseArgs a{};
  a.osrc = g.osrc; a.optr = g.optr; a.oidx = g.oidx; a.iptr = g.iptr; a.iidx = g.iidx;
  a.ow = g.ow; a.iw = g.iw; a.kdo = g.kdo; a.kdi = g.kdi;
  a.part = part;
  a.Md = m.Md; a.MTd = m.MTd; a.Sd = m.Sd; a.d_out = m.d_out; a.d_in = m.d_in;
  a.ld_out = m.ld_out; a.ld_in = m.ld_in;
  a.N = g.N; a.E = g.E; a.B = B;
  a.unit = g.unit;
  return a;
}

int32_t vg_block_terms(int32_t B) { return grid_for((long long)B * 32, 256, 8192); }
int32_t vg_block_draw(int32_t B) { return grid_for((long long)B * 8, 256, 8192); }
// The update's arguments for a batch: some 16 warps an SM where the batch
// has the vertices for it.
void set_update(DenseArgs& a, int32_t lo, int32_t count, const int32_t* newlab,
                const NodalAux& lists) {
  a.lo = lo;
  a.count = count;
  a.newlab = newlab;
  a.heavy = lists.heavy;
  a.nheavy = lists.nheavy;
  a.heavy_min = nodal_heavy_threshold();
  a.per_warp = std::max(1, std::min(kDuVerts, count / (148 * 16)));
  a.combine = a.B <= kDuCombine && a.per_warp > 1 ? 1 : 0;
}
int32_t vg_dense_update(const DenseArgs& a) {
  return a.nheavy + ceil_div(a.count, DenseUpdateBody::kThreads / 32 * a.per_warp);
}

const MultiKernel kmScanTile = multi_kernel_desc<ScanTileBody>("scan_tile");
const MultiKernel kmScanSingle = multi_kernel_desc<ScanSingleBody>("scan_single");
const MultiKernel kmScanApply = multi_kernel_desc<ScanApplyBody>("scan_apply");
const MultiKernel kmRbCount = multi_kernel_desc<RbCountBody>("rb_count");
const MultiKernel kmRbScatter = multi_kernel_desc<RbScatterBody>("rb_scatter");
const MultiKernel kmRbTile = multi_kernel_desc<RbTileBody>("rb_tile");
const MultiKernel kmRbRank = multi_kernel_desc<RbRankBody>("rb_rank");
const MultiKernel kmRbBig = multi_kernel_desc<RbBigBody>("rb_big");
const MultiKernel kmBlockDraw = multi_kernel_desc<BlockDrawBody>("block_draw");
const MultiKernel kmBlockTerms = multi_kernel_desc<BlockTermsBody>("block_terms");
const MultiKernel kmBlockTermsDense = multi_kernel_desc<BlockTermsDenseBody>("block_terms_dense");
const MultiKernel kmDenseEdges = multi_kernel_desc<DenseEdgesBody>("dense_edges");
const MultiKernel kmDenseFromCsr = multi_kernel_desc<DenseFromCsrBody>("dense_from_csr");
const MultiKernel kmDenseCsr = multi_kernel_desc<DenseCsrBody>("dense_csr");
const MultiKernel kmDenseDegrees = multi_kernel_desc<DenseDegreesBody>("dense_degrees");
const MultiKernel kmDenseLogs = multi_kernel_desc<DenseLogsBody>("dense_logs");
const MultiKernel kmDenseUpdate = multi_kernel_desc<DenseUpdateBody>("dense_update");
const MultiKernel kmMdlSum = multi_kernel_desc<MdlSumBody>("mdl_sum");
const MultiKernel kmSweepCtl = multi_kernel_desc<SweepCtlBody>("sweep_ctl");
const MultiKernel kmZero = multi_kernel_desc<ZeroBody>("zero");
const MultiKernel kmCopy = multi_kernel_desc<CopyBody>("copy");
const MultiKernel kmIota = multi_kernel_desc<IotaBody>("iota");

// One job's scan records: short arrays in one CTA, longer ones in three steps.
void add_scan(Slot* sl, const int32_t* in, int32_t* out, int32_t n, int32_t* tile,
              const int32_t* ctl) {
  ScanArgs a{};
  a.ctl = ctl;
  if (n <= kScanSingleMax) {
    a.in = in;
    a.out = out;
    a.n = n;
    slot_push(slot_bind(sl[1], kmScanSingle), a, 1);
    return;
  }
  const int32_t tiles = ceil_div(n, kScanTile);
  a.in = in;
  a.out = out;
  a.tile = tile;
  a.n = n;
  slot_push(slot_bind(sl[0], kmScanTile), a, tiles);
  ScanArgs b{};
  b.in = tile;
  b.out = tile + tiles;
  b.n = tiles;
  b.ctl = ctl;
  slot_push(slot_bind(sl[1], kmScanSingle), b, 1);
  a.tile = tile + tiles;
  slot_push(slot_bind(sl[2], kmScanApply), a, tiles);
}

}  // namespace

void add_exclusive_scan(Slot* sl, const int32_t* in, int32_t* out, int32_t n, int32_t* tile) {
  add_scan(sl, in, out, n, tile, nullptr);
}

cudaError_t init_kernel_attributes() {
  cudaError_t e = allow_smem<RbRankBody>();
  cudaError_t e2 = allow_smem<RbBigBody>();
  return e != cudaSuccess ? e : e2;
}

void scan_exclusive(const int32_t* in, int32_t* out, int32_t n, int32_t* tile, cudaStream_t st) {
  ScanArgs a{};
  a.in = in;
  a.out = out;
  a.n = n;
  if (n <= kScanSingleMax) {
    launch_single<ScanSingleBody>(a, 1, st);
    return;
  }
  int tiles = ceil_div(n, kScanTile);
  a.tile = tile;
  launch_single<ScanTileBody>(a, tiles, st);
  ScanArgs b{};
  b.in = tile;
  b.out = tile + tiles;
  b.n = tiles;
  launch_single<ScanSingleBody>(b, 1, st);
  a.tile = tile + tiles;
  launch_single<ScanApplyBody>(a, tiles, st);
}

RebuildListCaps rebuild_list_caps(int32_t N, int32_t E) {
  return RebuildListCaps{(size_t)std::min(N, E / 32) + 1, (size_t)E / 256 + 1,
                         (size_t)E / kBigCap + 1};
}

void rebuild_blockmodel(const DevGraph& g, const int32_t* part, int32_t B, DevBM& m,
                        RebuildScratch& rs, cudaStream_t st, const RebuildTune& t) {
  RbArgs a = rb_args(g, part, B, m, rs, t);
  for (int dir = 0; dir < 2; ++dir)
    cudaMemsetAsync(rs.d[dir].cnt, 0, sizeof(int32_t) * (size_t)B, st);
  cudaMemsetAsync(rs.nlist, 0, sizeof(int32_t) * kRebuildCounters, st);
  launch_single<RbCountBody>(a, vg_count(a), st);
  for (int dir = 0; dir < 2; ++dir)
    scan_exclusive(rs.d[dir].cnt, dir == 0 ? m.optr : m.iptr, B,
                   rs.tile + dir * (rs.tile_cap / 2), st);
  launch_single<RbScatterBody>(a, vg_scatter(a), st);
  launch_single<RbTileBody>(a, vg_tile(a), st);
  launch_single<RbRankBody>(a, vg_rank(a), st);
  launch_single<RbBigBody>(a, vg_big(a), st);
}

void compact_rows(const DevBM& m, int32_t B, bool in, RebuildScratch& rs, int32_t* ptr,
                  int32_t* col, uint32_t* cnt, cudaStream_t st) {
  const RebuildDir& r = rs.d[in ? 1 : 0];
  RbCompactArgs a{in ? m.iptr : m.optr, in ? m.iend : m.oend, in ? m.icol : m.ocol,
                  in ? m.icnt : m.ocnt, r.cnt, ptr, col, cnt, B, 0};
  const int32_t vg = grid_for((long long)B * 32, RbCompactBody::kThreads, 4096);
  launch_single<RbCompactBody>(a, vg, st);
  scan_exclusive(r.cnt, ptr, B, rs.tile, st);
  a.fill = 1;
  launch_single<RbCompactBody>(a, vg, st);
}

void block_terms(DevBM& m, int32_t B, int draws, uint64_t seed, uint32_t seq, cudaStream_t st) {
  const BtArgs a = bt_args(m, B, seed, seq);
  if (draws) launch_single<BlockDrawBody>(a, vg_block_draw(B), st);
  else launch_single<BlockTermsBody>(a, vg_block_terms(B), st);
}

void fill_xlx_table(double* tab, cudaStream_t st) {
  ++g_launches;
  fill_xlx_kernel<<<kXlxTable / 256, 256, 0, st>>>(tab);
}

void dense_build(const DevGraph& g, const int32_t* part, int32_t B, DevBM& m, cudaStream_t st) {
  size_t bb = (size_t)B * B;
  cudaMemsetAsync(m.Md, 0, bb * sizeof(uint32_t), st);
  cudaMemsetAsync(m.MTd, 0, bb * sizeof(uint32_t), st);
  cudaMemsetAsync(m.Sd, 0, (size_t)2 * B * ((B + 31) / 32) * sizeof(uint32_t), st);
  cudaMemsetAsync(m.d_out, 0, (size_t)B * sizeof(uint32_t), st);
  cudaMemsetAsync(m.d_in, 0, (size_t)B * sizeof(uint32_t), st);
  DenseArgs a = dense_args(g, part, B, m);
  if (g.E > 0) launch_single<DenseEdgesBody>(a, ceil_div(g.E, 256), st);
  launch_single<DenseDegreesBody>(a, ceil_div(g.N, 256), st);
  launch_single<DenseLogsBody>(a, ceil_div(B, 256), st);
}

void block_terms_dense(DevBM& m, int32_t B, int draws, uint64_t seed, uint32_t seq,
                       cudaStream_t st) {
  launch_single<BlockTermsDenseBody>(bt_dense_args(m, B, draws, seed, seq), vg_block_terms(B),
                                     st);
}

void mdl_data_sum(const DevBM& m, int32_t B, double* out, cudaStream_t st) {
  MdlArgs a{m.dSout, out, nullptr, B, 0};
  launch_single<MdlSumBody>(a, 1, st);
}

// -------------------------------------------------------------- autotuner --
// The rebuild's segment widths (the longest segment ranked by comparison, and
// the longest one a warp ranks through a bitmap) are picked by
// timing rebuilds of a job's own blockmodel, once per device and size class
// (log2 of B and of the mean segment length E/B).  Every candidate builds
// the same matrix, so the choice changes only the time.
namespace {
struct TuneKey {
  int device, lb, ls;
  bool operator<(const TuneKey& o) const {
    return device != o.device ? device < o.device : lb != o.lb ? lb < o.lb : ls < o.ls;
  }
};
std::mutex g_tune_mu;
std::map<TuneKey, RebuildTune> g_tune;

int ilog2(long long x) {
  int l = 0;
  while (x > 1) {
    x >>= 1;
    ++l;
  }
  return l;
}

TuneKey tune_key(int device, int32_t E, int32_t B) {
  return TuneKey{device, ilog2(std::max(B, 1)), ilog2(std::max<long long>(1, (long long)E / std::max(B, 1)))};
}
}  // namespace

bool rebuild_tuned(int device, int32_t E, int32_t B, RebuildTune* out) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  auto it = g_tune.find(tune_key(device, E, B));
  if (it == g_tune.end()) return false;
  *out = it->second;
  return true;
}

cudaError_t tune_rebuild(int device, const DevGraph& g, const int32_t* part, int32_t B, DevBM& m,
                         RebuildScratch& rs, cudaStream_t st, RebuildTune* out) {
  std::vector<RebuildTune> cands;
  for (int wc : {32, 64, 128})
    for (int be : {1024, 512}) cands.push_back(RebuildTune{wc, be});
  cudaEvent_t e0, e1;
  cudaError_t err = cudaEventCreate(&e0);
  if (err != cudaSuccess) return err;
  err = cudaEventCreate(&e1);
  if (err != cudaSuccess) {
    cudaEventDestroy(e0);
    return err;
  }
  RebuildTune best = RebuildTune{};
  float best_ms = 1e30f;
  for (const RebuildTune& c : cands) {
    rebuild_blockmodel(g, part, B, m, rs, st, c);  // warm
    float ms = 0.f;
    cudaEventRecord(e0, st);
    for (int r = 0; r < 2; ++r) rebuild_blockmodel(g, part, B, m, rs, st, c);
    cudaEventRecord(e1, st);
    err = cudaEventSynchronize(e1);
    if (err != cudaSuccess) break;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best_ms) {
      best_ms = ms;
      best = c;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune[tune_key(device, g.E, B)] = best;
  *out = best;
  return cudaSuccess;
}

// ------------------------------------------------------ multi-job records --
void RebuildSlots::clear() {
  for (Slot* x : all()) x->clear();
}

std::vector<Slot*> RebuildSlots::all() {
  return {&zero, &count, &scan1[0], &scan1[1], &scan1[2], &scatter, &tile, &rank, &big,
          &dense_count, &scan2[0], &scan2[1], &scan2[2], &dense_fill};
}

void add_csr_from_dense(RebuildSlots& s, int32_t B, DevBM& m, RebuildScratch& rs) {
  DenseCsrArgs a{m.Md, m.MTd, rs.d[0].cnt, rs.d[1].cnt, m.optr, m.iptr, m.oend, m.iend,
                 m.ocol, m.icol, m.ocnt, m.icnt, m.ocum, m.icum, m.nnz, B, 0};
  const int32_t vg = grid_for((long long)2 * B * 32, 256, 148 * 16);
  slot_push(slot_bind(s.dense_count, kmDenseCsr), a, vg);
  for (int dir = 0; dir < 2; ++dir)
    add_scan(s.scan2, rs.d[dir].cnt, dir == 0 ? m.optr : m.iptr, B,
             rs.tile + dir * (rs.tile_cap / 2), nullptr);
  a.fill = 1;
  slot_push(slot_bind(s.dense_fill, kmDenseCsr), a, vg);
}

void add_rebuild(RebuildSlots& s, const DevGraph& g, const int32_t* part, int32_t B, DevBM& m,
                 RebuildScratch& rs, const int32_t* ctl, const RebuildTune& t) {
  RbArgs a = rb_args(g, part, B, m, rs, t);
  a.ctl = ctl;
  for (int dir = 0; dir < 2; ++dir) add_zero(s.zero, rs.d[dir].cnt, (size_t)B, ctl);
  add_zero(s.zero, rs.nlist, kRebuildCounters, ctl);
  slot_push(slot_bind(s.count, kmRbCount), a, vg_count(a));
  for (int dir = 0; dir < 2; ++dir)
    add_scan(s.scan1, rs.d[dir].cnt, dir == 0 ? m.optr : m.iptr, B,
             rs.tile + dir * (rs.tile_cap / 2), ctl);
  slot_push(slot_bind(s.scatter, kmRbScatter), a, vg_scatter(a));
  slot_push(slot_bind(s.tile, kmRbTile), a, vg_tile(a));
  slot_push(slot_bind(s.rank, kmRbRank), a, vg_rank(a));
  slot_push(slot_bind(s.big, kmRbBig), a, vg_big(a));
}

void DenseBuildSlots::clear() {
  for (Slot* x : all()) x->clear();
}

std::vector<Slot*> DenseBuildSlots::all() { return {&zero, &edges, &mapped, &degrees, &logs}; }

void add_dense_build(DenseBuildSlots& s, const DevGraph& g, const int32_t* part, int32_t B,
                     DevBM& m) {
  const size_t bb = (size_t)B * B;
  add_zero(s.zero, m.Md, bb);
  add_zero(s.zero, m.MTd, bb);
  add_zero(s.zero, m.Sd, (size_t)2 * B * ((B + 31) / 32));
  add_zero(s.zero, m.d_out, (size_t)B);
  add_zero(s.zero, m.d_in, (size_t)B);
  DenseArgs a = dense_args(g, part, B, m);
  slot_push(slot_bind(s.edges, kmDenseEdges), a, g.E > 0 ? ceil_div(g.E, 256) : 0);
  slot_push(slot_bind(s.degrees, kmDenseDegrees), a, ceil_div(g.N, 256));
  slot_push(slot_bind(s.logs, kmDenseLogs), a, ceil_div(B, 256));
}

void add_dense_build_mapped(DenseBuildSlots& s, const DevGraph& g, const int32_t* part,
                            int32_t B, DevBM& m, int32_t B_old, const int32_t* map) {
  const size_t bb = (size_t)B * B;
  add_zero(s.zero, m.Md, bb);
  add_zero(s.zero, m.MTd, bb);
  add_zero(s.zero, m.Sd, (size_t)2 * B * ((B + 31) / 32));
  add_zero(s.zero, m.d_out, (size_t)B);
  add_zero(s.zero, m.d_in, (size_t)B);
  DenseMapArgs b{m.optr, m.oend, m.ocol, m.ocnt, map, m.Md, m.MTd, m.Sd, B_old, B};
  slot_push(slot_bind(s.mapped, kmDenseFromCsr), b, grid_for((long long)B_old * 32, 256, 148 * 16));
  DenseArgs a = dense_args(g, part, B, m);
  slot_push(slot_bind(s.degrees, kmDenseDegrees), a, ceil_div(g.N, 256));
  slot_push(slot_bind(s.logs, kmDenseLogs), a, ceil_div(B, 256));
}

void add_dense_update(Slot& s, const DevGraph& g, const int32_t* part, int32_t lo, int32_t count,
                      const int32_t* newlab, int32_t B, DevBM& m, const NodalAux& lists,
                      const int32_t* ctl) {
  if (count <= 0) return;
  DenseArgs a = dense_args(g, part, B, m);
  a.ctl = ctl;
  set_update(a, lo, count, newlab, lists);
  slot_push(slot_bind(s, kmDenseUpdate), a, vg_dense_update(a));
}

void add_block_terms(Slot& s, DevBM& m, int32_t B, const int32_t* ctl) {
  BtArgs a = bt_args(m, B, 0, 0);
  a.ctl = ctl;
  slot_push(slot_bind(s, kmBlockTerms), a, vg_block_terms(B));
}

void add_block_draw(Slot& s, DevBM& m, int32_t B, uint64_t seed, uint32_t seq,
                    const int32_t* ctl, uint32_t seq_mul) {
  BtArgs a = bt_args(m, B, seed, seq);
  a.ctl = ctl;
  a.seq_mul = seq_mul;
  slot_push(slot_bind(s, kmBlockDraw), a, vg_block_draw(B));
}

void add_block_terms_dense(Slot& s, DevBM& m, int32_t B, int draws, uint64_t seed,
                           uint32_t seq, const int32_t* ctl, uint32_t seq_mul) {
  BtDenseArgs a = bt_dense_args(m, B, draws, seed, seq);
  a.ctl = ctl;
  a.seq_mul = seq_mul;
  slot_push(slot_bind(s, kmBlockTermsDense), a, vg_block_terms(B));
}

void add_mdl_sum(Slot& s, const DevBM& m, int32_t B, double* out, const int32_t* ctl) {
  MdlArgs a{m.dSout, out, ctl, B, 0};
  slot_push(slot_bind(s, kmMdlSum), a, 1);
}

void add_sweep_ctl(Slot& s, int32_t* ctl, const double* dsum, const double* dataS,
                   double model_S, double thr, int32_t window, int32_t max_itr) {
  SweepCtlArgs a{ctl, dsum, dataS, model_S, thr, window, max_itr};
  slot_push(slot_bind(s, kmSweepCtl), a, 1);
}

void add_zero(Slot& s, void* p, size_t words, const int32_t* ctl) {
  WordsArgs a{(uint32_t*)p, nullptr, (long long)words, ctl};
  slot_push(slot_bind(s, kmZero), a, vg_words((long long)words));
}

void add_copy(Slot& s, void* dst, const void* src, size_t words) {
  WordsArgs a{(uint32_t*)dst, (const uint32_t*)src, (long long)words, nullptr};
  slot_push(slot_bind(s, kmCopy), a, vg_words((long long)words));
}

void add_iota(Slot& s, int32_t* p, int32_t n) {
  WordsArgs a{(uint32_t*)p, nullptr, (long long)n, nullptr};
  slot_push(slot_bind(s, kmIota), a, vg_words(n));
}

}  // namespace sbp
