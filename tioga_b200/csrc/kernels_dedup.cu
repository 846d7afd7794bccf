// Coincident query points: uniquenodes_octree / uniqNodesTree
// (src/utils.c:622-737), called by MeshBlock::search (src/search.C:242-263).
//
// The reference merges query points of one donor block that lie within TOL
// of each other (L1) and share the receptor mesh tag: the lower query index
// takes the larger receptor resolution, the higher one points to the lower
// one's representative (xtag), only representatives are searched and the
// others copy their donor, the donor side sends res_search[xtag[i]]
// (src/bookKeeping.C:108), and resetCoincident (src/bookKeeping.C:572-597)
// keeps a copy cancelled only if every copy is.
//
// Which points are compared, and in which order, follows the reference's
// octree exactly:
//  * a subset of more than 20 points is split at the middle of its bounding
//    box (widened by TOL) into octants, unless all of them fall into one
//    octant; the subsets depend only on the points, not on their order;
//  * each split reverses the order within an octant, so the points of a leaf
//    are in the donor list's order after an even number of splits and in the
//    reverse order after an odd number;
//  * the donor list's order is pair order, then the receptor block's
//    10x10x10 OBB bin (MeshBlock.C:171-224), then descending node id within a
//    bin, as getQueryPoints2 visits them (MeshBlock.C:953-1117).
// Here the subsets are emulated level by level on the device (exact FP64 box
// reductions with ordered keys, the reference's midpoint and octant
// arithmetic), three launches a level with the subsets' table on the device
// too: a split only has to put the points into the right subset, so points
// take their places by atomics, and the leaves sort their few members.  A warp
// per leaf then runs the reference's pairwise loop in that order.  (127 k query
// points: gathering and merging 1.57 ms with a radix sort, three uploads and a
// read-back per level, 0.46 ms now; 472 k points of cubic elements 3.0 ms less.)
#include "kernels.cuh"

namespace tb {

// the 10x10x10 bin of a node in its block's OBB frame (MeshBlock.C:171-224)
__device__ __forceinline__ short node_bin_of(const double p[3], const Obb& o) {
  int idx[3];
  for (int j = 0; j < 3; j++) {
    double xd = o.dxc[j];
    for (int k = 0; k < 3; k++) xd += (p[k] - o.xc[k]) * o.vec[j][k];
    const double mdx = 2 * o.dxc[j] / 10;
    int i = (mdx > 0) ? (int)(xd / mdx) : 0;
    idx[j] = min(max(i, 0), 9);
  }
  return (short)(idx[2] * 100 + idx[1] * 10 + idx[0]);
}

// ---------------------------------------------------------------------------
// Preprocess gate: does any block hold two nodes closer than delta (L1)?
// Each node files itself under every cell of a per-block grid that its
// delta-box touches (a cell is 32 delta wide: 1.2 cells on average), so two
// such nodes always share a cell.  The files are one open-addressing hash table of node ids
// (from the cell's hash in steps that the hash gives too): an entry that is filed
// walks past every entry filed under its cell before it, and is compared with
// each one it meets.  What the kernel takes is its longest walk, an atomic and a
// load a probe, which steps of one made long by their clusters (6 k nodes 27 us,
// 340 k 36 us; 18 and 24 us now).  The table is at most half full and there is one pass over the
// nodes; sorting the (cell, node) list instead took 13 launches and 24 bytes
// of traffic per node and radix pass (a host step of 340 k nodes 2722 us with
// it, 2482 us now; of 6 k nodes 1056 and 902 us).
//
// On a strongly graded block (nodes a few delta apart in a far field 10^5 of
// them wide) a filing cell holds thousands of nodes.  A walk longer than any on
// an ordinary mesh (at a table half full of 20 M entries the longest is about
// 25) therefore ends the pass as crowded, and the host has the gate decided on
// cells 2 delta wide instead: nodes that are not closer than delta lie at most
// some dozens in such a cell, whatever the mesh.  Each is filed once, under its
// own cell (k_coin_file), and then looks through the cells that its delta-box
// touches (k_coin_compare).  30^3 nodes two delta apart: a preprocess 0.30 ms; it
// took 29 ms with walks of up to 4096, and 0.55 ms with the sorted list.
// ---------------------------------------------------------------------------
constexpr int kCoinBits = 17;      // delta is a quarter of a cell of 2^17 per axis (at least 10 TOL)
constexpr int kCoinCoarse = 8;     // width of a filing cell in those cells
constexpr int kCoinWalk = 128;     // a longer walk counts as crowded
constexpr double kCoinFine = 2.01; // width of a crowded gate's cells in delta
constexpr int kCoinProbes = 4096;  // there a longer walk counts as close nodes (the merge then runs)
constexpr unsigned kCoinClose = 1u, kCoinCrowded = 2u;  // the gate's flag

// delta of a block, and a cell's place in the table
__device__ __forceinline__ double coin_delta(const BlockInfo& B) {
  double ext = 0;
  for (int k = 0; k < 3; k++) ext = fmax(ext, (double)B.bb_hi[k] - (double)B.bb_lo[k]);
  return 0.25 * fmax(ext / (double)(1 << kCoinBits), 40.0 * kTol);
}
__device__ __forceinline__ void coin_place(int b, int i, int j, int k, unsigned mask, unsigned& at, unsigned& step) {
  unsigned long long h = ((unsigned long long)b << 51) ^ ((unsigned long long)i << 34) ^ ((unsigned long long)j << 17) ^
                         (unsigned long long)k;
  h *= 0x9E3779B97F4A7C15ull;  // Fibonacci hashing: the high bits
  at = (unsigned)(h >> 32) & mask;
  step = (unsigned)(h >> 13) | 1u;  // (odd: the walk meets every entry)
}
__device__ __forceinline__ bool coin_close(const double* __restrict__ x, const blk_t* __restrict__ node_blk,
                                           const double p[3], int g, int b, int other, double delta) {
  const double* o = x + 3ll * other;  // (both loads under way at once)
  const int ob = node_blk[other];
  const double d = fabs(p[0] - o[0]) + fabs(p[1] - o[1]) + fabs(p[2] - o[2]);
  return other != g && ob == b && d < delta;
}

__global__ void k_coin_hash(const double* __restrict__ x, const blk_t* __restrict__ node_blk,
                            const BlockInfo* __restrict__ bi, long long ntot, short* __restrict__ node_bin,
                            int* __restrict__ table, unsigned mask, unsigned* __restrict__ flag) {
  const int cmax = (1 << kCoinBits) - 1;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ntot;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = node_blk[g];
    const BlockInfo& B = bi[b];
    const double p[3] = {x[3 * g], x[3 * g + 1], x[3 * g + 2]};
    node_bin[g] = node_bin_of(p, B.obb);
    const double delta = coin_delta(B), inv = 1.0 / (4 * kCoinCoarse * delta);
    constexpr double reach = 0.2501 / kCoinCoarse;  // delta in filing cells, with room for the rounding of t
    int c0[3], n[3];
    for (int k = 0; k < 3; k++) {
      const double t = (p[k] - (double)B.bb_lo[k]) * inv + 0.37;  // (a lattice's nodes off the cells' faces)
      c0[k] = min(max((int)floor(t - reach), 0), cmax);
      n[k] = min(max((int)floor(t + reach), 0), cmax) - c0[k] + 1;
    }
    // the (at most eight) cells' first entries all in flight together
    unsigned at[8], step[8];
    int old[8];
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int i = m & 1, j = (m >> 1) & 1, k = m >> 2;
      at[m] = step[m] = 0;
      old[m] = -1;
      if (i < n[0] && j < n[1] && k < n[2]) {
        coin_place(b, c0[0] + i, c0[1] + j, c0[2] + k, mask, at[m], step[m]);
        old[m] = atomicCAS(&table[at[m]], -1, (int)g);
      }
    }
    unsigned found = 0;
#pragma unroll
    for (int m = 0; m < 8; m++)
      for (int probe = 1; old[m] != -1 && !found; probe++) {
        if (coin_close(x, node_blk, p, (int)g, b, old[m], delta)) found = kCoinClose;
        else if (probe == kCoinWalk) found = kCoinCrowded;
        else if (probe % 16 == 0 && *(volatile unsigned*)flag) found = kCoinCrowded;  // (or decided: no more to do)
        if (found) break;
        at[m] = (at[m] + step[m]) & mask;
        old[m] = atomicCAS(&table[at[m]], -1, (int)g);
      }
    if (found) atomicOr(flag, found);
  }
}

// The crowded gate: every node under its own cell (the table is less than half
// full), then against the cells its delta-box touches.
__global__ void k_coin_file(const double* __restrict__ x, const blk_t* __restrict__ node_blk,
                            const BlockInfo* __restrict__ bi, long long ntot, int* __restrict__ table, unsigned mask,
                            unsigned* __restrict__ flag) {
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ntot;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = node_blk[g];
    const double p[3] = {x[3 * g], x[3 * g + 1], x[3 * g + 2]};
    const double delta = coin_delta(bi[b]), inv = 1.0 / (kCoinFine * delta);
    int c[3];
    for (int k = 0; k < 3; k++) c[k] = (int)floor((p[k] - (double)bi[b].bb_lo[k]) * inv + 0.37);
    unsigned at, step;
    coin_place(b, c[0], c[1], c[2], mask, at, step);
    for (int probe = 1;; probe++) {
      const int old = atomicCAS(&table[at], -1, (int)g);
      if (old == -1) break;
      if (coin_close(x, node_blk, p, (int)g, b, old, delta) || probe == kCoinProbes) {
        atomicOr(flag, kCoinClose);
        break;
      }
      if (probe % 16 == 0 && (*(volatile unsigned*)flag & kCoinClose)) break;
      at = (at + step) & mask;
    }
  }
}
__global__ void k_coin_compare(const double* __restrict__ x, const blk_t* __restrict__ node_blk,
                               const BlockInfo* __restrict__ bi, long long ntot, const int* __restrict__ table,
                               unsigned mask, unsigned* __restrict__ flag) {
  if (*(volatile unsigned*)flag & kCoinClose) return;  // decided (and the table may not be complete)
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ntot;
       g += (long long)gridDim.x * blockDim.x) {
    const int b = node_blk[g];
    const double p[3] = {x[3 * g], x[3 * g + 1], x[3 * g + 2]};
    const double delta = coin_delta(bi[b]), inv = 1.0 / (kCoinFine * delta);
    // delta in cells (1 / 2.01), with room for the rounding; a node's box touches two an axis at most
    constexpr double reach = 0.498;
    int c0[3], c1[3];
    for (int k = 0; k < 3; k++) {
      const double t = (p[k] - (double)bi[b].bb_lo[k]) * inv + 0.37;
      c0[k] = (int)floor(t - reach);
      c1[k] = (int)floor(t + reach);
    }
    bool close = false;
    for (int i = c0[0]; i <= c1[0]; i++)
      for (int j = c0[1]; j <= c1[1]; j++)
        for (int k = c0[2]; k <= c1[2]; k++) {
          unsigned at, step;
          coin_place(b, i, j, k, mask, at, step);
          for (int old = table[at]; old != -1 && !close; old = table[at = (at + step) & mask])
            close = coin_close(x, node_blk, p, (int)g, b, old, delta);
        }
    if (close) atomicOr(flag, kCoinClose);
  }
}

// ---------------------------------------------------------------------------
// Per call: donor-list order of every query, then the octree emulation.
// ---------------------------------------------------------------------------
// key = pair | receptor bin | descending node id (the pairs are sorted by
// donor block, so a donor's pairs are consecutive and in list order); sorting
// the queries by it gives every donor's list in the reference's order (gpos =
// position in that sorted order)
__global__ void k_dedup_keys(const int* __restrict__ qnode, long long nq, const int* __restrict__ pair_qoff,
                             int npairs, const short* __restrict__ node_bin, int node_bits,
                             unsigned long long* __restrict__ key, int* __restrict__ val) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
       q += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = npairs - 1;  // the last pair whose first query is <= q
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (pair_qoff[m] <= q) lo = m;
      else hi = m - 1;
    }
    const int g = qnode[q];
    key[q] = ((unsigned long long)lo << (node_bits + 10)) | ((unsigned long long)node_bin[g] << node_bits) |
             ((1ull << node_bits) - 1 - (unsigned long long)g);
    val[q] = (int)q;
  }
}

// the same for the high-order path's receptor points: within a pair the
// donor list holds them in point order (getExtraQueryPoints, highOrder.C:272-319)
__global__ void k_dedup_keys_pts(const int* __restrict__ qpt_local, long long nq, const int* __restrict__ pair_qoff,
                                 int npairs, int point_bits, unsigned long long* __restrict__ key,
                                 int* __restrict__ val) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
       q += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = npairs - 1;
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (pair_qoff[m] <= q) lo = m;
      else hi = m - 1;
    }
    key[q] = ((unsigned long long)lo << point_bits) | (unsigned long long)qpt_local[q];
    val[q] = (int)q;
  }
}

// ---------------------------------------------------------------------------
// Subsets.  Active subset s of a level is DedupSeg S[s], with the box of its
// points, their counts per octant and a cursor per octant; position i of perm
// belongs to active subset seg[i], or to a finished leaf (-1).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void dedup_seg_clear(DedupSeg& g) {
  for (int k = 0; k < 3; k++) {
    g.box[k] = ~0ull;
    g.box[k + 3] = 0ull;
  }
  for (int k = 0; k < 8; k++) g.cnt[k] = g.cur[k] = 0;
}

// the points' bounds into their subsets' boxes: lanes of one subset are
// neighbours, so each run of equal subsets is reduced in the warp first
__device__ __forceinline__ void dedup_box_add(DedupSeg* __restrict__ S, int s, const double p[3]) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int s0 = __shfl_sync(all, s, 0);
  if (__all_sync(all, s == s0)) {  // one subset (or none) in the whole warp
    if (s0 < 0) return;
    for (int k = 0; k < 3; k++) {
      double lo = p[k], hi = p[k];
      for (int o = 16; o > 0; o >>= 1) {
        lo = dmin(lo, __shfl_xor_sync(all, lo, o));
        hi = dmax(hi, __shfl_xor_sync(all, hi, o));
      }
      if (lane == 0) {
        atomicMin(&S[s0].box[k], dkey(lo));
        atomicMax(&S[s0].box[k + 3], dkey(hi));
      }
    }
    return;
  }
  if (s < 0) return;
  for (int k = 0; k < 3; k++) {
    const unsigned long long v = dkey(p[k]);
    if (v < S[s].box[k]) atomicMin(&S[s].box[k], v);  // (a stale bound only costs the atomic)
    if (v > S[s].box[k + 3]) atomicMax(&S[s].box[k + 3], v);
  }
}

// the donors' lists (start, count) as the first level: lists of more than
// kDedupLeaf points are subsets, the others leaves
__global__ void k_dedup_start(const int2* __restrict__ lists, int nlists, DedupSeg* __restrict__ S,
                              int* __restrict__ seg_of_list, int4* __restrict__ leaves, int* __restrict__ cnt) {
  for (int l = threadIdx.x; l < nlists; l += blockDim.x) {
    const int2 L = lists[l];
    seg_of_list[l] = -1;
    if (L.y > kDedupLeaf) {
      const int s = atomicAdd(&cnt[kDedupSegs], 1);
      S[s].start = L.x;
      S[s].len = L.y;
      S[s].depth = 0;
      dedup_seg_clear(S[s]);
      seg_of_list[l] = s;
    } else if (L.y > 0) {
      leaves[atomicAdd(&cnt[kDedupLeaves], 1)] = make_int4(L.x, L.y, 0, 0);
    }
  }
}

// gpos-indexed copies: point, receptor mesh tag, resolution, xtag = self
// (query q is point qnode[q] of x; its receptor block is node_blk[qnode[q]],
// or qrec[q] when node_blk is null); with lists, also every position's place
// in the first level and the subsets' boxes
__global__ void k_dedup_gather(const int* __restrict__ refq, long long n, const int* __restrict__ qnode,
                               const double* __restrict__ qres, const double* __restrict__ x,
                               const blk_t* __restrict__ node_blk, const int* __restrict__ qrec,
                               const BlockInfo* __restrict__ bi, const int2* __restrict__ lists, int nlists,
                               const int* __restrict__ seg_of_list, DedupSeg* __restrict__ S, double* __restrict__ xg,
                               int* __restrict__ mtag, double* __restrict__ rtag, int* __restrict__ itag,
                               int* __restrict__ perm, int* __restrict__ member, int* __restrict__ seg,
                               int* __restrict__ gpos_of) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const long long i = i0 + (threadIdx.x & 31);
    double p[3] = {0.0, 0.0, 0.0};
    int sg = -1;
    if (i < n) {
      const int q = refq[i];
      const int g = qnode[q];
      for (int k = 0; k < 3; k++) xg[3 * i + k] = p[k] = x[3ll * g + k];
      mtag[i] = bi[node_blk ? node_blk[g] : qrec[q]].tag;
      rtag[i] = qres[q];
      itag[i] = (int)i;
      gpos_of[q] = (int)i;
      if (lists) {
        int lo = 0, hi = nlists - 1;  // the last list that starts at or before i
        while (lo < hi) {
          const int m = (lo + hi + 1) >> 1;
          if (lists[m].x <= i) lo = m;
          else hi = m - 1;
        }
        sg = seg_of_list[lo];
        perm[i] = member[i] = (int)i;
        seg[i] = sg;
      }
    }
    if (lists) dedup_box_add(S, sg, p);
  }
}

// octant of every point of an active subset, counted per subset
// (uniqNodesTree: xmid = (xmax + xmin) * 0.5, dx = (xmax - xmin) * 0.5 + TOL,
// iv = floor((x - xmid) / dx) + 1, box = 4 iv0 + 2 iv1 + iv2)
__global__ void k_dedup_octant(long long n, const int* __restrict__ seg, const int* __restrict__ perm,
                               const double* __restrict__ xg, DedupSeg* __restrict__ S,
                               unsigned char* __restrict__ oct, const int* __restrict__ nseg) {
  if (*nseg == 0) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const long long i = i0 + (threadIdx.x & 31);
    const int s = i < n ? seg[i] : -1;
    int key = -1;
    if (s >= 0) {
      const double* p = xg + 3ll * perm[i];
      int b = 0;
      for (int k = 0; k < 3; k++) {
        const double xmin = dkey_inv(S[s].box[k]), xmax = dkey_inv(S[s].box[k + 3]);
        const double mid = (xmax + xmin) * 0.5, dx = (xmax - xmin) * 0.5 + kTol;
        const double xp = p[k] - mid;
        b = 2 * b + min(max((int)floor(xp / dx) + 1, 0), 1);
      }
      oct[i] = (unsigned char)b;
      key = 8 * s + b;
    }
    const unsigned same = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&S[s].cnt[key & 7], __popc(same));
  }
}

// every active subset's children: the next level's subsets, or leaves (child
// of octant o: first position base[o], next-level subset child[o] or -1).  All
// points in one octant: the subset itself is a leaf (icheck).  On the last level
// every child is a leaf.
__global__ void k_dedup_split(DedupSeg* __restrict__ S, DedupSeg* __restrict__ T, int4* __restrict__ leaves,
                              int* __restrict__ cnt, const int* __restrict__ nseg, int* __restrict__ nnext, int last) {
  const int ns = *nseg;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
    DedupSeg& g = S[s];
    int at = g.start;
    bool one = false;
    for (int o = 0; o < 8; o++) one = one || g.cnt[o] == g.len;
    if (one) leaves[atomicAdd(&cnt[kDedupLeaves], 1)] = make_int4(g.start, g.len, g.depth, 0);
    for (int o = 0; o < 8; o++) {
      const int m = g.cnt[o];
      g.base[o] = at;
      g.child[o] = -1;
      if (m > 0 && !one) {
        if (m > kDedupLeaf && !last) {
          const int t = atomicAdd(nnext, 1);
          T[t].start = at;
          T[t].len = m;
          T[t].depth = g.depth + 1;
          dedup_seg_clear(T[t]);
          g.child[o] = t;
        } else {
          leaves[atomicAdd(&cnt[kDedupLeaves], 1)] = make_int4(at, m, g.depth + 1, 0);
        }
      }
      at += m;
    }
  }
}

// every point of an active subset to a place of its child's range (any place:
// the leaves sort), into the leaves' member list when the child is a leaf, and
// the next level's boxes
__global__ void k_dedup_scatter(long long n, const int* __restrict__ seg, const int* __restrict__ perm,
                                const double* __restrict__ xg, DedupSeg* __restrict__ S, DedupSeg* __restrict__ T,
                                const unsigned char* __restrict__ oct, const int* __restrict__ nseg,
                                int* __restrict__ seg2, int* __restrict__ perm2, int* __restrict__ member) {
  if (*nseg == 0) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const long long i = i0 + (threadIdx.x & 31);
    const int s = i < n ? seg[i] : -1;
    const int key = s >= 0 ? 8 * s + oct[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31, lead = __ffs(same) - 1;
    int base = 0;
    if (key >= 0 && lane == lead) base = atomicAdd(&S[s].cur[key & 7], __popc(same));
    base = __shfl_sync(0xffffffffu, base, lead);
    int t = -1;
    double p[3] = {0.0, 0.0, 0.0};
    if (key >= 0) {
      const int o = key & 7;
      const int at = S[s].base[o] + base + __popc(same & ((1u << lane) - 1u));
      const int v = perm[i];
      t = S[s].child[o];
      seg2[at] = t;
      if (t >= 0) {
        perm2[at] = v;
        for (int k = 0; k < 3; k++) p[k] = xg[3ll * v + k];
      } else {
        member[at] = v;
      }
    } else if (i < n) {
      seg2[i] = -1;
    }
    dedup_box_add(T, t, p);
  }
}

// the reference's pairwise loop over one leaf (uniqNodesTree, utils.c:693-713);
// leaf = (start, count, depth): the members (positions) in ascending donor-list
// order, visited in that order after an even number of splits, else reversed.
// A warp per leaf of up to 32 points: lane j holds the j-th point visited, and
// each point is compared with all later ones at once; the merges are made in
// order by lane 0.  Larger leaves (coincident points only) are sorted and
// walked by one lane.
__device__ __forceinline__ void dedup_merge_pair(int p1, int p2, double* __restrict__ rtag, int* __restrict__ itag) {
  if (p1 > p2) {
    rtag[p2] = dmax(rtag[p1], rtag[p2]);
    itag[p1] = itag[p2];
  } else {
    rtag[p1] = dmax(rtag[p1], rtag[p2]);
    itag[p2] = itag[p1];
  }
}

__global__ void k_dedup_leaves(const int4* __restrict__ leaves, const int* __restrict__ nleaves,
                               int* __restrict__ member, const double* __restrict__ xg,
                               const int* __restrict__ mtag, double* rtag, int* itag) {
  const int lane = threadIdx.x & 31, nl = *nleaves;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < nl; l += nw) {
    const int4 L = leaves[l];
    const int n = L.y;
    const bool rev = L.z & 1;
    if (n <= 32) {
      const int mine = lane < n ? member[L.x + lane] : 0x7fffffff;
      int rank = 0;  // the point's place in the order of visits
      for (int j = 0; j < n; j++) {
        const int v = __shfl_sync(0xffffffffu, mine, j);
        rank += rev ? (v > mine) : (v < mine);
      }
      // lane r takes the point of rank r
      int src = lane;
      for (int j = 0; j < n; j++)
        if (__shfl_sync(0xffffffffu, rank, j) == lane) src = j;
      const int v = __shfl_sync(0xffffffffu, mine, src);
      double p0 = 0, p1 = 0, p2 = 0;
      int tag = -1;
      if (lane < n) {
        p0 = xg[3ll * v];
        p1 = xg[3ll * v + 1];
        p2 = xg[3ll * v + 2];
        tag = mtag[v];
      }
      for (int i = 0; i + 1 < n; i++) {
        const double a0 = __shfl_sync(0xffffffffu, p0, i), a1 = __shfl_sync(0xffffffffu, p1, i),
                     a2 = __shfl_sync(0xffffffffu, p2, i);
        const int at = __shfl_sync(0xffffffffu, tag, i), av = __shfl_sync(0xffffffffu, v, i);
        const bool hit = lane > i && lane < n && fabs(a0 - p0) + fabs(a1 - p1) + fabs(a2 - p2) < kTol && at == tag;
        unsigned hits = __ballot_sync(0xffffffffu, hit);
        while (hits) {
          const int j = __ffs(hits) - 1;
          hits &= hits - 1;
          const int bv = __shfl_sync(0xffffffffu, v, j);
          if (lane == 0) dedup_merge_pair(av, bv, rtag, itag);
        }
      }
    } else if (lane == 0) {
      int* m = member + L.x;
      for (int i = 1; i < n; i++) {
        const int v = m[i];
        int j = i - 1;
        for (; j >= 0 && m[j] > v; j--) m[j + 1] = m[j];
        m[j + 1] = v;
      }
      for (int i = 0; i < n; i++) {
        const int p1 = m[rev ? n - 1 - i : i];
        for (int j = i + 1; j < n; j++) {
          const int p2 = m[rev ? n - 1 - j : j];
          if (fabs(xg[3ll * p1] - xg[3ll * p2]) + fabs(xg[3ll * p1 + 1] - xg[3ll * p2 + 1]) +
                      fabs(xg[3ll * p1 + 2] - xg[3ll * p2 + 2]) < kTol &&
              mtag[p1] == mtag[p2])
            dedup_merge_pair(p1, p2, rtag, itag);
        }
      }
    }
  }
}

// per query: xtag (gpos), representative (query id; the one really searched,
// every xtag chain points to lower positions and ends there) and the
// receptor resolution the donor side reports, res_search[xtag[i]]
__global__ void k_dedup_apply(const int* __restrict__ refq, long long n, const int* __restrict__ itag,
                              const double* __restrict__ rtag, double* __restrict__ qres,
                              int* __restrict__ q_xt, int* __restrict__ q_rep, unsigned* __restrict__ err,
                              unsigned long long* __restrict__ counters) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int q = refq[i];
    const int xt = itag[i];
    qres[q] = rtag[xt];
    q_xt[q] = xt;
    int r = (int)i;
    for (int guard = 0; itag[r] != r; guard++) {
      if (guard > (1 << 20) || itag[r] > r) {
        atomicOr(err, kErrBadIndex);
        break;
      }
      r = itag[r];
    }
    q_rep[q] = refq[r];
    if (xt != (int)i) atomicAdd(&counters[7], 1ull);  // merged into another query
  }
}

// ---------------------------------------------------------------------------
// The node-global-id merge (uniquenode_map, search.C:48-74, in the build with
// TIOGA_HAS_NODEGID): in every donor's list (positions in the reference's
// order), the first query with a node id represents all later ones with that
// id and takes their largest resolution.  Positions are sorted stably by id,
// then by donor block, so each (donor, id) run is in position order.
// ---------------------------------------------------------------------------
__global__ void k_gid_keys(const int* __restrict__ refq, long long n, const int* __restrict__ qnode,
                           const int* __restrict__ qdon, const unsigned long long* __restrict__ node_gid,
                           unsigned long long* __restrict__ gkey, int* __restrict__ dkey16, int* __restrict__ pos) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int q = refq[i];
    gkey[i] = node_gid[qnode[q]];
    dkey16[i] = qdon[q];
    pos[i] = (int)i;
  }
}

// sorted index j: head of its (donor, id) run -> j, else 0 (a max-scan then
// gives every entry its run's first index)
__global__ void k_gid_heads(const int* __restrict__ pos, long long n, const unsigned long long* __restrict__ gkey_of_pos,
                            const int* __restrict__ don_of_pos, int* __restrict__ head) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    bool h = j == 0;
    if (!h) {
      const int a = pos[j], b = pos[j - 1];
      h = gkey_of_pos[a] != gkey_of_pos[b] || don_of_pos[a] != don_of_pos[b];
    }
    head[j] = h ? (int)j : 0;
  }
}

// itag[position] = its run's first position; the run's largest resolution at
// that first position (ordered keys, exact)
__global__ void k_gid_apply(const int* __restrict__ pos, const int* __restrict__ first, long long n,
                            int* __restrict__ itag, const double* __restrict__ rtag,
                            unsigned long long* __restrict__ rmax) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x) {
    const int rep = pos[first[j]];
    itag[pos[j]] = rep;
    atomicMax(&rmax[rep], dkey(rtag[pos[j]]));
  }
}

__global__ void k_gather_i32(const int* __restrict__ src, const int* __restrict__ idx, long long n,
                             int* __restrict__ out) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n;
       j += (long long)gridDim.x * blockDim.x)
    out[j] = src[idx[j]];
}

__global__ void k_gid_res(const int* __restrict__ itag, long long n, const unsigned long long* __restrict__ rmax,
                          double* __restrict__ rtag) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    if (itag[i] == (int)i) rtag[i] = dkey_inv(rmax[i]);
}

// after the search: a merged query takes its representative's donor
__global__ void k_dedup_copy(const int* __restrict__ q_rep, long long nq, int* __restrict__ qcell,
                             unsigned char* __restrict__ qtie) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
       q += (long long)gridDim.x * blockDim.x) {
    const int r = q_rep[q];
    if (r != q) {
      qcell[q] = qcell[r];
      qtie[q] = qtie[r];
    }
  }
}

// resetCoincident (bookKeeping.C:572-597): over the records of the donor's
// queries, a cancelled record stays cancelled only if every record sharing
// its xtag is
__global__ void k_reset_coincident_min(const int* __restrict__ interp2rec, const int* __restrict__ q_xt,
                                       long long nq, const unsigned char* __restrict__ it_cancel,
                                       int* __restrict__ ireset) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
       q += (long long)gridDim.x * blockDim.x) {
    const int r = interp2rec[q];
    if (r >= 0) atomicMin(&ireset[q_xt[q]], (int)it_cancel[r]);
  }
}

__global__ void k_reset_coincident_set(const int* __restrict__ interp2rec, const int* __restrict__ q_xt,
                                       long long nq, const int* __restrict__ ireset,
                                       unsigned char* __restrict__ it_cancel) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
       q += (long long)gridDim.x * blockDim.x) {
    const int r = interp2rec[q];
    if (r >= 0 && it_cancel[r] == 1) it_cancel[r] = (unsigned char)ireset[q_xt[q]];
  }
}

}  // namespace tb
