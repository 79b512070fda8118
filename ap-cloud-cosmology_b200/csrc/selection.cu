// Computational-particle selection on the device.
//
// Reference: Octree::select_computational_particles_2to1_3d (octree.cpp:1050-3001), a
// serial breadth-first refinement followed by a serial bottom-up 2:1 balance.  This
// file computes the same cell set in the same output order with level-parallel passes.
//
// Top-down (octree.cpp:1161-1790).  A node is opened when n*h^2 > c and level < depth.
// n and h both shrink with depth, so the opened set is every octree node that passes
// the test.  Each level is one parallel pass over the opened nodes of the level above.
// The child particle ranges come from binary searches in the sorted keys.  The
// reference's temp-node order is breadth-first, octants in Morton order, so the
// opened list built level by level (stable compaction) is in that same order.  The
// temp index of child c of the r-th opened node is 1 + 8r + c.
//
// Bottom-up 2:1 balance (octree.cpp:1793-2718).  At sweep ln every node of level ln
// looks at its six same-level face neighbours.  If the leaf containing a neighbour is
// coarser than ln-1, the leaf and its descendants down to level ln-2 along that
// position are opened.  Requests within a sweep do not interact, so a sweep is one
// parallel pass.  The reference creates those cells in the order of its first
// requester: temp index of the requesting node, then direction, then level.  That
// order is rebuilt exactly by keeping, per requested cell, the minimum of
// (temp index << 8 | direction << 5 | level) and sorting on it.
//
// Output (octree.cpp:2720-3000).  Cells are the unopened children of opened nodes, in
// temp-index order: top-down leaves (Type 0) first, then balance leaves (Type -1).
// Neigh24 is rebuilt from location codes in the reference's direction order
// x+, x-, y+, y-, z+, z-.  A neighbour is one same-or-coarser cell or the 4 finer
// cells on the shared face.
//
// The tree (top-down levels, balance sweeps, numbering of the leaves) is one cooperative
// kernel, select_tree: its phases are separated by the bounded grid barrier (1.2 us) where
// launches with a host read of each level's size took 20-30 us per level and sweep.  The host
// reads the sizes once, sizes the cell arrays and queues the output kernels.
//
// Location code of a cell at level L with Morton prefix P: (1 << 3L) | P.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "apc_internal.cuh"

namespace {

constexpr int kT = 256;

__device__ __forceinline__ int lower_digit(const uint64_t *keys, int lo, int hi, int shift, int d) {
  // first index in [lo, hi) whose digit ((key >> shift) & 7) >= d; digits ascend in range
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if ((int)((keys[mid] >> shift) & 7ull) < d) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ int lower_key(const uint64_t *keys, int n, uint64_t v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (keys[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// particle range [first, first+count) of the cell with location code `code`
__device__ __forceinline__ void cell_range(const uint64_t *keys, int n, int depth, uint64_t code,
                                           int *first, int *count) {
  const int L = code_level(code);
  const uint64_t prefix = code ^ (1ull << (3 * L));
  const int s = 3 * (depth - L);
  const uint64_t lo = prefix << s;
  const uint64_t hi = (s >= 63 && L == 0) ? (1ull << 63) : ((prefix + 1) << s);
  int a = lower_key(keys, n, lo);
  int b = (L == 0) ? n : lower_key(keys, n, hi);
  *first = a;
  *count = b - a;
}

// ------------------------------------------------------------------ balance

__device__ __forceinline__ bool neighbour_code(uint64_t code, int L, int di, int bc, uint64_t *out) {
  const uint64_t prefix = code ^ (1ull << (3 * L));
  long long ix = (long long)compact3(prefix >> 2), iy = (long long)compact3(prefix >> 1),
            iz = (long long)compact3(prefix);
  // direction numbering of the reference's temp links: 0 x+, 1 x-, 2 y-, 3 y+, 4 z+, 5 z-
  switch (di) {
    case 0: ++ix; break;
    case 1: --ix; break;
    case 2: --iy; break;
    case 3: ++iy; break;
    case 4: ++iz; break;
    default: --iz; break;
  }
  const long long side = 1ll << L;
  if (ix < 0 || ix >= side || iy < 0 || iy >= side || iz < 0 || iz >= side) {
    if (bc != 1) return false;
    ix = (ix + side) & (side - 1);
    iy = (iy + side) & (side - 1);
    iz = (iz + side) & (side - 1);
  }
  *out = (1ull << (3 * L)) | (spread3((uint64_t)ix) << 2) | (spread3((uint64_t)iy) << 1) |
         spread3((uint64_t)iz);
  return true;
}

// ------------------------------------------------------------------ the tree

constexpr int kTreeThreads = 512;
constexpr int kTreeWarps = kTreeThreads / 32;
constexpr int kTreeLevels = 24;
constexpr int kReqChunk = 4096;  // requests of a sweep that are ordered together (a power of two)
constexpr int kReqKeys = 4;      // and keys that a thread looks up in each chunk at a time
constexpr int kTreeBlocks = 2;   // blocks per SM, for trees of more than kTreeTwo opened nodes
constexpr int kTreeTwo = 1 << 20;

// what the host reads back: the sizes, and why the kernel stopped early
enum : int { TREE_FULL = 1, TREE_DEEPER = 2 };
struct TreeOut {
  int stop;                 // TREE_* bits: a table was full, the sort was too shallow
  int maxlev;               // level of the last temp node (octree.cpp:1792 ml)
  int n_open_td, n_open;    // opened nodes: top-down, all
  int nc;                   // leaves of top-down opened nodes (Type 0 cells)
};

struct TreeArgs {
  const uint64_t *keys;
  int n, depth, sorted_levels, bc;
  double h0, c;
  uint64_t *hkeys;          // opened-node hash
  int *hvals;
  int hcap;                 // at most hcap / 2 nodes are opened
  uint64_t *rkeys[2];       // balance requests: two tables, used in turn, empty between selections
  unsigned long long *rvals[2];
  int *rlist[2];            // their used slots
  int rcap;
  uint64_t *op_code;
  int *op_base, *op_first, *op_count;
  uint32_t *words[2];       // one bit per child, in child order
  int2 *crange;             // particle range of each child of the level in hand
  uint32_t *leaf;           // one bit per child of every opened node: a leaf
  int *leaf_base;           // leaves before each word
  int *nreq;                // requests of each sweep, zeroed before the launch
  TreeOut *out;
  GridBar *bar;
  int *err;
};

// first index in [lo, hi) whose digit ((key >> shift) & 7) >= d, by a warp: 32 probes a round
__device__ __forceinline__ int warp_lower_digit(const uint64_t *keys, int lo, int hi, int shift, int d, int lane) {
  while (hi - lo > 0) {
    const int step = (hi - lo + 31) / 32;
    const int p = min(lo + lane * step, hi - 1);  // probes ascend, the first is lo
    const bool below = (int)((keys[p] >> shift) & 7ull) < d;
    const int k = __popc(__ballot_sync(0xffffffffu, below));  // a prefix of the lanes is below
    if (k == 0) return lo;
    const int nlo = min(lo + (k - 1) * step, hi - 1) + 1;
    const int nhi = k < 32 ? min(lo + k * step, hi) : hi;
    lo = nlo;
    hi = max(nlo, nhi);
  }
  return lo;
}

// One sweep ln's requests by one (opened node, child) pair: the child, a node of level ln,
// requests the opening of the coarse cells that break 2:1 across its six faces.
__device__ __forceinline__ void request_openings(const TreeArgs &A, int ln, int o, int ch, int tab) {
  const uint64_t pcode = A.op_code[o];
  if (code_level(pcode) != ln - 1) return;
  const uint64_t code = (pcode << 3) | (uint64_t)ch;
  const unsigned long long tidx = (unsigned long long)(A.op_base[o] + ch);
  for (int di = 0; di < 6; ++di) {
    uint64_t nc;
    if (!neighbour_code(code, ln, di, A.bc, &nc)) continue;
    if (ln >= 2 && hash_find(A.hkeys, A.hcap, nc >> 6) >= 0) continue;  // leaf at level >= ln-1
    int lstar = 0;
    for (int l = ln - 3; l >= 0; --l)
      if (hash_find(A.hkeys, A.hcap, nc >> (3 * (ln - l))) >= 0) { lstar = l; break; }
    for (int l = lstar + 1; l <= ln - 2; ++l) {
      const uint64_t target = nc >> (3 * (ln - l));
      const unsigned long long key = (tidx << 8) | ((unsigned long long)di << 5) | (unsigned long long)l;
      bool fresh;
      const int s = hash_insert(A.rkeys[tab], A.rcap, target, &fresh);
      if (s < 0) {
        atomicOr(A.err, DERR_HASH_FULL);
        continue;
      }
      if (fresh) {
        const int q = atomicAdd(&A.nreq[ln], 1);
        if (q < A.rcap / 2) A.rlist[tab][q] = s;
      }
      atomicMin(&A.rvals[tab][s], key);
    }
  }
}

__device__ __forceinline__ void open_node(const TreeArgs &A, int q, uint64_t code, int base, int first, int count) {
  A.op_code[q] = code;
  A.op_base[q] = base;
  A.op_first[q] = first;
  A.op_count[q] = count;
  bool fresh;
  const int s = hash_insert(A.hkeys, A.hcap, code, &fresh);
  if (s < 0) atomicOr(A.err, DERR_HASH_FULL);
  else A.hvals[s] = q;
}

// The cell whose opening a request asks for, from its first requester's key (request_openings):
// the requester is child tidx - 1 of the opened nodes' children in order.
__device__ __forceinline__ uint64_t requested_cell(const TreeArgs &A, int ln, unsigned long long key) {
  const int q = (int)(key >> 8) - 1, di = (int)(key >> 5) & 7, l = (int)key & 31;
  uint64_t nc = 0;
  neighbour_code((A.op_code[q >> 3] << 3) | (uint64_t)(q & 7), ln, di, A.bc, &nc);
  return nc >> (3 * (ln - l));
}

// By the block: the chunk of kReqChunk keys from list entry c0 on, into `sorted` in ascending
// order.  (No part of the loop over the sweeps: inlined, it costs every selection registers.)
__device__ __noinline__ void sort_requests(const int *list, const unsigned long long *vals, int nreq, int c0,
                                           unsigned long long *s_key, unsigned long long *sorted) {
  const int t = threadIdx.x, cn = min(kReqChunk, nreq - c0);
  __syncthreads();
  for (int i = t; i < kReqChunk; i += kTreeThreads)
    s_key[i] = i < cn ? __ldcg(vals + __ldcg(list + c0 + i)) : ~0ull;
  for (int k = 2; k <= kReqChunk; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int e = t; e < kReqChunk / 2; e += kTreeThreads) {
        const int lo = 2 * e - (e & (j - 1)), hi = lo + j;
        const unsigned long long a = s_key[lo], c = s_key[hi];
        if ((a > c) == ((lo & k) == 0)) {
          s_key[lo] = c;
          s_key[hi] = a;
        }
      }
    }
  __syncthreads();
  for (int i = t; i < cn; i += kTreeThreads) sorted[c0 + i] = s_key[i];
}

// By the block: the number of requests below each of a thread's keys, chunk by chunk.  The
// thread's key q is key i + q stride, the block's first i0 + q stride.
__device__ __noinline__ void rank_requests(const unsigned long long *sorted, int nreq, int i0, int stride,
                                           unsigned long long *s_key, unsigned long long (&key)[kReqKeys],
                                           int (&rank)[kReqKeys]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < kReqKeys; ++q) {
    const long long i = i0 + t + (long long)q * stride;
    key[q] = i < nreq ? __ldcg(sorted + i) : 0ull;
    rank[q] = 0;
  }
  for (int c0 = 0; c0 < nreq; c0 += kReqChunk) {
    __syncthreads();
    for (int j = t; j < kReqChunk; j += kTreeThreads) s_key[j] = c0 + j < nreq ? __ldcg(sorted + c0 + j) : ~0ull;
    __syncthreads();
    int at[kReqKeys];
#pragma unroll
    for (int q = 0; q < kReqKeys; ++q) at[q] = 0;
    const int keys = i0 + (long long)stride < nreq ? kReqKeys : 1;  // the same for the whole block
    if (keys == 1) {
#pragma unroll
      for (int step = kReqChunk / 2; step > 0; step >>= 1)
        if (s_key[at[0] + step - 1] < key[0]) at[0] += step;
      rank[0] += at[0] + (s_key[at[0]] < key[0] ? 1 : 0);
      continue;
    }
#pragma unroll
    for (int step = kReqChunk / 2; step > 0; step >>= 1)
#pragma unroll
      for (int q = 0; q < kReqKeys; ++q)
        if (s_key[at[q] + step - 1] < key[q]) at[q] += step;
#pragma unroll
    for (int q = 0; q < kReqKeys; ++q) rank[q] += at[q] + (s_key[at[q]] < key[q] ? 1 : 0);
  }
}

// The opened nodes of the octree (top-down refinement, then the 2:1 balance) in the
// reference's temp-node order, and the numbering of their leaves.  The root is open (the host
// tests it).  Every block takes the same branches: the counts it branches on are read after a
// barrier.  What bounds it is the chain of ~4 barriers and dependent key probes per level.
__global__ void __launch_bounds__(kTreeThreads, kTreeBlocks) select_tree(const __grid_constant__ TreeArgs A) {
  __shared__ int sm[kTreeWarps], off_s[kTreeLevels + 1], s_base[kTreeThreads];
  __shared__ uint32_t s_word[kTreeThreads];
  __shared__ unsigned long long s_key[kReqChunk];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int G = gridDim.x, b = blockIdx.x;
  const int gthreads = G * kTreeThreads, gt = b * kTreeThreads + t;
  const int gwarps = G * kTreeWarps, gwarp = b * kTreeWarps + warp;
  unsigned epoch = 0;
  int stop = 0;

  // the bits of words [0, nwords) before the block's share [w0, w1), and in all
  auto share = [&](const uint32_t *words, int nwords, int &w0, int &w1, int &before, int &total) {
    const int per = (nwords + G - 1) / G;
    w0 = min(nwords, b * per);
    w1 = min(nwords, w0 + per);
    int lo = 0, all = 0;
    for (int w = t; w < nwords; w += kTreeThreads) {
      const int p = __popc(__ldcg(words + w));
      all += p;
      if (w < w0) lo += p;
    }
    before = block_sum_int<kTreeThreads>(lo, sm);
    total = block_sum_int<kTreeThreads>(all, sm);
  };
  auto finish = [&](int maxlev, int n_open_td, int n_open) {
    if (b == 0 && t == 0) {
      A.out->stop = stop;
      A.out->maxlev = maxlev;
      A.out->n_open_td = n_open_td;
      A.out->n_open = n_open;
    }
  };

  if (b == 0) {
    if (t == 0) {
      open_node(A, 0, 1ull, 1, 0, A.n);
      A.words[0][0] = 0u;
    }
  }
  if (t == 0) {
    off_s[0] = 0;
    off_s[1] = 1;
  }
  if (!grid_sync(A.bar, G, epoch, A.err)) return;

  // ---- top-down, level by level ----
  int off = 0, cnt = 1, n_open = 1, maxlev = 0, cur = 0;
  double hchild = A.h0;
  for (int L = 0; L < A.depth && cnt > 0; ++L) {
    // children at level L + 1 need the particles sorted by that many levels of key bits
    if (L + 1 > A.sorted_levels) {
      stop |= TREE_DEEPER;
      break;
    }
    maxlev = L + 1;
    hchild *= 0.5;  // exact: h0 2^-(L + 1)
    const int m8 = 8 * cnt, shift = 3 * (A.depth - L - 1);
    uint32_t *words = A.words[cur];
    const bool deeper = L + 1 < A.depth;
    // particle ranges of the children and the refinement test n h^2 > c (octree.cpp:1165-1183)
    auto opens = [&](int np) {
      double v = 1.0 * np;
      v = __dmul_rn(v, hchild);
      v = __dmul_rn(v, hchild);
      return v > A.c && deeper;
    };
    if (m8 <= gwarps) {
      // few children with long ranges: a warp per child (words zeroed beforehand)
      for (int q = gwarp; q < m8; q += gwarps) {
        const int o = off + (q >> 3), ch = q & 7;
        const int lo = A.op_first[o], hi = lo + A.op_count[o];
        const int a = warp_lower_digit(A.keys, lo, hi, shift, ch, lane);
        const int e = ch == 7 ? hi : warp_lower_digit(A.keys, a, hi, shift, ch + 1, lane);
        if (lane == 0) {
          A.crange[q] = make_int2(a, e - a);
          if (opens(e - a)) atomicOr(words + (q >> 5), 1u << (q & 31));
        }
      }
    } else {
      const int rounds = (m8 + gthreads - 1) / gthreads;
      for (int r = 0; r < rounds; ++r) {
        const int q = r * gthreads + gt;  // a warp's lanes share a word
        const bool act = q < m8;
        int a = 0, hi = 0;
        if (act) {
          const int o = off + (q >> 3);
          const int lo = A.op_first[o];
          hi = lo + A.op_count[o];
          a = lower_digit(A.keys, lo, hi, shift, q & 7);
        }
        const int nxt = __shfl_down_sync(0xffffffffu, a, 1);
        const int np = ((q & 7) == 7 ? hi : nxt) - a;
        const bool f = act && opens(np);
        if (f) A.crange[q] = make_int2(a, np);
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        if (lane == 0 && act) words[q >> 5] = bal;
      }
    }
    if (!grid_sync(A.bar, G, epoch, A.err)) return;
    // the opened children in order: their place is the number of opened children before them
    const int nwords = (m8 + 31) / 32, off_next = off + cnt;
    int w0, w1, before, total;
    share(words, nwords, w0, w1, before, total);
    if (2ll * (off_next + total) > A.hcap) {
      stop |= TREE_FULL;
      break;
    }
    for (int wb = w0; wb < w1; wb += kTreeThreads) {
      const uint32_t word = wb + t < w1 ? __ldcg(words + wb + t) : 0u;
      int sum;
      const int ex = block_scan_int<kTreeThreads>(__popc(word), sm, &sum);
      s_base[t] = before + ex;
      s_word[t] = word;
      __syncthreads();
      const int items = min(kTreeThreads, w1 - wb) * 32;
      for (int i = t; i < items; i += kTreeThreads) {
        const uint32_t wd = s_word[i >> 5];
        if (!((wd >> (i & 31)) & 1u)) continue;
        const int q = wb * 32 + i, o = off + (q >> 3);
        const int at = off_next + s_base[i >> 5] + __popc(wd & ((1u << (i & 31)) - 1u));
        const int2 rg = A.crange[q];
        open_node(A, at, (A.op_code[o] << 3) | (uint64_t)(q & 7), 1 + 8 * at, rg.x, rg.y);
      }
      before += sum;
      __syncthreads();
    }
    cur ^= 1;
    if (8 * total <= gwarps)
      for (int w = gt; w < (8 * total + 31) / 32; w += gthreads) A.words[cur][w] = 0u;
    off = off_next;
    cnt = total;
    n_open = off + cnt;
    if (t == 0 && L + 2 <= kTreeLevels) off_s[L + 2] = n_open;
    if (!grid_sync(A.bar, G, epoch, A.err)) return;
  }
  const int n_open_td = n_open, child_base = 1 + 8 * n_open_td;

  // ---- bottom-up 2:1 balance, sweeps ln = maxlev .. 2 ----
  int tab = 0, dirty[2] = {0, 0};
  for (int ln = maxlev; ln > 1 && !stop; --ln) {
    const int td_a = off_s[ln - 1], ntd = off_s[ln] - td_a, nbal = n_open - n_open_td;
    // the nodes opened by the balance are of all levels: as many as one round holds are taken as
    // they come; beyond it a warp picks those of level ln - 1 among its share, up to 32 of them,
    // and its lanes take four of these at a time (6.6 -> 4.1 ms for 2,000 groups in empty space)
    const bool pick = 8ll * nbal > gthreads;
    const int share_bal = min(32, (nbal + gwarps - 1) / gwarps);
    for (int q = gt; q < 8 * (pick ? ntd : ntd + nbal); q += gthreads) {
      const int r = q >> 3;
      request_openings(A, ln, r < ntd ? td_a + r : n_open_td + (r - ntd), q & 7, tab);
    }
    for (int o0 = share_bal * gwarp; o0 < nbal && pick; o0 += share_bal * gwarps) {
      const bool of_level = lane < share_bal && o0 + lane < nbal && code_level(A.op_code[n_open_td + o0 + lane]) == ln - 1;
      for (unsigned todo = __ballot_sync(0xffffffffu, of_level); todo;) {
        unsigned rest = todo;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < (lane >> 3)) rest &= rest - 1u;
          todo &= todo - 1u;
        }
        if (rest) request_openings(A, ln, n_open_td + o0 + __ffs(rest) - 1, lane & 7, tab);
        __syncwarp();
      }
    }
    if (!grid_sync(A.bar, G, epoch, A.err)) return;
    const int nreq = __ldcg(A.nreq + ln);
    if (nreq == 0) continue;
    if (nreq > A.rcap / 2 || 2ll * (n_open + nreq) > A.hcap) {
      stop |= TREE_FULL;
      break;
    }
    // a request's place is its rank by first requester
    const int *list = A.rlist[tab];
    const unsigned long long *vals = A.rvals[tab];
    auto open_request = [&](int rank, uint64_t code) {
      int f, cn;
      cell_range(A.keys, A.n, A.depth, code, &f, &cn);
      open_node(A, n_open + rank, code, child_base + 8 * (n_open - n_open_td + rank), f, cn);
    };
    if (nreq <= kReqChunk) {
      // few (a percent of the cells at most in the collapse runs): each counts the smaller keys
      const int rounds = (nreq + gthreads - 1) / gthreads;
      for (int r = 0; r < rounds; ++r) {
        if (r * gthreads + b * kTreeThreads >= nreq) continue;  // no request of this block's
        const int i = r * gthreads + gt;
        const int slot = i < nreq ? __ldcg(list + i) : 0;
        const unsigned long long key = i < nreq ? __ldcg(vals + slot) : 0ull;
        int rank = 0;
        for (int j0 = 0; j0 < nreq; j0 += kTreeThreads) {
          __syncthreads();
          if (j0 + t < nreq) s_key[t] = __ldcg(vals + __ldcg(list + j0 + t));
          __syncthreads();
          const int jn = min(kTreeThreads, nreq - j0);
          for (int j = 0; j < jn; ++j) rank += s_key[j] < key ? 1 : 0;
        }
        if (i < nreq) open_request(rank, A.rkeys[tab][slot]);
      }
    } else {
      // many (clumps or walls in empty space): chunks are sorted, and each request adds up its
      // places in all of them.  Counting alone grows with the square of the requests: 20,000
      // groups of 20 particles, 10^5 requests a sweep, took 129 ms to select, 28 ms this way.
      // At the line one chunk's sort and the count cost about the same.
      unsigned long long *sorted = reinterpret_cast<unsigned long long *>(A.crange);  // not used past the levels
      for (int c0 = b * kReqChunk; c0 < nreq; c0 += G * kReqChunk) sort_requests(list, vals, nreq, c0, s_key, sorted);
      if (!grid_sync(A.bar, G, epoch, A.err)) return;
      for (long long i0 = b * kTreeThreads; i0 < nreq; i0 += (long long)kReqKeys * gthreads) {
        unsigned long long key[kReqKeys];
        int rank[kReqKeys];
        rank_requests(sorted, nreq, (int)i0, gthreads, s_key, key, rank);
        for (int q = 0; q < kReqKeys; ++q)
          if (i0 + t + (long long)q * gthreads < nreq) open_request(rank[q], requested_cell(A, ln, key[q]));
      }
    }
    n_open += nreq;
    dirty[tab] = nreq;
    // the other table's entries of the sweep before are no longer read: empty it
    tab ^= 1;
    for (int i = gt; i < dirty[tab]; i += gthreads) {
      const int slot = __ldcg(A.rlist[tab] + i);
      A.rkeys[tab][slot] = 0ull;
      A.rvals[tab][slot] = ~0ull;
    }
    dirty[tab] = 0;
    if (!grid_sync(A.bar, G, epoch, A.err)) return;
  }
  tab ^= 1;  // the last table used
  for (int i = gt; i < dirty[tab] && !stop; i += gthreads) {
    const int slot = __ldcg(A.rlist[tab] + i);
    A.rkeys[tab][slot] = 0ull;
    A.rvals[tab][slot] = ~0ull;
  }
  if (stop) {
    finish(maxlev, n_open_td, n_open);
    return;
  }

  // ---- the leaves: unopened children of opened nodes ----
  const int m8 = 8 * n_open, nwords = (m8 + 31) / 32;
  for (int r = 0; r < (m8 + gthreads - 1) / gthreads; ++r) {
    const int q = r * gthreads + gt;
    const bool f = q < m8 && hash_find(A.hkeys, A.hcap, (A.op_code[q >> 3] << 3) | (uint64_t)(q & 7)) < 0;
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (lane == 0 && q < m8) A.leaf[q >> 5] = bal;
  }
  if (!grid_sync(A.bar, G, epoch, A.err)) return;
  int w0, w1, before, total;
  share(A.leaf, nwords, w0, w1, before, total);
  const int split = 8 * n_open_td;  // children of top-down opened nodes
  if (b == 0 && t == 0 && (split >> 5) >= nwords) A.out->nc = total;
  for (int wb = w0; wb < w1; wb += kTreeThreads) {
    const uint32_t word = wb + t < w1 ? __ldcg(A.leaf + wb + t) : 0u;
    int sum;
    const int ex = block_scan_int<kTreeThreads>(__popc(word), sm, &sum);
    if (wb + t < w1) {
      A.leaf_base[wb + t] = before + ex;
      if (wb + t == split >> 5) A.out->nc = before + ex + __popc(word & ((1u << (split & 31)) - 1u));
    }
    before += sum;
  }
  finish(maxlev, n_open_td, n_open);
}

// ------------------------------------------------------------------ output

// cell centre by replaying the reference's parent-centre +- h/4 recursion from the root
// (octree.cpp:1233-1235 and siblings), so that every rounding step is the same
__global__ void leaf_emit(int n_open, int n_open_td, const uint32_t *__restrict__ leaf,
                          const int *__restrict__ leaf_base, const uint64_t *__restrict__ op_code,
                          const int *__restrict__ op_first, const int *__restrict__ op_count,
                          const uint64_t *__restrict__ keys, int depth, double cx0,
                          double cy0, double cz0, double hx0, double hy0, double hz0, double h0,
                          double *cx, double *cy, double *cz, double *ch, int *cfirst, int *ccount,
                          int *ctype, uint64_t *ccode, uint64_t *lkeys, int *lvals, int lcap,
                          int *err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  // the child's first particle, searched in its parent's range; its end is the next child's
  const bool in = t < 8 * n_open;
  const uint64_t code = in ? (op_code[t >> 3] << 3) | (uint64_t)(t & 7) : 8ull;
  const int L = code_level(code);
  int f = 0, end = 0;
  if (in) {
    f = op_first[t >> 3];
    end = f + op_count[t >> 3];
    f = lower_digit(keys, f, end, 3 * (depth - L), t & 7);
  }
  const int next = __shfl_down_sync(0xffffffffu, f, 1);
  if (!in) return;
  const uint32_t word = leaf[t >> 5];
  if (!((word >> (t & 31)) & 1u)) return;
  const int i = leaf_base[t >> 5] + __popc(word & ((1u << (t & 31)) - 1u));
  const int c = ((t & 7) == 7 ? end : next) - f;
  double x = cx0, y = cy0, z = cz0;
  for (int l = 0; l < L; ++l) {
    const unsigned dgt = (unsigned)((code >> (3 * (L - 1 - l))) & 7ull);
    const double qx = 0.25 * ldexp(hx0, -l), qy = 0.25 * ldexp(hy0, -l), qz = 0.25 * ldexp(hz0, -l);
    x = (dgt & 4) ? __dadd_rn(x, qx) : __dsub_rn(x, qx);
    y = (dgt & 2) ? __dadd_rn(y, qy) : __dsub_rn(y, qy);
    z = (dgt & 1) ? __dadd_rn(z, qz) : __dsub_rn(z, qz);
  }
  cx[i] = x;
  cy[i] = y;
  cz[i] = z;
  ch[i] = ldexp(h0, -L);
  cfirst[i] = f;
  ccount[i] = c;
  ctype[i] = (t >> 3) < n_open_td ? 0 : -1;
  ccode[i] = code;
  bool fresh;
  int s = hash_insert(lkeys, lcap, code, &fresh);
  if (s < 0) atomicOr(err, DERR_HASH_FULL);
  else lvals[s] = i;
}

// Neigh24 of every cell (octree.cpp:2764-2975): direction order x+, x-, y+, y-, z+, z-;
// a finer neighbour contributes the 4 cells on the shared face in the reference's order
__global__ void neigh24_build(int m, int bc, const uint64_t *__restrict__ ccode,
                              const uint64_t *__restrict__ hkeys, int hcap,
                              const uint64_t *__restrict__ lkeys, const int *__restrict__ lvals,
                              int lcap, int *nb24, int *nnb, int *err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint64_t code = ccode[i];
  const int L = code_level(code);
  const int order[6] = {0, 1, 3, 2, 4, 5};
  // faces of a finer neighbour adjacent to this cell, indexed by link direction
  const int quad[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {2, 3, 6, 7}, {0, 1, 4, 5}, {0, 2, 4, 6}, {1, 3, 5, 7}};
  int k = 0;
  for (int dd = 0; dd < 6; ++dd) {
    const int di = order[dd];
    uint64_t nc;
    if (!neighbour_code(code, L, di, bc, &nc)) {
      atomicOr(err, DERR_NEIGH);  // non-periodic boundary cells are not produced here
      continue;
    }
    const bool exists = (L == 0) || hash_find(hkeys, hcap, nc >> 3) >= 0;
    if (exists) {
      int s = hash_find(lkeys, lcap, nc);
      if (s >= 0) {
        nb24[24 * (size_t)i + k++] = lvals[s];
      } else {
        for (int a = 0; a < 4; ++a) {
          int s2 = hash_find(lkeys, lcap, (nc << 3) | (uint64_t)quad[di][a]);
          if (s2 < 0) { atomicOr(err, DERR_NEIGH); continue; }
          nb24[24 * (size_t)i + k++] = lvals[s2];
        }
      }
    } else {
      int s = hash_find(lkeys, lcap, nc >> 3);
      if (s < 0) { atomicOr(err, DERR_NEIGH); continue; }
      nb24[24 * (size_t)i + k++] = lvals[s];
    }
  }
  nnb[i] = k;
}

int next_pow2(long long v) {
  long long p = 1;
  while (p < v) p <<= 1;
  return (int)std::min<long long>(p, 1ll << 30);
}

int grid_for(long long n) { return (int)std::max<long long>(1, (n + kT - 1) / kT); }

}  // namespace

static int ensure_hash(apc_context *c, uint64_t **keys, void **vals, size_t val_size, int *cap, int want) {
  if (want > *cap) {
    *cap = 0;  // until both are there
    apc_free(c, *keys);
    apc_free(c, *vals);
    *keys = nullptr;
    *vals = nullptr;
    APC_TRY(apc_alloc(c, (void **)keys, sizeof(uint64_t) * (size_t)want));
    APC_TRY(apc_alloc(c, vals, val_size * (size_t)want));
    *cap = want;
  }
  return APC_OK;
}

// The selection's buffers for tables of `want` slots.  The request tables hold one entry per
// coarse cell to be opened, a small part of the opened nodes.
static int ensure_tree(apc_context *c, int want) {
  if (!c->tree_out)
    APC_TRY(apc_alloc(c, (void **)&c->tree_out, sizeof(TreeOut) + sizeof(GridBar) + kTreeLevels * sizeof(int)));
  if (want <= c->hcap) return APC_OK;
  // hcap stands for every table below: none until the last of them is there, so that the call
  // after a failed allocation allocates what is missing
  int hash_cap = c->hcap;
  c->hcap = 0;
  c->r_dirty = true;
  APC_TRY(ensure_hash(c, &c->h_keys, (void **)&c->h_vals, sizeof(int), &hash_cap, want));
  const size_t open = (size_t)want / 2, rcap = std::max<size_t>(1 << 16, (size_t)want / 4);
  APC_TRY(apc_ensure(c, &c->op_code, open));
  APC_TRY(apc_ensure(c, &c->op_base, open));
  APC_TRY(apc_ensure(c, &c->op_first, open));
  APC_TRY(apc_ensure(c, &c->op_count, open));
  APC_TRY(apc_ensure(c, &c->r_keys, 2 * rcap));
  APC_TRY(apc_ensure(c, &c->r_vals, 2 * rcap));
  APC_TRY(apc_ensure(c, &c->r_list, rcap));
  APC_TRY(apc_ensure(c, &c->child_words, 3 * (open / 4)));
  APC_TRY(apc_ensure(c, &c->leaf_base, open / 4));
  APC_TRY(apc_ensure(c, &c->child_range, 8 * open));
  c->rcap = (int)rcap;
  c->hcap = hash_cap;
  return APC_OK;
}

// One attempt at the whole selection with the current table capacities.
static int select_once(apc_context *c, int *hash_full) {
  const int n = c->n, D = c->cfg.depth;
  const double cc = c->cfg.gfd_c;
  *hash_full = 0;

  // ---- level 0 (octree.cpp:1114-1160, 1165-1183) ----
  double temp = 1.0 * n;
  temp = temp * c->h0;
  temp = temp * c->h0;
  if (!(n > 0 && temp > cc && 0 < D)) {
    // the root is the only cell (octree.cpp:1785-1788 leaf[0] = 1)
    int derr = 0;
    APC_TRY(apc_read_errors(c, &derr));
    if (derr & DERR_NOT_FINITE) {
      c->err = "non-finite particle coordinates";
      return APC_ERR_NOT_FINITE;
    }
    c->nc = 1;
    c->nv = 0;
    c->nb = 0;
    return APC_ERR_UNSUPPORTED;
  }
  TreeArgs A{};
  A.keys = c->keys;
  A.n = n;
  A.depth = D;
  A.sorted_levels = c->sorted_levels;
  A.bc = c->cfg.bc;
  A.h0 = c->h0;
  A.c = cc;
  A.hkeys = c->h_keys;
  A.hvals = c->h_vals;
  A.hcap = c->hcap;
  for (int k = 0; k < 2; ++k) {
    A.rkeys[k] = c->r_keys + (size_t)k * c->rcap;
    A.rvals[k] = (unsigned long long *)c->r_vals + (size_t)k * c->rcap;
    A.rlist[k] = c->r_list + (size_t)k * (c->rcap / 2);
  }
  A.rcap = c->rcap;
  A.op_code = c->op_code;
  A.op_base = c->op_base;
  A.op_first = c->op_first;
  A.op_count = c->op_count;
  const size_t nw = (size_t)c->hcap / 8;  // words for the children of hcap / 2 nodes
  A.words[0] = c->child_words;
  A.words[1] = c->child_words + nw;
  A.leaf = c->child_words + 2 * nw;
  A.leaf_base = c->leaf_base;
  A.crange = (int2 *)c->child_range;
  A.out = (TreeOut *)c->tree_out;
  A.bar = (GridBar *)(c->tree_out + sizeof(TreeOut));
  A.nreq = (int *)(c->tree_out + sizeof(TreeOut) + sizeof(GridBar));
  A.err = c->d_err;
  if (c->r_dirty) {
    APC_CUDA_TRY(c, cudaMemsetAsync(c->r_keys, 0, sizeof(uint64_t) * 2 * c->rcap, c->s));
    APC_CUDA_TRY(c, cudaMemsetAsync(c->r_vals, 0xff, sizeof(uint64_t) * 2 * c->rcap, c->s));
  }
  APC_CUDA_TRY(c, cudaMemsetAsync(c->tree_out, 0, sizeof(TreeOut) + sizeof(GridBar) + kTreeLevels * sizeof(int), c->s));
  APC_CUDA_TRY(c, cudaMemsetAsync(c->h_keys, 0, sizeof(uint64_t) * c->hcap, c->s));
  // a block for every 2048 particles (about as many children of opened nodes as threads), or for
  // every 256 nodes that the last selection or attempt opened: groups in empty space open more
  // nodes than they have particles (2,000 groups of 64: 4.1 ms by particles, 3.3 ms by nodes).
  // Two blocks per SM where the probes miss L2 anyway: at 2.5M nodes 16.8 and 15.7 ms, at 0.3M
  // 3.3 and 3.5.
  const int sms = apc_sm_count(c);
  const int blocks = c->open_hint > kTreeTwo
                         ? kTreeBlocks * sms
                         : std::max(1, std::min(sms, std::max(n / 2048, c->open_hint / 256)));
  void *args[] = {&A};
  APC_CUDA_TRY(c, cudaLaunchCooperativeKernel((const void *)select_tree, dim3(blocks), dim3(kTreeThreads), args, 0,
                                              c->s));
  apc_count_launch(c);
  // the sizes and the error flags in one round trip (pinned words 20 ..)
  static_assert(sizeof(TreeOut) <= 20 * sizeof(int), "the pinned words reserved for it");
  APC_CUDA_TRY(c, cudaMemcpyAsync(c->h_pinned + 20, c->tree_out, sizeof(TreeOut), cudaMemcpyDeviceToHost, c->s));
  APC_CUDA_TRY(c, cudaMemcpyAsync(c->h_pinned + 1, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->s));
  c->r_dirty = true;  // until the kernel is known to have emptied the request tables
  APC_CUDA_TRY(c, apc_stream_wait(c));
  TreeOut T;
  memcpy(&T, c->h_pinned + 20, sizeof(T));
  int derr = c->h_pinned[1];
  if (derr & DERR_SORT) {
    c->err = "radix sort: a tile's look-back wait ran past its bound";
    return APC_ERR_TIMEOUT;
  }
  if (derr & DERR_NOT_FINITE) {
    c->err = "non-finite particle coordinates";
    return APC_ERR_NOT_FINITE;
  }
  if (derr & DERR_KRYLOV) {
    c->err = "selection kernel grid barrier timed out";
    return APC_ERR_TIMEOUT;
  }
  c->open_hint = T.n_open;
  if (T.stop & TREE_DEEPER) return APC_RETRY_FULL_SORT;
  if ((T.stop & TREE_FULL) || (derr & DERR_HASH_FULL)) {
    *hash_full = 1;
    return APC_OK;
  }
  c->r_dirty = false;
  const int n_open = T.n_open, n_open_td = T.n_open_td;
  c->n_open_td = n_open_td;
  c->n_open = n_open;
  c->levels_hint = T.maxlev;

  // ---- output cells: of the 8 children of each opened node all but the other opened nodes ----
  const int M = 7 * n_open + 1;
  c->nc = T.nc;
  c->nv = M - T.nc;
  c->nb = 0;
  // capacities for cells
  const size_t mc = (size_t)M + 1;
  APC_TRY(apc_ensure(c, &c->cx, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->cy, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->cz, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->ch, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->cfirst, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->ccount, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->ctype, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->ccode, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->nnb, mc, nullptr));
  APC_TRY(apc_ensure(c, &c->nb24, 24 * mc, nullptr));
  const int want_l = next_pow2(2ll * M + 1024);
  APC_TRY(ensure_hash(c, &c->l_keys, (void **)&c->l_vals, sizeof(int), &c->lcap, want_l));
  APC_CUDA_TRY(c, cudaMemsetAsync(c->l_keys, 0, sizeof(uint64_t) * c->lcap, c->s));
  leaf_emit<<<grid_for(8ll * n_open), kT, 0, c->s>>>(n_open, n_open_td, A.leaf, A.leaf_base, c->op_code, c->op_first,
                                                     c->op_count, c->keys, D, c->cx0, c->cy0, c->cz0, c->hx0, c->hy0,
                                                     c->hz0, c->h0, c->cx, c->cy, c->cz, c->ch, c->cfirst, c->ccount,
                                                     c->ctype, c->ccode, c->l_keys, c->l_vals, c->lcap, c->d_err);
  neigh24_build<<<grid_for(M), kT, 0, c->s>>>(M, c->cfg.bc, c->ccode, c->h_keys, c->hcap, c->l_keys,
                                               c->l_vals, c->lcap, c->nb24, c->nnb, c->d_err);
  apc_count_launch(c, 2);
  APC_CUDA_TRY(c, cudaGetLastError());
  APC_CUDA_TRY(c, cudaEventRecord(c->ev[1], c->s));
  APC_TRY(apc_read_errors(c, &derr));
  if (derr & DERR_HASH_FULL) { *hash_full = 1; return APC_OK; }
  if (derr & DERR_NEIGH) {
    c->err = c->cfg.bc == 1 ? "2:1 face neighbour missing in the selected cell set"
                             : "non-periodic boundary cells are not supported";
    return c->cfg.bc == 1 ? APC_ERR_CUDA : APC_ERR_UNSUPPORTED;
  }
  return APC_OK;
}

int apc_selection(apc_context *c) {
  // hash capacities: opened nodes are ~1/7 of the cells; start generously and double
  // on overflow (the device reports a full table instead of probing without bound)
  int want_h = next_pow2(std::max<long long>(1 << 16, (long long)c->n / 2));
  for (int attempt = 0; attempt < 8; ++attempt) {
    APC_TRY(ensure_tree(c, want_h));
    if (attempt > 0) APC_CUDA_TRY(c, cudaMemsetAsync(c->d_err, 0, sizeof(int), c->s));
    int full = 0;
    int rc = select_once(c, &full);
    if (rc != APC_OK) return rc;
    if (!full) {
      // temp-node budget of the reference (mover.cpp:20,36-41, octree.cpp:1781-1782):
      // the run fails when 1 + 8 * opened + 8 exceeds the budget, which doubles while
      // below the cap
      if (c->cfg.nmax_cap > 0 && c->n_open > 0) {
        const long long need = 1ll + 8ll * c->n_open + 8;
        int ok = 0;
        while (!ok && c->maxnc_state < c->cfg.nmax_cap) {
          if (need <= c->maxnc_state) ok = 1;
          else c->maxnc_state *= 2;
        }
        if (!ok) {
          c->err = "selection needs more temp nodes than the budget cap allows";
          return APC_ERR_NMAX;
        }
      }
      return APC_OK;
    }
    want_h = 2 * c->hcap;
  }
  c->err = "selection hash tables kept overflowing";
  return APC_ERR_OUT_OF_MEMORY;
}
