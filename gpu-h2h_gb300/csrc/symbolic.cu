// symbolic.cu -- the elimination order and the upper neighbours X(v)\{v} of
// every vertex, without weights: the same eliminations as contract.cu's list
// kernels (makeCHPerHeight_2 / makeCHPerHeight_D_2, kernel_functions.cu:
// 309-553, and TDInCPU / CHUsingHeap_2, Traditional_H2H.cu:6-118, :216-351),
// on neighbour sets.
//
// Which vertex is eliminated next depends on degrees and heights alone, never
// on weights, and a list's order and weights reach no later pick.  So a cell
// keeps, for each of its alive members (candidates and the boundary that
// stays), the set of its neighbours inside the cell as a bit row over the
// members in id order, and what the reference's list lengths count besides:
// entries outside the cell, repeated entries of parallel arcs, the junk
// prefix a list keeps when every valid entry vanished (kernel_functions.cu:
// 353-360, :381-388).  Eliminating v is row(u) |= row(v) for every u in
// row(v), minus u and v; the degree is a population count.  An elimination
// that rebuilds weighted lists took 10-32 us (merge walks of dependent loads
// and a grid barrier); on bit rows in shared memory it is a block argmin and
// a few word operations per neighbour.  The weights are computed afterwards,
// for all vertices, over the blocks of the finished tree (fill_blocks.cu).
// On one GB300, against the list kernels: partition levels 23 -> 2.9 ms and
// global order 18.8 -> 2.8 ms (1.8 us a pick) on a 264k-vertex road graph, 81
// -> 8.0 and 45.9 -> 6.7 ms on a 1M-vertex one, where they also made the
// weights (1.5 and 4.6 ms here); a rebuild after new weights repeats no
// elimination (16 graphs: 27 -> 2.5 ms).  Bound: the chain of picks; a pick is
// an argmin over the row groups, two or three barriers and one pass over the
// neighbours' rows.
//
// One thread-block cluster per cell; member l's row, counters and key belong
// to CTA l mod CS.  Per elimination: every CTA's best key (degree + height,
// degree, id -- packed, members being numbered in id order) goes to all CTAs
// through distributed shared memory, one cluster barrier, then each CTA copies
// v's row from its owner and updates the rows it owns, a warp per row.
//
// A cell whose rows outgrow a cluster's shared memory keeps them in global
// memory (L2) and, where the launch has few enough cells, takes up to 128 CTAs
// that meet at a counter in global memory instead of a cluster barrier (kGrid,
// a cooperative launch; every wait is bounded).  Its picks are bound by the
// neighbours' rows, of which a lane has eight words in flight: the global order of a
// 6.26M-vertex graph (7,801 members) 141 ms on one cluster, 91 on 128 CTAs a
// word at a time, 38 now; of a 3.6M-vertex one (5,940) 68, 50 and 28 ms.
//
// Rules kept from the reference: a cell's first pick uses the stale keys
// (input degree, height 0), later picks live ones (kernel_functions.cu:462-476);
// a neighbour's height becomes max(height, HeightNow + 1); the global order
// starts with live keys that still count repeated entries, then drops them
// (unordered_map::emplace).
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "graph.h"

namespace cg = cooperative_groups;

namespace gh {

namespace {

constexpr int kErrOverflow = 1;  // a list outgrew its capacity
constexpr int kErrEmpty = 2;     // eliminated a vertex without neighbours
constexpr int kErrTimeout = 4;   // a grid barrier wait ran out
constexpr int kErrPick = 5;      // no candidate left to pick, or a vertex outside its cell
constexpr int kErrPool = 6;      // the list pool is full

constexpr int kIdxBits = 14, kDegBits = 22, kSumBits = 28;  // a key: degree + height, degree, member
constexpr int kMaxMembers = 1 << kIdxBits;
constexpr int kMaxGroups = 64;
constexpr unsigned long long kNoKey = ~0ull;

struct SymCell {
  int start, count, size;       // candidates in elim; members
  int64_t mem, out;             // members; where the ones that stay go (a run of the parent's members)
  int obase;                    // that run's start within the parent's members
};

struct SymArgs {
  const SymCell *cells;
  int *pool;          // lists, each written once and taken from the pool's end
  int64_t *slot_off;  // where a vertex's list is
  int *lsize, *ljunk, *extra, *height, *elim, *members, *err;
  const int *cap, *deg0, *adj_off, *adj_v;
  unsigned *grows;  // rows in global memory (kGlobal)
  unsigned long long *pool_next;
  int64_t pool_size;
  int smax, npow, heap;
  // kGrid: CTAs per cell, their best keys [cell][2][cs], arrivals per cell
  int cs;
  unsigned long long *best;
  unsigned *arrived;
  long long spin_limit;
};

__device__ __forceinline__ unsigned long long pack_key(int deg, int height, int l) {
  return ((unsigned long long)(deg + height) << (kIdxBits + kDegBits)) | ((unsigned long long)deg << kIdxBits) |
         (unsigned)l;
}

__device__ __forceinline__ int find_id(const int *ids, int n, int x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ids[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo < n && ids[lo] == x ? lo : -1;
}

__device__ __forceinline__ unsigned long long warp_min(unsigned long long k) {
  const unsigned hi = __reduce_min_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned lo = __reduce_min_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : ~0u);
  return ((unsigned long long)hi << 32) | lo;
}

// All cs CTAs of a cell meet; `target` arrivals end the wait.  Writes before it
// are seen by all after it.  False once a wait has run out (A.err is set, and
// every CTA of the launch gives up at its next barrier).
__device__ bool grid_meet(unsigned *arrived, unsigned target, const SymArgs &A, int *s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived, 1);
    int ok = 1;
    const long long t0 = clock64();
    unsigned seen;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
      if (seen >= target) break;
      if (*(volatile int *)A.err == kErrTimeout || clock64() - t0 > A.spin_limit) {
        atomicCAS(A.err, 0, kErrTimeout);
        ok = 0;
        break;
      }
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

template <bool kGlobal, bool kGrid>
__global__ void __launch_bounds__(512, 2) symbolic_kernel(SymArgs A) {
  static_assert(kGlobal || !kGrid, "a grid's rows are in global memory");
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_gmin[2][kMaxGroups];  // best key of every group of rows
  __shared__ unsigned long long s_best[2][16];          // best key of every CTA
  cg::cluster_group cluster = cg::this_cluster();
  const int CS = kGrid ? A.cs : (int)cluster.num_blocks();
  const int rank = kGrid ? (int)(blockIdx.x % CS) : (int)cluster.block_rank();
  const int ci = (int)(blockIdx.x / CS);
  __shared__ int s_ok;
  unsigned meets = 0;
  const SymCell c = A.cells[ci];
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nthr >> 5;
  const int S = c.size, k = c.count, W = (S + 31) >> 5;
  if (S == 0) return;  // uniform across the cluster
  const int csh = 31 - __clz(CS);  // clusters are powers of two
  const int ownmax = (A.smax + CS - 1) >> csh, Wm = ((A.smax + 31) >> 5) | 1;  // odd row stride: no bank conflicts
  const int nown = (S - rank + CS - 1) >> csh;
  unsigned long long *key = (unsigned long long *)smem;
  int *ids = (int *)(key + ownmax);
  int *vc = ids + A.npow;   // neighbours inside the cell
  int *outc = vc + ownmax;  // entries outside it
  int *ext = outc + ownmax; // repeated entries
  int *junk = ext + ownmax;
  int *hgt = junk + ownmax;
  int *cap = hgt + ownmax;  // list capacity (partition cells)
  int *map = cap + ownmax;  // place in id order of every entry of the members' array; then the rank of the ones that stay
  unsigned *rowv = (unsigned *)(map + A.smax);
  unsigned *cand = rowv + Wm;
  unsigned *srows = cand + Wm;
  unsigned *const grows = kGlobal ? A.grows + (int64_t)ci * A.smax * Wm : nullptr;
  auto own_row = [&](int r) -> unsigned * {
    return kGlobal ? grows + (int64_t)(r * CS + rank) * Wm : srows + (int64_t)r * Wm;
  };
  // ---- members in id order
  int np2 = 1;
  while (np2 < S) np2 <<= 1;
  for (int i = tid; i < np2; i += nthr) ids[i] = i < S ? A.members[c.mem + i] : INT_MAX;
  for (int i = tid; i < W; i += nthr) cand[i] = 0;
  __syncthreads();
  for (int kk = 2; kk <= np2; kk <<= 1)
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < np2 >> 1; t += nthr) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), p = i | j;
        const int x = ids[i], y = ids[p];
        if ((x > y) == ((i & kk) == 0)) {
          ids[i] = y;
          ids[p] = x;
        }
      }
      __syncthreads();
    }
  for (int i = tid; i < S; i += nthr) map[i] = find_id(ids, S, A.members[c.mem + i]);
  for (int i = tid; i < k; i += nthr) {
    const int l = find_id(ids, S, A.elim[c.start + i]);
    if (l >= 0) atomicOr(cand + (l >> 5), 1u << (l & 31));
    else atomicCAS(A.err, 0, kErrPick);
  }
  __syncthreads();
  // ---- rows and counters of the owned members, a warp per member
  for (int r = wid; r < nown; r += nw) {
    const int l = r * CS + rank, u = ids[l];
    unsigned *row = own_row(r);
    for (int w = lane; w < W; w += 32) row[w] = 0;
    __syncwarp();
    const int64_t off = A.slot_off[u];
    const int n = A.lsize[u];
    const int *list = A.pool + off;
    // an entry is a place in the members' array, or ~id of a vertex that was
    // outside the cell below
    int out = 0;
#pragma unroll 4
    for (int e = lane; e < n; e += 32) {
      const int y = __ldcg(list + e);
      const int x = y < 0 ? find_id(ids, S, ~y) : y < S ? map[y] : -1;
      if (x >= 0) atomicOr(row + (x >> 5), 1u << (x & 31));
      else out++;
    }
    out = __reduce_add_sync(0xffffffffu, out);
    if (lane == 0) {
      const int ex = A.extra[u], J = A.ljunk[u], h = A.height[u], in = n - out;
      vc[r] = in;
      outc[r] = out;
      hgt[r] = h;
      cap[r] = A.heap ? INT_MAX : A.cap[u];
      ext[r] = A.heap ? 0 : ex;
      junk[r] = A.heap ? 0 : J;
      unsigned long long kk = kNoKey;
      if ((cand[l >> 5] >> (l & 31)) & 1u) kk = A.heap ? pack_key(n + ex, h, l) : pack_key(A.deg0[u], 0, l);
      key[r] = kk;
    }
  }
  __syncthreads();
  if (kGrid) {
    if (!grid_meet(A.arrived + ci, ++meets * CS, A, &s_ok)) return;
  } else if (CS > 1) {
    cluster.sync();
  }
  // Row r belongs to group r mod G, a lane of the group's warp (neighbours
  // have close ids, so they spread over the groups).  Each group's best key is
  // kept, so a pick looks at the groups and an update at the groups it hits.
  // Two ways through v's neighbours.  Few of them: a group's warp takes its
  // rows one at a time, a lane per word.  Many: T lanes take a row, 32 / T rows
  // at once, so the cost is the rows' words and not their number, and every
  // group's best key is taken anew.  The second way pays from about dense_deg
  // neighbours (60 cycles a row against 10 a word).
  const int G = max(nw, (nown + 31) >> 5);
  for (int g = tid; g < 2 * kMaxGroups; g += nthr) s_gmin[g / kMaxGroups][g % kMaxGroups] = kNoKey;
  __syncthreads();
  auto regroup = [&](int buf) {  // every group's best key
    for (int g = wid; g < G; g += nw) {
      const int r = lane * G + g;
      const unsigned long long best = warp_min(r < nown ? key[r] : kNoKey);
      if (lane == 0) s_gmin[buf][g] = best;
    }
    __syncthreads();
  };
  regroup(0);
  int T = 1;
  while (T < 8 && 2 * T * nown <= nthr) T <<= 1;
  const int per = 32 / T, rounds = (nown + per * nw - 1) / (per * nw);
  const int dense_deg = kGlobal ? INT_MAX : max(4, rounds * (W / T + 4) * nw * CS / 6);
  // the counters of owned member r after its row became pc neighbours
  auto settle = [&](int r, int pc, int lv, int hnow) {
    const int l = r * CS + rank;
    int ex = ext[r], mult = 1;  // entries of v in the list
    const int valid = vc[r] + outc[r] + ex;
    if (ex > 0) {
      const int u = ids[l], v = ids[lv];
      mult = 0;
      for (int e = A.adj_off[u]; e < A.adj_off[u + 1]; e++) mult += A.adj_v[e] == v;
      mult = max(1, mult);
      ex -= mult - 1;
      ext[r] = ex;
    }
    int J = junk[r];
    J = valid - mult > 0 || A.heap ? 0 : J + valid;  // nothing valid left: the stale size stays as junk
    const int size = J + pc + outc[r] + ex;
    const int h = max(hgt[r], hnow + 1);
    vc[r] = pc;
    junk[r] = J;
    hgt[r] = h;
    if (key[r] != kNoKey) key[r] = pack_key(size, h, l);
    if (size > cap[r]) atomicCAS(A.err, 0, kErrOverflow);
  };
  for (int j = 0; j < k; j++) {
    const int par = j & 1;
    // ---- the pick
    unsigned long long b;
    {
      const unsigned long long x = s_gmin[par][lane], y = s_gmin[par][lane + 32];
      b = x < y ? x : y;
    }
    if (kGrid) {
      unsigned long long *best = A.best + ((int64_t)ci * 2 + par) * CS;
      if (wid == 0) {
        b = warp_min(b);
        if (lane == 0) best[rank] = b;
      }
      if (!grid_meet(A.arrived + ci, ++meets * CS, A, &s_ok)) return;
      b = kNoKey;
      for (int i = lane; i < CS; i += 32) {
        const unsigned long long x = __ldcg(best + i);
        b = x < b ? x : b;
      }
      b = warp_min(b);
    } else if (CS == 1) {
      b = warp_min(b);
    } else {
      if (wid == 0) {
        b = warp_min(b);
        if (lane < CS) *cluster.map_shared_rank(&s_best[par][rank], lane) = b;
      }
      cluster.sync();
      b = warp_min(lane < CS ? s_best[par][lane] : kNoKey);
    }
    if (b == kNoKey) {  // the same in every CTA of the cluster
      if (rank == 0 && tid == 0) atomicCAS(A.err, 0, kErrPick);
      break;
    }
    const int lv = (int)(b & (kMaxMembers - 1));
    const int hnow = (int)(b >> (kIdxBits + kDegBits)) - (int)((b >> kIdxBits) & ((1u << kDegBits) - 1));
    const int owner = lv & (CS - 1);
    const unsigned *rv;
    if (CS == 1 && !kGlobal) {
      rv = own_row(lv);
    } else {
      const unsigned *src = kGlobal ? grows + (int64_t)lv * Wm
                                    : cluster.map_shared_rank(srows, owner) + (int64_t)(lv >> csh) * Wm;
      for (int w = tid; w < W; w += nthr) rowv[w] = kGlobal ? __ldcg(src + w) : src[w];
      __syncthreads();
      rv = rowv;
    }
    // ---- its neighbours among the owned members
    const int rlv = owner == rank ? lv >> csh : -1;  // v's own row, if it is one of this CTA's
    auto retire = [&]() {
      key[rlv] = kNoKey;
      A.elim[c.start + j] = ids[lv];
      if (vc[rlv] == 0 && !A.heap) atomicCAS(A.err, 0, kErrEmpty);  // a partition cell never isolates a candidate
    };
    if ((int)((b >> kIdxBits) & ((1u << kDegBits) - 1)) < dense_deg) {
      for (int g = wid; g < G; g += nw) {
        const int r0 = lane * G + g, l0 = r0 * CS + rank;
        const bool hit = r0 < nown && ((rv[l0 >> 5] >> (l0 & 31)) & 1u);
        unsigned todo = __ballot_sync(0xffffffffu, hit);
        const bool mine = __any_sync(0xffffffffu, r0 == rlv);
        unsigned long long best = s_gmin[par][g];
        if (todo || mine) {
          int deg = 0;
          while (todo) {
            const int at = __ffs(todo) - 1, r = at * G + g, l = r * CS + rank;
            todo &= todo - 1;
            unsigned *row = own_row(r);
            int pc = 0;
            constexpr int kAhead = kGlobal ? 8 : 1;  // words of a lane in flight
            for (int w0 = lane; w0 < W; w0 += 32 * kAhead) {
              unsigned x[kAhead];
#pragma unroll
              for (int q = 0; q < kAhead; q++) {
                const int w = w0 + 32 * q;
                x[q] = kGlobal ? (w < W ? __ldcg(row + w) : 0) : row[w];
              }
#pragma unroll
              for (int q = 0; q < kAhead; q++) {
                const int w = w0 + 32 * q;
                if (kGlobal && w >= W) break;
                unsigned y = x[q] | rv[w];
                if (w == (l >> 5)) y &= ~(1u << (l & 31));
                if (w == (lv >> 5)) y &= ~(1u << (lv & 31));
                row[w] = y;
                pc += __popc(y);
              }
            }
            pc = __reduce_add_sync(0xffffffffu, pc);
            if (lane == at) deg = pc;
          }
          if (hit) settle(r0, deg, lv, hnow);
          if (r0 == rlv) retire();
          best = warp_min(r0 < nown ? key[r0] : kNoKey);  // each lane reads the key it alone writes
        }
        if (lane == 0) s_gmin[par ^ 1][g] = best;
      }
      __syncthreads();
    } else {
      const int sub = lane & (T - 1);
      for (int g = wid; g * per < nown; g += nw) {
        const int r = g * per + lane / T, l = r * CS + rank;
        const bool hit = r < nown && ((rv[l >> 5] >> (l & 31)) & 1u);
        int pc = 0;
        if (hit) {
          unsigned *row = own_row(r);
          for (int w = sub; w < W; w += T) {
            unsigned x = row[w] | rv[w];
            if (w == (l >> 5)) x &= ~(1u << (l & 31));
            if (w == (lv >> 5)) x &= ~(1u << (lv & 31));
            row[w] = x;
            pc += __popc(x);
          }
        }
        for (int o = 1; o < T; o <<= 1) pc += __shfl_xor_sync(0xffffffffu, pc, o);
        if (hit && sub == 0) settle(r, pc, lv, hnow);
      }
      if (rlv >= 0 && tid == 0) retire();
      __syncthreads();
      regroup(par ^ 1);
    }
    if (j == 0 && !A.heap) {  // live keys from the second pick on
      for (int r = tid; r < nown; r += nthr)
        if (key[r] != kNoKey) key[r] = pack_key(junk[r] + vc[r] + outc[r] + ext[r], hgt[r], r * CS + rank);
      __syncthreads();
      regroup(par ^ 1);
    }
  }
  // ---- lists: an eliminated member's row is its X in id order; a member that
  // stays lists its entries outside the cell, then its row as places in the
  // parent's members (the ones that stay go there in id order)
  if (wid == 0) {
    int q = 0;
    for (int l0 = 0; l0 < S; l0 += 32) {
      const int l = l0 + lane;
      const bool stay = l < S && !((cand[l >> 5] >> (l & 31)) & 1u);
      const unsigned bal = __ballot_sync(0xffffffffu, stay);
      const int at = q + __popc(bal & ((1u << lane) - 1u));
      if (l < S) map[l] = c.obase + at;
      if (stay && rank == 0 && c.out >= 0) A.members[c.out + at] = ids[l];
      q += __popc(bal);
    }
  }
  // the lists' places: one run of the pool for the CTA
  __syncthreads();
  if (wid == 0) {
    unsigned long long total = 0;
    for (int r0 = 0; r0 < nown; r0 += 32) {
      const int r = r0 + lane, l = r * CS + rank;
      const int len = r < nown ? vc[r] + ((cand[l >> 5] >> (l & 31)) & 1u ? 0 : outc[r]) : 0;
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (r < nown) key[r] = total + (unsigned)(incl - len);
      total += (unsigned)__shfl_sync(0xffffffffu, incl, 31);
    }
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(A.pool_next, total);
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int r = lane; r < nown; r += 32) key[r] += at;
  }
  __syncthreads();
  for (int r = wid; r < nown; r += nw) {
    const int l = r * CS + rank, u = ids[l];
    const bool gone = (cand[l >> 5] >> (l & 31)) & 1u;
    const int out = gone ? 0 : outc[r], len = vc[r] + out;
    const int64_t old = A.slot_off[u], off = (int64_t)key[r];
    const bool room = off + len <= A.pool_size, fits = room && len <= cap[r];
    if (fits) {
      int *dst = A.pool + off;
      int q = 0;
      if (out > 0) {
        const int *list = A.pool + old;
        const int n0 = A.lsize[u];
        for (int e0 = 0; e0 < n0 && q < out; e0 += 32) {
          const int y = e0 + lane < n0 ? __ldcg(list + e0 + lane) : 0;
          const bool o = y < 0 && find_id(ids, S, ~y) < 0;
          const unsigned bal = __ballot_sync(0xffffffffu, o);
          if (o) dst[q + __popc(bal & ((1u << lane) - 1u))] = y;
          q += __popc(bal);
        }
      }
      const unsigned *row = own_row(r);
      const int *name = gone ? ids : map;
      for (int w = 0; w < W; w++) {
        const unsigned x = kGlobal ? __ldcg(row + w) : row[w];
        if ((x >> lane) & 1u) dst[q + __popc(x & ((1u << lane) - 1u))] = name[w * 32 + lane];
        q += __popc(x);
      }
    }
    if (lane == 0) {
      if (!fits) atomicCAS(A.err, 0, room ? kErrOverflow : kErrPool);
      A.slot_off[u] = off;
      A.lsize[u] = fits ? len : 0;
      A.ljunk[u] = gone ? 0 : junk[r];
      A.extra[u] = ext[r];
      A.height[u] = hgt[r];
    }
  }
  if (!kGrid && CS > 1) cluster.sync();  // no CTA leaves while a peer may still read its rows
}

// Distinct neighbours of every vertex's input list as ~id, in the list's order,
// and the number of repeated entries.  A thread takes a list of up to 32
// entries, its warp the longer ones: comparing every pair in one thread took
// 3.7 s for a vertex of 16,000 neighbours (the whole contraction takes 0.2 s).
__global__ void distinct_lists_kernel(const int *adj_off, const int *adj_v, int64_t *slot_off, int *pool, int *lsize,
                                      int *extra, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~int64_t(31); v0 < n;
       v0 += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)v0 + lane;
    const int b = v < n ? adj_off[v] : 0, e = v < n ? adj_off[v + 1] : 0;
    if (v < n) slot_off[v] = b;  // the pool starts with the input lists' places
    if (v < n && e - b <= 32) {
      int *list = pool + b;
      int c = 0;
      for (int i = b; i < e; i++) {
        const int x = ~adj_v[i];
        bool seen = false;
        for (int q = 0; q < c && !seen; q++) seen = list[q] == x;
        if (!seen) list[c++] = x;
      }
      lsize[v] = c;
      extra[v] = e - b - c;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, e - b > 32); todo; todo &= todo - 1) {
      const int from = __ffs(todo) - 1;
      const int lb = __shfl_sync(0xffffffffu, b, from), le = __shfl_sync(0xffffffffu, e, from);
      int c = 0;
      for (int i0 = lb; i0 < le; i0 += 32) {
        const int i = i0 + lane, x = i < le ? adj_v[i] : -1;
        bool fresh = i < le;
        for (int q0 = lb; q0 < i0; q0 += 32) {  // a lane per earlier entry, handed round
          const int y = adj_v[q0 + lane];
#pragma unroll
          for (int q = 0; q < 32; q++) fresh &= __shfl_sync(0xffffffffu, y, q) != x;
        }
#pragma unroll
        for (int q = 0; q < 31; q++) {
          const int y = __shfl_sync(0xffffffffu, x, q);
          if (q < lane) fresh &= y != x;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, fresh);
        if (fresh) pool[lb + c + __popc(bal & ((1u << lane) - 1u))] = ~x;
        c += __popc(bal);
      }
      if (lane == 0) {
        lsize[v0 + from] = c;
        extra[v0 + from] = le - lb - c;
      }
    }
  }
}

// The final lists one after another.  One warp per vertex.
__global__ void gather_ids_kernel(const int64_t *slot_off, const int *lsize, const int *pool, const int64_t *out_off,
                                  int *out_nbr, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; v < n;
       v += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int *src = pool + slot_off[v];
    const int64_t oo = out_off[v];
    const int s = lsize[v];
    for (int i = lane; i < s; i += 32) out_nbr[oo + i] = src[i];
  }
}

// A graph's members before its first level, in partition order (in id order
// where no level runs).
__global__ void members_kernel(const int *part, int *members, int n, int vb) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
    members[q] = (part ? part[q] : q) + vb;
}

// Alive members of every cell at its level, or false when the cut rows do not
// nest (each level tiling the positions, a cell split by its two children).
bool cell_sizes(const Graph &g, std::vector<int> &size) {
  const int64_t cells = (int64_t(1) << g.H) - 1;
  size.assign(cells, 0);
  if (g.cut_l[0] != 0 || g.cut_r[0] != g.n) return false;
  const int64_t inner = (int64_t(1) << (g.H - 1)) - 1;
  for (int64_t c = 0; c < inner; c++)
    if (g.cut_l[2 * c + 1] != g.cut_l[c] || g.cut_r[2 * c + 1] != g.cut_l[2 * c + 2] ||
        g.cut_r[2 * c + 2] != g.cut_r[c])
      return false;
  for (int64_t c = cells - 1; c >= 0; c--) {
    size[c] = c >= inner ? g.cut_r[c] - g.cut_l[c]
                         : size[2 * c + 1] - g.cell_count[2 * c + 1] + size[2 * c + 2] - g.cell_count[2 * c + 2];
    if (size[c] < g.cell_count[c]) return false;
  }
  return true;
}

}  // namespace

// Lays out the elimination on bit rows, if every cell's members fit a row
// (up to 16,384) and the partition nests.  False: the list kernels run, as
// they also do when one of their switches is set.  A 16,384-member cell takes
// 32 MB of rows and about 10 us a pick; past that, sparse lists are the
// smaller working set (a global order over a whole 264k-vertex graph would
// scan 33 KB per row).
bool ElimPlan::plan_bits() {
  for (const char *e : {"GPUH2H_CLUSTER_HEAP", "GPUH2H_GRID_CELLS", "GPUH2H_GLOBAL_STAGING", "GPUH2H_GRID_ARENA",
                        "GPUH2H_ELIM_BALANCE", "GPUH2H_LIST_ELIM"})
    if (std::getenv(e)) return false;
  const int K = (int)gs.size();
  if (N >= (1 << (kSumBits - 2)) || gs[0]->sets->cap_max >= (1 << (kDegBits - 1))) return false;
  struct Host {
    SymCell c;
    int level;
  };
  std::vector<std::vector<Host>> steps;
  std::vector<std::vector<int>> sizes(K);
  int nsteps = 0;
  for (int i = 0; i < K; i++) {
    if (!cell_sizes(*gs[i], sizes[i])) return false;
    nsteps = std::max(nsteps, gs[i]->H - gs[i]->C);
  }
  steps.resize(nsteps + 1);
  int64_t mem_total = N;  // the bottom cells' members come first, in partition order
  for (int i = 0; i < K; i++) {
    const Graph &g = *gs[i];
    const int vb = vbase[i], levels = g.H - g.C;
    std::vector<int64_t> region(sizes[i].size(), -1);
    int64_t heap_region = levels > 0 ? -1 : vb;
    int heap_n = 0;
    for (int64_t c = 0; c < (int64_t)sizes[i].size() && c < (int64_t(1) << g.C) - 1; c++) heap_n += g.cell_count[c];
    if (heap_n > kMaxMembers) return false;
    if (levels > 0) {
      heap_region = mem_total;
      mem_total += heap_n;
    }
    int64_t heap_at = heap_region;
    for (int h = g.H; h > g.C; h--) {
      const int64_t lo = (int64_t(1) << (h - 1)) - 1, hi = (int64_t(1) << h) - 2;
      for (int64_t c = lo; c <= hi; c++) {
        if (sizes[i][c] > kMaxMembers) return false;
        if (h == g.H) region[c] = vb + g.cut_l[c];
        const int stay = sizes[i][c] - g.cell_count[c];
        int64_t out, parent;
        if (h - 1 > g.C) {
          const int64_t p = (c - 1) / 2;
          if (region[p] < 0) {
            region[p] = mem_total;
            mem_total += sizes[i][p];
          }
          parent = region[p];
          out = parent + (c & 1 ? 0 : sizes[i][c - 1] - g.cell_count[c - 1]);
        } else {
          parent = heap_region;
          out = heap_at;
          heap_at += stay;
        }
        const int st = g.H - h;
        steps[st].push_back({{vb + g.cell_start[c], g.cell_count[c], sizes[i][c], region[c], out,
                              (int)(out - parent)},
                             K > 1 ? -(st + 1) : h});
      }
    }
    if (levels > 0 && heap_at != heap_region + heap_n) return false;
    int heap_start = g.n - heap_n;
    steps[nsteps].push_back({{vb + heap_start, heap_n, heap_n, heap_region, -1, 0}, 0});
  }
  // ---- launches: a step's cells by size class, each class with its own
  // cluster size.  A pick costs a fixed part (argmin and barriers: 1.1 us in
  // one CTA, 1.5 us across a cluster) and its neighbours' rows, 1 us + 45 ps
  // per word of the cell, which a cluster shares.  Measured us per pick with 1
  // / 2 / 4 / 8 / 16 CTAs: 716 members 3.4 / 2.9 / 2.3 / 1.9 / 1.9, 1,604 members
  // - / - / 2.5 / 2.0 / 1.8, 2,968 members - / - / - / 2.7 / 2.3.  The bottom
  // cells' members have the input's few arcs, so their rows cost a tenth: 32 cells
  // of 469 members 0.44 ms with one CTA each, 0.62 with 2, 0.59 with 4, 0.70 with 16.  Cells that
  // outnumber the SMs keep few warps (1,024 cells of 259 members: 0.54 ms with
  // 4 warps, 0.67 with 8; 2,048 cells of 489: 3.7 with 4, 2.8 with 8, 3.9 with 16).
  // A shallow partition has many bottom cells of thousands of members, whose rows
  // fill a cluster's shared memory, so that only a dozen cells run at a time.
  // With the rows in global memory a cell takes as few CTAs as its other tables
  // need, a pick 2.2 us + 0.4 ns per owned member + 0.1 ns per member:
  // 256 cells of 3,907 members 221 ms in shared memory on 16 CTAs each, 27 in
  // global memory on 2 (71 on the list kernels); 64 of 4,131 65.6 -> 11.9 (46.7);
  // 128 of 7,813 187 on 16 CTAs -> 89 on 8 (77.6); 512 of 1,954 41.6 -> 11.4 (49.9).
  const int smem_dyn = enable_max_dynamic_smem(symbolic_kernel<false, false>);
  enable_max_dynamic_smem(symbolic_kernel<true, false>);
  const int smem_grid = enable_max_dynamic_smem(symbolic_kernel<true, true>);
  GH_CUDA(cudaFuncSetAttribute(symbolic_kernel<false, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  GH_CUDA(cudaFuncSetAttribute(symbolic_kernel<true, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  int dev = 0;
  GH_CUDA(cudaGetDevice(&dev));
  GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  auto pow2 = [](int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
  };
  auto smem_for = [&](int smax, int cs, bool global) -> int64_t {
    const int64_t own = (smax + cs - 1) / cs, w = (smax + 31) / 32 | 1;
    return own * (8 + 24) + 4LL * smax + 4LL * pow2(smax) + 8 * w + (global ? 0 : 4 * own * w);
  };
  // room for the rows of a launch's cells in global memory; asked only where
  // they take more than 64 MB
  auto rows_fit = [&](int ncell, int smax) {
    const int64_t bytes = 4LL * ncell * smax * ((smax + 31) / 32 | 1);
    if (bytes <= (int64_t(64) << 20)) return true;
    size_t fr = 0, tot = 0;
    GH_CUDA(cudaMemGetInfo(&fr, &tot));
    return (uint64_t)bytes <= fr / 4;
  };
  std::vector<SymCell> table;
  int64_t grow_words = 0, grid_best = 0;
  grid_cells = 0;
  for (int st = 0; st <= nsteps; st++) {
    std::vector<Host> &cells = steps[st];
    std::stable_sort(cells.begin(), cells.end(), [](const Host &a, const Host &b) { return a.c.size > b.c.size; });
    int64_t step_words = 0;
    for (size_t g0 = 0; g0 < cells.size();) {
      if (cells[g0].c.size == 0) break;  // only empty cells are left
      const int smax = cells[g0].c.size;
      size_t g1 = g0;
      while (g1 < cells.size() && cells[g1].c.size * 3 > smax * 2) g1++;  // within a third of the largest
      SymLaunch L{};
      L.step = st;
      L.level = cells[g0].level;
      L.heap = st == nsteps;
      L.lo = (int64_t)table.size();
      L.ncell = (int)(g1 - g0);
      L.smax = smax;
      L.npow = pow2(smax);
      L.kmax = 0;
      for (size_t c = g0; c < g1; c++) {
        table.push_back(cells[c].c);
        L.kmax = std::max(L.kmax, cells[c].c.count);
      }
      double best = 1e300;
      const bool bottom = st == 0 && nsteps > 0;
      // rows in global memory only for bottom cells, or where nothing else fits
      for (int global = 0; global < 2 && (best > 1e299 || (bottom && rows_fit(L.ncell, smax))); global++)
        for (int cs = 1; cs <= 16; cs <<= 1) {
          const int64_t sm = smem_for(smax, cs, global);
          if (sm > smem_dyn || (global && cs < 16 && !bottom)) continue;
          const int own = (smax + cs - 1) / cs, w = (smax + 31) / 32;
          int nw = cs > 1 ? (own >= 64 ? 16 : 8) : L.ncell > 4 * nsm ? (own >= 384 ? 8 : 4) : own >= 300 ? 16 : 8;
          if ((own + 31) / 32 > kMaxGroups) continue;
          const double rows = (bottom ? 0.1 : 1.0) * (1.0 + 4.5e-5 * smax * w);
          const double pick = global && bottom ? 2.2 + 4e-4 * own + 1e-4 * smax : (cs == 1 ? 1.1 : 1.5) + rows / cs;
          // with an SM's 64 warps full it would not be better: the occupancy need not be asked
          if (std::ceil((double)L.ncell * cs * nw / (64.0 * nsm)) * pick >= best * 0.99) continue;
          int fit = 0;
          cudaLaunchConfig_t cfg = {};
          cudaLaunchAttribute attr[1];
          attr[0].id = cudaLaunchAttributeClusterDimension;
          attr[0].val.clusterDim.x = cs;
          attr[0].val.clusterDim.y = 1;
          attr[0].val.clusterDim.z = 1;
          cfg.attrs = attr;
          cfg.numAttrs = 1;
          cfg.blockDim = dim3(nw * 32);
          cfg.dynamicSmemBytes = (size_t)sm;
          cfg.gridDim = dim3(L.ncell * cs);
          const cudaError_t e = global ? cudaOccupancyMaxActiveClusters(&fit, symbolic_kernel<true, false>, &cfg)
                                       : cudaOccupancyMaxActiveClusters(&fit, symbolic_kernel<false, false>, &cfg);
          if (e != cudaSuccess || fit < 1) {
            cudaGetLastError();
            continue;
          }
          const double waves = std::ceil((double)L.ncell / fit);
          const double cost = waves * pick;
          if (cost < best * 0.99) {
            best = cost;
            L.cs = cs;
            L.nw = nw;
            L.smem = sm;
            L.global = global != 0;
          }
        }
      // rows in global memory: a pick reads its neighbours' rows from L2, 11 us of
      // it with 16 CTAs and 5,940 members, and more CTAs pay for the dearer
      // barrier (4.8 us a pick with 128)
      if (L.global || best > 1e299)
        for (int cs = 32; cs <= 128 && cs * L.ncell <= nsm; cs <<= 1) {
          const int64_t sm = smem_for(smax, cs, true);
          const int own = (smax + cs - 1) / cs, w = (smax + 31) / 32, nw = 16;
          int per_sm = 0;
          if (sm > smem_grid || (own + 31) / 32 > kMaxGroups) continue;
          GH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, symbolic_kernel<true, true>, nw * 32, (size_t)sm));
          if (per_sm < 1) continue;
          const double cost = 3.8 + (1.0 + 4.5e-5 * smax * w) / cs;
          if (cost < best * 0.99) {
            best = cost;
            L.cs = cs;
            L.nw = nw;
            L.smem = sm;
            L.global = L.grid = true;
          }
        }
      if (best > 1e299) return false;
      if (L.grid) {
        L.best_off = grid_best;
        L.arrived_off = grid_cells;
        grid_best += 2 * (int64_t)L.ncell * L.cs;
        grid_cells += L.ncell;
      }
      if (L.global) {
        L.rows_off = step_words;
        step_words += (int64_t)L.ncell * smax * ((smax + 31) / 32 | 1);
      }
      sym.push_back(L);
      g0 = g1;
    }
    grow_words = std::max(grow_words, step_words);
  }
  max_group = 1;
  for (size_t i = 0; i < sym.size();) {
    size_t j = i;
    while (j < sym.size() && sym[j].step == sym[i].step) j++;
    max_group = std::max(max_group, (int)(j - i));
    i = j;
  }
  try {
    members = mem.get<int>(mem_total);
    extra = mem.get<int>(N);
    sym_cells = mem.get<unsigned char>(sizeof(SymCell) * table.size());
    if (grow_words) grows = mem.get<unsigned>(grow_words);
    if (grid_cells) {
      sym_best = mem.get<unsigned long long>(grid_best);
      sym_arrived = mem.get<unsigned>(grid_cells);
    }
    for (int i = 0; i < K; i++) {
      const int n = gs[i]->n;
      members_kernel<<<std::max(1, std::min(4096, (n + 255) / 256)), 256>>>(
          gs[i]->H > gs[i]->C ? input_device(*gs[i]).part : nullptr, members + vbase[i], n, vbase[i]);
      GH_CUDA(cudaGetLastError());
    }
    GH_CUDA(cudaMemcpy(sym_cells, table.data(), sizeof(SymCell) * table.size(), cudaMemcpyHostToDevice));
  } catch (...) {
    release();
    throw;
  }
  return true;
}

void ElimPlan::enqueue_bits(cudaStream_t s, cudaEvent_t *heap_ev, bool trace) {
  GH_CUDA(cudaMemcpyAsync(elim, elim_init, sizeof(int) * N, cudaMemcpyDeviceToDevice, s));
  GH_CUDA(cudaMemcpyAsync(pool_next, pool_first, sizeof(unsigned long long), cudaMemcpyDeviceToDevice, s));
  GH_CUDA(cudaMemsetAsync(height, 0, sizeof(int) * N, s));
  GH_CUDA(cudaMemsetAsync(ljunk, 0, sizeof(int) * N, s));
  GH_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
  if (grid_cells) GH_CUDA(cudaMemsetAsync(sym_arrived, 0, sizeof(unsigned) * grid_cells, s));
  distinct_lists_kernel<<<std::max(1, std::min(4096, (N + 255) / 256)), 256, 0, s>>>(adj_off, adj_v, slot_off, pool,
                                                                                     lsize, extra, N);
  GH_CUDA(cudaGetLastError());
  auto launch = [&](const SymLaunch &L, cudaStream_t ls) {
    SymArgs A{};
    A.cells = reinterpret_cast<const SymCell *>(sym_cells) + L.lo;
    A.pool = pool;
    A.slot_off = slot_off;
    A.lsize = lsize;
    A.ljunk = ljunk;
    A.extra = extra;
    A.height = height;
    A.elim = elim;
    A.members = members;
    A.err = err;
    A.cap = cap_init;
    A.deg0 = deg_init;
    A.adj_off = adj_off;
    A.adj_v = adj_v;
    A.grows = L.global ? grows + L.rows_off : nullptr;
    A.pool_next = pool_next;
    A.pool_size = pool_size;
    A.smax = L.smax;
    A.npow = L.npow;
    A.heap = L.heap;
    if (L.grid) {
      A.cs = L.cs;
      A.best = sym_best + L.best_off;
      A.arrived = sym_arrived + L.arrived_off;
      A.spin_limit = spin_limit_cycles();
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    if (L.grid) {
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
    } else {
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = L.cs;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(L.nw * 32);
    cfg.dynamicSmemBytes = (size_t)L.smem;
    cfg.gridDim = dim3(L.ncell * L.cs);
    cfg.stream = ls;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (trace) { cudaEventCreate(&e0); cudaEventCreate(&e1); cudaEventRecord(e0, ls); }
    if (L.grid) GH_CUDA(cudaLaunchKernelEx(&cfg, symbolic_kernel<true, true>, A));
    else if (L.global) GH_CUDA(cudaLaunchKernelEx(&cfg, symbolic_kernel<true, false>, A));
    else GH_CUDA(cudaLaunchKernelEx(&cfg, symbolic_kernel<false, false>, A));
    if (trace) {
      cudaEventRecord(e1, ls);
      cudaEventSynchronize(e1);
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      std::fprintf(stderr, "[gpuh2h] elim bits %s %d: %d cells x %d CTAs x %d warps, kmax %d, members %d, smem %lld%s: %.3f ms\n",
                   L.heap ? "heap" : "level", L.level, L.ncell, L.cs, L.nw, L.kmax, L.smax, (long long)L.smem,
                   L.grid ? " (one grid)" : L.global ? " (rows in global memory)" : "", ms);
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
    }
  };
  for (size_t li = 0; li < sym.size();) {
    size_t lj = li;
    while (lj < sym.size() && sym[lj].step == sym[li].step) lj++;
    if (sym[li].heap && heap_ev) GH_CUDA(cudaEventRecord(heap_ev[0], s));
    if (lj - li > 1) GH_CUDA(cudaEventRecord(ev_fork, s));
    for (size_t k = li; k < lj; k++) {
      cudaStream_t ls = s;
      if (k > li) {
        ls = side[k - li - 1];
        GH_CUDA(cudaStreamWaitEvent(ls, ev_fork, 0));
      }
      launch(sym[k], ls);
      if (k > li) GH_CUDA(cudaEventRecord(ev_join[k - li - 1], ls));
    }
    for (size_t k = li + 1; k < lj; k++) GH_CUDA(cudaStreamWaitEvent(s, ev_join[k - li - 1], 0));
    li = lj;
  }
  if (heap_ev) {
    if (sym.empty() || !sym.back().heap) GH_CUDA(cudaEventRecord(heap_ev[0], s));
    GH_CUDA(cudaEventRecord(heap_ev[1], s));
  }
}

// A larger pool for another run, unless the list kernels' slot arrays would
// take no more.
bool ElimPlan::grow_pool() {
  const int64_t most = 2 * (slots_size + 4);
  if (pool_size >= most) return false;
  free_pool();
  pool_size = std::min(most, 4 * pool_size);
  if (std::getenv("GPUH2H_TRACE"))
    std::fprintf(stderr, "[gpuh2h] elim bits: list pool grown to %lld entries\n", (long long)pool_size);
  if (cudaMalloc(&pool, sizeof(int) * (size_t)pool_size) != cudaSuccess) {
    cudaGetLastError();
    pool = nullptr;
    return false;
  }
  own_pool = true;
  slot_bytes = 4 * pool_size;
  return true;
}

void ElimPlan::free_pool() {
  if (own_pool) cudaFree(pool);
  pool = nullptr;
  own_pool = false;
  slot_bytes = 0;
}

void ElimPlan::gather_bits(cudaStream_t s) {
  gather_ids_kernel<<<std::max(1, std::min(8192, (N * 32 + 255) / 256)), 256, 0, s>>>(
      slot_off, lsize, pool, lists.off, lists.id, N);
  GH_CUDA(cudaGetLastError());
}

}  // namespace gh
