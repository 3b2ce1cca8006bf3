// fill_blocks.cu -- the no-hub L4 label fill (the work of
// makeH2HLabel_noHub_noComm_3 / makeH2HLabel_noCommunication_D_noHub_3,
// tanslate.cu:511-617, kernel_functions.cu:717-796, with the L4 block
// :738-743 enabled) as min-plus products over blocks of the tree.
//
// Row v holds dis[v][j] = D(v, a_j), the distance to the ancestor a_j at depth
// j + 1, and
//   D(v, a) = min over u in X(v)\{v} of sc(v, u) + E(u, a),
//   E(u, a) = dis[u][j] (u below a), 0 (u = a), dis[a][p_u] (u above a).
// Node by node that is a load per (v, u, j) and a dependency per tree level.
// Here the tree is cut into blocks of at most 32 nodes, each a connected piece
// with one top t.  Every node i of a block has its upper neighbours among the
// block's own nodes and X(t) (the lists nest: X(v) without v's father lies in
// X(father)), so replacing a neighbour inside the block by that neighbour's
// own recursion leaves, for every ancestor a above the block,
//   D(i, a) = min over u in X(t) of S(i, u) + E(u, a),
//   S(i, u) = min(sc(i, u), min over w in X(i) inside the block of sc(i, w) + S(w, u)).
// S needs no label (closure_kernel computes it for all blocks at once), and
// the columns above the block become one min-plus product [32 x |X(t)|] by
// [|X(t)| x depth(t)] whose second factor is loaded once for 32 rows.  For two
// nodes i below a of one block the way either stays inside the block or passes
// a last u in X(t),
//   D(i, a) = min(W(i, a), min over u in X(t) of S(i, u) + D(a, u)),
// where W, the recursion over the block's nodes alone, needs no label either
// (inner_closure_kernel) and column u of row a has just been computed.  D is
// the distance in the graph whose arc {v, u} weighs what the endpoint eliminated
// first says, so both forms of a sum agree.  Sums are taken in unsigned 32-bit
// arithmetic, where two values below 2^31 cannot wrap, with INT_MAX for "no
// entry".
//
// A fill that takes a warp per (node, column block, separator chunk) tile is
// bound by one L2 load per update and 13 us per tree level of the narrow top.
// On one GB300 the blocks took the fill of a 264k-vertex road graph (4.5e9
// updates) from 28.4 to 2.1 ms and of a 1M-vertex one (3.8e10) from 104 to 11.1
// ms.  Narrow levels are a chain of blocks (about 22 us each, a step of 32
// members 3,100 clocks); below them a term costs an ALU slot of half rate and the
// kernel fills over half of those slots.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <utility>

#include "graph.h"
#include "scan.h"

namespace gh {

namespace {

constexpr int kRows = 32;     // nodes of a block (rows of its product)
constexpr int kSmall = 16;    // largest light subtree that joins its father's block whole
constexpr int kCols = 64;     // columns of one step of the product
constexpr int kMembers = 32;  // separator members of one step
constexpr int kMaxTiles = 64; // most tiles (of kCols columns) in a task
constexpr int kEStride = 84;  // row stride of the staged second factor: 16-byte stores of eight rows hit all banks, of two rows nearly
constexpr unsigned kInf = 0x7fffffffu;

constexpr int kErrWait = 4;    // a dependency wait ran out
constexpr int kErrNested = 6;  // an upper neighbour is missing from the block top's separator

__device__ __forceinline__ void cp_async16(void *smem, const void *global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed(const int *p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned add_min(unsigned a, unsigned b, unsigned c) { return __viaddmin_u32(a, b, c); }

// ------------------------------------------------------------ the plan
//
// Blocks from the heavy-path layout (hld: a depth-first order that visits the
// heavy child first, so a subtree is a range of it).  A light subtree of at
// most kSmall nodes joins its father's block; the nodes left are paths, cut
// greedily from the top so that a path node with its small subtrees stays in
// one block and a block holds at most kRows nodes.  A path node whose small
// subtrees alone exceed a block leaves each of them a block of its own.  On a
// 264k-vertex road graph: 11.2k blocks of 23.5 nodes on average, 67 blocks
// from the root to the deepest leaf (1,347 nodes), 9e9 product terms for
// 4.6e9 updates of the recursion, and 3e8 loads of E in place of 4.6e9.  With
// kSmall 8 the blocks average 19 nodes; blocks of 64 nodes would halve the
// loads again but add 15% terms and double the top's in-block pass.

// size of the subtree at every position, if at most kSmall (else kSmall + 1)
__global__ void small_size_kernel(const int *hld, const int *depth, int *size, int *weight, int n) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int d = depth[hld[k]];
    int s = 1;
    while (s <= kSmall && k + s < n && depth[hld[k + s]] > d) s++;
    size[k] = s;
    weight[k] = 1;
  }
}

// weight of a path node: itself and its small light subtrees
__global__ void hang_weight_kernel(const int *father, const int *htop, const int *hpos, const int *size, int *weight,
                                   int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int f = father[v];
    if (f < 0 || htop[v] != v) continue;
    const int s = size[hpos[v]];
    if (s <= kSmall) atomicAdd(weight + hpos[f], s);
  }
}

// Greedy cut of every long path, one warp per path: lanes load 32 path nodes,
// the running weight goes through them by shuffles.
__global__ void cut_paths_kernel(const int *father, const int *htop, const int *hpos, const int *hld, const int *size,
                                 const int *weight, int *block_top, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n;
       base += ((gridDim.x * (int64_t)blockDim.x) >> 5) * 32) {
    const int v = (int)base + lane;
    const bool path = v < n && htop[v] == v && (father[v] < 0 || size[hpos[v]] > kSmall);
    unsigned todo = __ballot_sync(0xffffffffu, path);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const int top = (int)base + l;
      int cur = kRows, bt = top;  // the first node opens a block
      for (int64_t k0 = hpos[top]; k0 < n; k0 += 32) {
        const int64_t k = k0 + lane;
        const int u = k < n ? hld[k] : -1;
        const bool on = u >= 0 && htop[u] == top;
        int w = on ? weight[k] : 0;
        if (w > kRows) w = 1;
        const unsigned live = __ballot_sync(0xffffffffu, on);
        const int cnt = live == 0xffffffffu ? 32 : __ffs(~live) - 1;  // the path's nodes are contiguous
        int mine = 0;
        for (int s = 0; s < cnt; s++) {
          const int ws = __shfl_sync(0xffffffffu, w, s), us = __shfl_sync(0xffffffffu, u, s);
          if (cur + ws > kRows) {
            cur = 0;
            bt = us;
          }
          cur += ws;
          if (s == lane) mine = bt;
        }
        if (lane < cnt) block_top[k] = mine;
        if (cnt < 32) break;
      }
    }
  }
}

// Every node's block top; nodes and separator work per block top and level.
__global__ void node_block_kernel(const int *father, const int *htop, const int *hpos, const int *depth,
                                  const int64_t *pos_hash, const int *size, const int *weight, const int *block_top,
                                  int *top_of, int *count, int *lvl_tops, int *lvl_width, unsigned long long *lvl_work,
                                  int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    int u = v, c = -1;
    for (;;) {
      const int t = htop[u], f = father[t];
      if (f < 0 || size[hpos[t]] > kSmall) break;
      c = t;
      u = f;
    }
    const int bt = c >= 0 && weight[hpos[u]] > kRows ? c : block_top[hpos[u]];
    const int d = depth[v];
    top_of[v] = bt;
    atomicAdd(count + bt, 1);
    if (bt == v) atomicAdd(lvl_tops + d - 1, 1);
    atomicAdd(lvl_width + d - 1, 1);
    atomicAdd(lvl_work + d - 1, (unsigned long long)(pos_hash[v + 1] - pos_hash[v] - 1) * (unsigned long long)d);
  }
}

// Blocks in the order of their tops' depths: a block's father block (the
// block of its top's father) comes before it.
__global__ void order_blocks_kernel(const int *top_of, const int *depth, const int64_t *lvl_first, int *lvl_next,
                                    int *blk_top, int *blk_of_top, int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    if (top_of[v] != v) continue;
    const int d = depth[v] - 1;
    const int b = (int)lvl_first[d] + atomicAdd(lvl_next + d, 1);
    blk_top[b] = v;
    blk_of_top[v] = b;
  }
}

// The longest chain first: blocks in the order of the depth still below their
// tops, which a father has more of than its children.  deep: the deepest level
// under every block, by doubling over the father blocks (a block's value goes
// to the block 2^k up; a maximum may be taken in place).
__global__ void block_depth_kernel(const int *top_of, const int *blk_of_top, const int *depth, int *deep, int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    atomicMax(deep + blk_of_top[top_of[v]], depth[v]);
}

__global__ void father_block_kernel(const int *blk_top, const int *father, const int *top_of, const int *blk_of_top,
                                    int *up, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += gridDim.x * blockDim.x) {
    const int f = father[blk_top[b]];
    up[b] = f < 0 ? -1 : blk_of_top[top_of[f]];
  }
}

__global__ void deepest_round_kernel(const int *up, int *up_next, int *deep, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += gridDim.x * blockDim.x) {
    const int u = up[b];
    if (u >= 0) atomicMax(deep + u, *(volatile int *)(deep + b));
    up_next[b] = u >= 0 ? up[u] : -1;
  }
}

// place: how far a block's chain falls short of the longest possible
__global__ void chain_count_kernel(const int *blk_top, const int *depth, int *deep, int *cnt, int nlev, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += gridDim.x * blockDim.x) {
    const int place = max(0, min(nlev - 1, nlev - 1 - (deep[b] - depth[blk_top[b]])));
    deep[b] = place;
    atomicAdd(cnt + place, 1);
  }
}

__global__ void chain_order_kernel(const int *tops, const int *place, const int64_t *first, int *next, int *blk_top,
                                   int *blk_of_top, int nblk) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nblk; i += gridDim.x * blockDim.x) {
    const int b = (int)first[place[i]] + atomicAdd(next + place[i], 1);
    blk_top[b] = tops[i];
    blk_of_top[tops[i]] = b;
  }
}

// Level classes of TilePolicy: 0 narrow (fewer nodes than SMs), 2 heavy
// (wider, its nodes averaging at least per_node updates), 1 the others.
__global__ void level_class_kernel(const int *width, const unsigned long long *work, int nlev, int nsm,
                                   unsigned long long per_node, int *cls) {
  for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < nlev; l += gridDim.x * blockDim.x)
    cls[l] = width[l] < nsm ? 0 : work[l] >= per_node * (unsigned long long)width[l] ? 2 : 1;
}

__global__ void block_sizes_kernel(const int *blk_top, const int *count, const int64_t *pos_hash, int *rows, int *mem,
                                   int *cells, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblk; b += gridDim.x * blockDim.x) {
    int r = 0, m = 0;
    if (b < nblk) {
      const int t = blk_top[b];
      r = count[t];
      m = (int)(pos_hash[t + 1] - pos_hash[t]) - 1;
    }
    const int rp = (r + 3) & ~3;
    rows[b] = r;
    mem[b] = m;
    cells[b] = (m + rp) * rp;
  }
}

// Tasks of every block: the columns above it in one task, or cut into
// policy.col_block columns each.
__global__ void block_tasks_kernel(const int *blk_top, const int *depth, const int *mem, const int64_t *boff,
                                   const int *lvl_cls, TilePolicy pol, int *ntask, int *pieces, int *tcols, int *several, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblk; b += gridDim.x * blockDim.x) {
    int nt = 0, tc = kCols;
    if (b < nblk) {
      const int d = depth[blk_top[b]], m = mem[b];
      const int wb = lvl_cls[d - 1], sb = m <= 16 ? 0 : m <= 64 ? 1 : m <= 256 ? 2 : 3;
      const int cols = d - 1;
      tc = (pol.col_block[wb][sb] + kCols - 1) / kCols * kCols;
      if ((int64_t)m * d <= pol.small_work[wb][sb]) tc = max(kCols, (cols + kCols - 1) / kCols * kCols);
      tc = min(tc, kCols * kMaxTiles);
      nt = max(1, (cols + tc - 1) / tc);
    }
    ntask[b] = nt;
    pieces[b] = b < nblk ? nt * (int)(boff[b + 1] - boff[b]) : 0;
    tcols[b] = tc;
    several[b] = nt > 1;
  }
}

__global__ void narrow_kernel(const int64_t *in, int *out, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = (int)in[i];
}

__global__ void scatter_nodes_kernel(const int *top_of, const int *blk_of_top, const int64_t *boff, int *fill, int *bnode,
                                     int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int b = blk_of_top[top_of[v]];
    const int64_t at = boff[b] + atomicAdd(fill + b, 1);
    if (at < boff[b + 1]) bnode[at] = v;
  }
}

// A block's nodes in depth-first order (ancestors first), every node's block
// and place in it, and the top's members (positions, row offsets).  One warp
// per block.
__global__ void block_nodes_kernel(const int *blk_top, const int64_t *boff, const int64_t *moff, const int *hpos,
                                   const int64_t *pos_hash, const int *pos_pos, const int *pos_id, const int64_t *drow,
                                   int *bnode, int *blk_of, unsigned char *loc_of, int *bm_p, int64_t *bm_row,
                                   int nblk) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; b < nblk;
       b += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int64_t o = boff[b];
    const int R = (int)(boff[b + 1] - o);
    const int v = lane < R ? bnode[o + lane] : -1;
    const int k = lane < R ? hpos[v] : INT_MAX;
    int r = 0;
    for (int s = 0; s < R; s++) r += __shfl_sync(0xffffffffu, k, s) < k;
    __syncwarp();
    if (lane < R) {
      bnode[o + r] = v;
      blk_of[v] = (int)b;
      loc_of[v] = (unsigned char)r;
    }
    const int64_t pb = pos_hash[blk_top[b]], m0 = moff[b];
    const int m = (int)(moff[b + 1] - m0);
    for (int i = lane; i < m; i += 32) {
      bm_p[m0 + i] = pos_pos[pb + i];
      bm_row[m0 + i] = drow[pos_id[pb + i]];
    }
  }
}

__global__ void expand_tasks_kernel(const int64_t *task0, int *task_blk, int nblk) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; b < nblk;
       b += (gridDim.x * (int64_t)blockDim.x) >> 5)
    for (int64_t t = task0[b] + lane; t < task0[b + 1]; t += 32) task_blk[t] = (int)b;
}

// ------------------------------------------------------------ the closure

struct BlockArgs {
  const int *blk_top;
  const int64_t *boff, *moff, *soff;  // first node, first member, first cell of S and of the direct weights
  const int *bnode;
  const int *blk_of;
  const unsigned char *loc_of;
  const int *bm_p;
  const int64_t *bm_row;
  const int *father, *depth;
  const int64_t *drow, *pos_hash;
  const int *pos_pos, *pos_id, *pos_w;
  // per block [column][row], rows padded to a multiple of four: the columns
  // are the top's members, then the block's own nodes (closed: W)
  unsigned *direct, *closed;
  unsigned *anc;  // per node in the blocks' order: its ancestors inside the block, a bit per place
  int nblk;
  int *err;
};

// Members of X(v) inside the block (the end of v's position list, v itself
// excluded: positions at or below the top's), one per lane: place and weight
// into tl / tw; returns their number in every lane.
__device__ __forceinline__ int stage_inner(const BlockArgs &A, int v, int dt, unsigned char *tl, int *tw, int lane) {
  const int64_t pb = A.pos_hash[v], e = A.pos_hash[v + 1] - 2 - lane;
  const bool in = e >= pb && __ldg(A.pos_pos + e) >= dt;
  if (in) {
    tl[lane] = A.loc_of[__ldg(A.pos_id + e)];
    tw[lane] = __ldg(A.pos_w + e);
  }
  return __popc(__ballot_sync(0xffffffffu, in));
}

constexpr int kClosureWarps = 4;

// S of every block from the lists, 32 members at a time: a warp scatters its
// block's list entries into a 32 x 32 tile (row i, member), then lane k carries
// member k's column through the block's nodes in depth-first order.  Columns are independent, so the
// chunks of a wide separator run in different warps (blockIdx.y).  Bound:
// latency of the scattered list reads; 0.1 ms beside the product's 2 ms on
// the 264k-vertex graph.
__global__ void __launch_bounds__(32 * kClosureWarps) closure_kernel(BlockArgs A) {
  __shared__ unsigned s_row[kClosureWarps][kRows * 33];
  __shared__ int s_tw[kClosureWarps][kRows * 32];
  __shared__ unsigned char s_tl[kClosureWarps][kRows * 32];
  __shared__ int s_p[kClosureWarps][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int b = blockIdx.x * kClosureWarps + wid;
  if (b >= A.nblk) return;
  const int64_t m0 = A.moff[b];
  const int m = (int)(A.moff[b + 1] - m0);
  if ((int)blockIdx.y * 32 >= m) return;
  unsigned *row = s_row[wid];
  int *tw = s_tw[wid], *sp = s_p[wid];
  unsigned char *tl = s_tl[wid];
  const int64_t o = A.boff[b];
  const int R = (int)(A.boff[b + 1] - o), Rp = (R + 3) & ~3;
  const int dt = A.depth[A.blk_top[b]] - 1;
  int tc = 0;  // lane i: inner members of node i
  for (int i = 0; i < R; i++) {
    const int c = stage_inner(A, A.bnode[o + i], dt, tl + 32 * i, tw + 32 * i, lane);
    if (lane == i) tc = c;
  }
  int64_t lb = 0, le = 0;  // lane i: node i's list entries above the block
  if (lane < R) {
    const int v = A.bnode[o + lane];
    lb = A.pos_hash[v];
    le = A.pos_hash[v + 1] - 1 - tc;
  }
  __syncwarp();
  for (int k0 = blockIdx.y * 32; k0 < m; k0 += gridDim.y * 32) {
    const int kn = min(32, m - k0);
    const int p = k0 + lane < m ? A.bm_p[m0 + k0 + lane] : INT_MAX;
    sp[lane] = p;
    const int pfirst = __shfl_sync(0xffffffffu, p, 0), plast = __shfl_sync(0xffffffffu, p, kn - 1);
    for (int64_t a = lb, z = le; lane < R;) {  // first entry of node `lane` at or after the chunk
      if (a >= z) {
        lb = a;
        break;
      }
      const int64_t mid = (a + z) >> 1;
      if (__ldg(A.pos_pos + mid) < pfirst) a = mid + 1; else z = mid;
    }
    for (int i = 0; i < R; i++) row[i * 33 + lane] = kInf;
    __syncwarp();
    for (int i = 0; i < R; i++) {
      const int64_t e = __shfl_sync(0xffffffffu, lb, i) + lane;
      if (e >= __shfl_sync(0xffffffffu, le, i)) continue;
      const int q = __ldg(A.pos_pos + e);
      if (q > plast) continue;
      int x = 0, y = kn - 1;
      while (x < y) {
        const int mid = (x + y) >> 1;
        if (sp[mid] < q) x = mid + 1; else y = mid;
      }
      if (sp[x] == q) row[i * 33 + x] = (unsigned)__ldg(A.pos_w + e);
      else atomicCAS(A.err, 0, kErrNested);
    }
    __syncwarp();
    const int64_t out = A.soff[b] + (int64_t)k0 * Rp;
    for (int i = 1; i < R; i++) {
      unsigned r = row[i * 33 + lane];
      const int c = __shfl_sync(0xffffffffu, tc, i);
      for (int x = 0; x < c; x++) r = add_min((unsigned)tw[32 * i + x], row[tl[32 * i + x] * 33 + lane], r);
      row[i * 33 + lane] = r;
    }
    __syncwarp();
    for (int k = 0; k < kn; k++)
      if (lane < Rp) A.closed[out + k * Rp + lane] = lane < R ? row[lane * 33 + k] : kInf;
    __syncwarp();
  }
}

// W of every block and the nodes' ancestors inside it: a warp takes the block's
// nodes in depth-first order, lane a holding the entry for the node at place a.
// The matrix stays symmetric over finished pairs, so W between an inner
// neighbour w and a is one read whichever lies deeper.  Bound: a chain of up to
// 31 rows, 0.4 us each; it used to end every block of the fill (14 us of the 45 a
// narrow level took), here all blocks run side by side (0.39 ms on the
// 1M-vertex graph).
__global__ void __launch_bounds__(32 * kClosureWarps) inner_closure_kernel(BlockArgs A) {
  __shared__ unsigned s_M[kClosureWarps][kRows * 33];
  __shared__ int s_tw[kClosureWarps][kRows * 32];
  __shared__ unsigned char s_tl[kClosureWarps][kRows * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int b = blockIdx.x * kClosureWarps + wid;
  if (b >= A.nblk) return;
  unsigned *M = s_M[wid];
  int *tw = s_tw[wid];
  unsigned char *tl = s_tl[wid];
  const int64_t o = A.boff[b];
  const int R = (int)(A.boff[b + 1] - o), Rp = (R + 3) & ~3;
  const int m = (int)(A.moff[b + 1] - A.moff[b]);
  const int dt = A.depth[A.blk_top[b]] - 1;
  int tc = 0, par = 0;  // lane i: inner members of node i, its father's place
  int64_t pb = 0, pe = 0;
  if (lane < R) {
    const int v = A.bnode[o + lane];
    pb = A.pos_hash[v];
    pe = A.pos_hash[v + 1] - 2;
    if (lane > 0) par = A.loc_of[A.father[v]];
  }
#pragma unroll 4
  for (int i = 0; i < R; i++) {  // stage_inner for every node, several in flight
    const int64_t e = __shfl_sync(0xffffffffu, pe, i) - lane;
    const bool in = e >= __shfl_sync(0xffffffffu, pb, i) && __ldg(A.pos_pos + e) >= dt;
    if (in) {
      tl[32 * i + lane] = A.loc_of[__ldg(A.pos_id + e)];
      tw[32 * i + lane] = __ldg(A.pos_w + e);
    }
    const int c = __popc(__ballot_sync(0xffffffffu, in));
    if (lane == i) tc = c;
  }
  for (int i = 0; i < kRows; i++) M[i * 33 + lane] = kInf;
  __syncwarp();
  unsigned anc = 0;
  for (int i = 1; i < R; i++) {
    const int pi = __shfl_sync(0xffffffffu, par, i);
    const unsigned ai = __shfl_sync(0xffffffffu, anc, pi) | (1u << pi);
    if (lane == i) anc = ai;
    unsigned r = kInf;
    const int c = __shfl_sync(0xffffffffu, tc, i);
#pragma unroll 4
    for (int x = 0; x < c; x++) {
      const int w = tl[32 * i + x];
      r = add_min((unsigned)tw[32 * i + x], w == lane ? 0u : M[w * 33 + lane], r);
    }
    __syncwarp();
    if ((ai >> lane) & 1u) {
      M[i * 33 + lane] = r;
      M[lane * 33 + i] = r;
    }
    __syncwarp();
  }
  if (lane < R) A.anc[o + lane] = anc;
  unsigned *out = A.closed + A.soff[b] + (int64_t)m * Rp;
  for (int c = 0; c < R; c++)
    if (lane < Rp) out[c * Rp + lane] = M[lane * 33 + c];  // rows past R: no entry
}

// ------------------------------------------------------------ the weights
//
// With the order and the lists known (symbolic.cu), the shortcut weights are
// an elimination over the blocks, leaves to root: a block's rows hold the
// weights between its nodes and its nodes' upper neighbours, first the input
// arcs and what the blocks below add; eliminating the nodes deepest first
// gives row(u)[x] = min(row(u)[x], row(i)[u] + row(i)[x]) for u, x upper
// neighbours of i.  Inside the block that is a 32 x 32 triangle; each further
// column is a triangular solve of its own; and what the block adds between
// two of its top's members x, y -- min over its nodes i of row(i)[x] +
// row(i)[y] -- is a min-plus product that goes to the parent block by
// atomicMin.  Every sum is one the list kernels take, with the row of the
// vertex eliminated first (arcs' weights may differ by direction).
//
// Repeated arcs: a row takes the smallest, except in the global order, whose
// lists keep the first of equal ids (unordered_map::emplace).

// Each member's column in the parent block (its place there, encoded ~place,
// or its index among the parent's members), and how many tasks a parent waits
// for.  One warp per block.
__global__ void parent_columns_kernel(BlockArgs B, const int64_t *wtask0, int *blk_up, int *bm_up, int *pend) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; b < B.nblk;
       b += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int top = B.blk_top[b], f = B.father[top];
    const int p = f < 0 ? -1 : B.blk_of[f];
    if (lane == 0) {
      blk_up[b] = p;
      if (p >= 0) atomicAdd(pend + p, (int)(wtask0[b + 1] - wtask0[b]));
    }
    if (p < 0) continue;
    const int64_t pb = B.pos_hash[top], m0 = B.moff[b], pm0 = B.moff[p];
    const int m = (int)(B.moff[b + 1] - m0), pm = (int)(B.moff[p + 1] - pm0);
    const int pdt = B.depth[B.blk_top[p]] - 1;
    for (int k = lane; k < m; k += 32) {
      const int q = B.pos_pos[pb + k];
      int code;
      if (q >= pdt) {
        code = ~(int)B.loc_of[B.pos_id[pb + k]];
      } else {
        int lo = 0, hi = pm;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (B.bm_p[pm0 + mid] < q) lo = mid + 1; else hi = mid;
        }
        if (lo >= pm || B.bm_p[pm0 + lo] != q) {
          atomicCAS(B.err, 0, kErrNested);
          lo = 0;
        }
        code = lo;
      }
      bm_up[m0 + k] = code;
    }
  }
}

__global__ void weight_tasks_kernel(const int *mem, int *ntask, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblk; b += gridDim.x * blockDim.x) {
    const int nt = b < nblk ? max(1, (mem[b] + 63) / 64) : 0;
    ntask[b] = nt * (nt + 1) / 2;
  }
}

// Entries of a block's update triangle: none where no block lies below.
__global__ void update_sizes_kernel(const int *mem, const int *pend, int64_t *cells, int nblk) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblk; b += gridDim.x * blockDim.x)
    cells[b] = b < nblk && pend[b] > 0 ? (int64_t)mem[b] * (mem[b] - 1) / 2 : 0;
}

__global__ void mark_kernel(const int *verts, int n, unsigned char *flag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flag[verts[i]] = 1;
}

constexpr int64_t kOnce = int64_t(1) << 62;  // of a cell that only the first of its arcs may enter

// The cell every arc v -> x with x an upper neighbour of v starts from; -1 for
// the other direction.  A thread per arc (a thread per vertex is as slow as its
// longest list): a warp finds the tails of its first and last arc, its lanes
// theirs between the two.
__global__ void arc_cells_kernel(BlockArgs B, const int *adj_off, const int *adj_v, const unsigned char *global,
                                 int64_t *arc_cell, unsigned *first, int n, int64_t m) {
  const int lane = threadIdx.x & 31;
  auto tail = [&](int64_t e, int lo, int hi) {  // the last list that starts at or before e
    while (lo < hi) {
      const int mid = lo + (hi - lo + 1) / 2;
      if (adj_off[mid] <= e) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~int64_t(31); base < m;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int end = tail(lane == 0 ? base : min(base + 31, m - 1), 0, n - 1);
    const int v0 = __shfl_sync(0xffffffffu, end, 0), v1 = __shfl_sync(0xffffffffu, end, 31);
    const int64_t e = base + lane;
    if (e >= m) continue;
    const int v = tail(e, v0, v1), x = adj_v[e], p = B.depth[x] - 1;
    int64_t cell = -1;
    if (p < B.depth[v] - 1) {
      const int b = B.blk_of[v];
      const int64_t m0 = B.moff[b];
      const int mem = (int)(B.moff[b + 1] - m0), Rp = ((int)(B.boff[b + 1] - B.boff[b]) + 3) & ~3;
      int c;
      if (p >= B.depth[B.blk_top[b]] - 1) {
        c = mem + B.loc_of[x];
      } else {
        int lo = 0, hi = mem;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (B.bm_p[m0 + mid] < p) lo = mid + 1; else hi = mid;
        }
        c = lo;
        if (lo >= mem || B.bm_p[m0 + lo] != p) {
          atomicCAS(B.err, 0, kErrNested);
          c = -1;
        }
      }
      if (c >= 0) {
        cell = B.soff[b] + (int64_t)c * Rp + B.loc_of[v];
        if (global[v]) {
          first[cell] = kInf;
          cell |= kOnce;
        }
      }
    }
    arc_cell[e] = cell;
  }
}

// Of the repeated arcs of the global order the first one stays: `first` takes
// the smallest place per cell, then the others are dropped.
__global__ void first_arcs_kernel(const int64_t *arc_cell, unsigned *first, int64_t m) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = arc_cell[e];
    if (c >= 0 && (c & kOnce)) atomicMin(first + (c & ~kOnce), (unsigned)e);
  }
}

__global__ void drop_arcs_kernel(int64_t *arc_cell, const unsigned *first, int64_t m) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = arc_cell[e];
    if (c >= 0 && (c & kOnce)) arc_cell[e] = first[c & ~kOnce] == (unsigned)e ? c & ~kOnce : -1;
  }
}

__global__ void fill_inf_kernel(unsigned *p, int64_t n) {
  const int64_t q = n >> 2;
  uint4 *p4 = reinterpret_cast<uint4 *>(p);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < q; i += (int64_t)gridDim.x * blockDim.x)
    p4[i] = make_uint4(kInf, kInf, kInf, kInf);
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) p[4 * q + threadIdx.x] = kInf;
}

__global__ void scatter_arcs_kernel(const int64_t *arc_cell, const int *w, unsigned *cells, int64_t m) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = arc_cell[e];
    if (c >= 0) atomicMin(cells + c, (unsigned)w[e]);
  }
}

struct WeightArgs {
  BlockArgs B;
  const int *blk_up, *bm_up;
  const int64_t *uoff;
  unsigned *upd;  // per block with blocks below it: pairs (x < y) of members at y (y - 1) / 2 + x
  const int *task_blk;
  const int64_t *task0;
  int ntasks;
  int *pending, *next;
  long long spin_limit;
};

// A CTA takes a 64 x 64 tile of a block's update triangle, blocks from the
// deepest up (a block's tasks wait for the tasks of the blocks below it).  One
// warp eliminates the block's triangle and closes it: C(i, u) is the least sum
// of weights down a chain i > .. > u of the block's nodes.  With C a column's
// elimination is a product, col(u) = min over i >= u of C(i, u) + col(i), and so
// is its closure, S(i) = min over u <= i of C(i, u) + col(u).  Then the CTA forms
// the tile; the diagonal tiles write their columns back, direct and closed,
// after the parent has been told.  A tile may read columns another has already
// written back, which solves to the same values (C is closed).
//
// Bound: the chain of blocks, 13 us each: 1 for the loads, 5 for the triangle, 2
// for the columns, 1.5 for the tile and 3 for its atomics (66 blocks of a
// 264k-vertex graph 1.48 -> 1.18 ms, 118 of a 1M-vertex one 4.55 -> 3.45).  The
// loops over nodes stay loops: as straight-line code (6 us for the triangle, 4.5
// for the columns) they ran at the speed of instruction fetches.  Four warps
// to the triangle lose more in barriers (1.39 and 3.98 ms).
__global__ void __launch_bounds__(128, 4) weights_kernel(WeightArgs A) {
  __shared__ __align__(16) unsigned s_L[kRows * 36];   // row i of the triangle, columns moved up by kRows - 1 - i
  __shared__ __align__(16) unsigned s_C[kRows * 36];   // C(i, u), [i][u] and [u][i]
  __shared__ __align__(16) unsigned s_Ct[kRows * 36];
  __shared__ __align__(16) unsigned s_P[2][kRows * 68];
  __shared__ int s_up[2][64];
  __shared__ int64_t s_pso, s_puo;  // the parent's cells, triangle, members and row padding
  __shared__ int s_pm, s_pRp;
  __shared__ int s_t, s_flag;
  const BlockArgs &B = A.B;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_t = atomicAdd(A.next, 1);
    __syncthreads();
    if (s_t >= A.ntasks) return;
    const int t = A.ntasks - 1 - s_t;  // deepest blocks first
    const int b = __ldg(A.task_blk + t);
    int sub = t - (int)__ldg(A.task0 + b);
    const int64_t bo = __ldg(B.boff + b), m0 = __ldg(B.moff + b), so = __ldg(B.soff + b);
    const int R = (int)(__ldg(B.boff + b + 1) - bo), Rp = (R + 3) & ~3;
    const int m = (int)(__ldg(B.moff + b + 1) - m0);
    int X = 0, Y = 0;  // tile (X, Y), X <= Y, numbered Y (Y + 1) / 2 + X
    Y = (int)((sqrtf(8.0f * (float)sub + 1.0f) - 1.0f) * 0.5f);
    while ((Y + 1) * (Y + 2) / 2 <= sub) Y++;
    while (Y * (Y + 1) / 2 > sub) Y--;
    X = sub - Y * (Y + 1) / 2;
    const int p = __ldg(A.blk_up + b);
    const bool diag = X == Y;
    if (p >= 0) {
      const int k = 64 * (tid < 64 ? X : Y) + (tid & 63);
      s_up[tid >> 6][tid & 63] = k < m ? __ldg(A.bm_up + m0 + k) : 0;
      if (tid == 32) {
        s_pso = __ldg(B.soff + p);
        s_puo = __ldg(A.uoff + p);
        s_pm = (int)(__ldg(B.moff + p + 1) - __ldg(B.moff + p));
        s_pRp = ((int)(__ldg(B.boff + p + 1) - __ldg(B.boff + p)) + 3) & ~3;
      }
    }
    if (tid == 0) {
      int ok = 1;
      const int *flag = A.pending + b;
      const long long t0 = clock64();
      while (ld_acquire(flag) != 0) {
        if (ld_relaxed(B.err) != 0 || clock64() - t0 > A.spin_limit) {
          atomicCAS(B.err, 0, kErrWait);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
      s_flag = ok;
    }
    __syncthreads();
    if (!s_flag) return;
    unsigned *const cells = B.direct + so;
    // loads first: the update triangle's tile (what the blocks below added),
    // the columns, one per lane, and the block's own triangle
    const int xg = tid & 15, yg = tid >> 4;  // this thread's patch: 4 x by 8 y, lanes along x
    const int x0 = 64 * X + 4 * xg, y0 = 64 * Y + 8 * yg;
    const int half = wid >> 1;  // warps 0, 1: X's columns; 2, 3: Y's
    const int k = 64 * (half ? Y : X) + 32 * (wid & 1) + lane;
    const bool solve = !(diag && half) && 64 * (half ? Y : X) + 32 * (wid & 1) < m;
    unsigned acc[8][4];
    {
      const int64_t uo = __ldg(A.uoff + b);
      const bool below = __ldg(A.uoff + b + 1) > uo;
#pragma unroll
      for (int y = 0; y < 8; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const int xx = x0 + x, yy = y0 + y;
          acc[y][x] = below && yy < m && xx < yy ? __ldcg(A.upd + uo + (int64_t)yy * (yy - 1) / 2 + xx) : kInf;
        }
    }
    unsigned col[kRows];
    if (solve) {
      const uint4 *src = reinterpret_cast<const uint4 *>(cells + (int64_t)min(k, m - 1) * Rp);
#pragma unroll
      for (int q = 0; q < kRows / 4; q++) {
        const uint4 x = 4 * q < Rp && k < m ? __ldcg(src + q) : make_uint4(kInf, kInf, kInf, kInf);
        col[4 * q] = x.x;
        col[4 * q + 1] = x.y;
        col[4 * q + 2] = x.z;
        col[4 * q + 3] = x.w;
      }
    }
    // the block's own triangle, by the last warp (which on the diagonal has no
    // columns): lane i holds row i, whose columns move up a register per node
    // so that the node's own column is always the last.  Node w's row is final
    // when its turn comes; rows above it (lanes below w) take the elimination's
    // update, rows below it (lanes above w) extend their chains through w.
    if (wid == 3) {
      unsigned row[kRows];
#pragma unroll
      for (int q = 0; q < kRows; q++) {
        const int c = q - (kRows - R);
        row[q] = c >= 0 && c < lane && lane < R ? __ldcg(cells + (int64_t)(m + c) * Rp + lane) : kInf;
      }
      for (int w = R; w < Rp; w++) s_C[lane * 36 + w] = kInf;  // the rows' padding
#pragma unroll 1
      for (int w = R - 1; w >= 0; w--) {
        unsigned *const piv = s_L + w * 36;
        if (lane == w) {
#pragma unroll
          for (int q = 0; q < kRows / 4; q++)
            reinterpret_cast<uint4 *>(piv)[q] = make_uint4(row[4 * q], row[4 * q + 1], row[4 * q + 2], row[4 * q + 3]);
        }
        const unsigned chain = lane > w ? row[kRows - 1] : lane == w ? 0 : kInf;  // C(lane, w)
        s_C[lane * 36 + w] = chain;
        s_Ct[w * 36 + lane] = chain;
        __syncwarp();
        const unsigned by = lane < w ? piv[lane + kRows - 1 - w] : lane > w ? chain : kInf;
#pragma unroll
        for (int q = kRows / 4 - 1; q >= 0; q--) {
          const uint4 x = reinterpret_cast<const uint4 *>(piv)[q];
          if (q < kRows / 4 - 1) row[4 * q + 4] = add_min(by, x.w, row[4 * q + 3]);
          row[4 * q + 3] = add_min(by, x.z, row[4 * q + 2]);
          row[4 * q + 2] = add_min(by, x.y, row[4 * q + 1]);
          row[4 * q + 1] = add_min(by, x.x, row[4 * q]);
        }
        row[0] = kInf;
      }
    }
    if (solve) {
#pragma unroll
      for (int i = 0; i < kRows; i++) s_P[half][i * 68 + 32 * (wid & 1) + lane] = col[i];
    }
    __syncthreads();
    // the tile's columns
    unsigned *const mine = s_P[half] + 32 * (wid & 1) + lane;
    if (solve) {
#pragma unroll 1
      for (int i = 1; i < R; i++) {  // col holds row i itself: C(i, i) = 0
        const unsigned x = mine[i * 68];
#pragma unroll
        for (int q = 0; q < kRows / 4; q++) {
          const uint4 y = *reinterpret_cast<const uint4 *>(s_C + i * 36 + 4 * q);
          col[4 * q] = add_min(y.x, x, col[4 * q]);
          col[4 * q + 1] = add_min(y.y, x, col[4 * q + 1]);
          col[4 * q + 2] = add_min(y.z, x, col[4 * q + 2]);
          col[4 * q + 3] = add_min(y.w, x, col[4 * q + 3]);
        }
      }
#pragma unroll
      for (int i = 0; i < kRows; i++) mine[i * 68] = col[i];
    }
    __syncthreads();
    if (p >= 0 && x0 < m && y0 < m) {
      const unsigned *px = s_P[0] + 4 * xg, *py = s_P[diag ? 0 : 1] + 8 * yg;
#pragma unroll 2
      for (int i = 0; i < R; i++) {
        const uint4 a = *reinterpret_cast<const uint4 *>(px + i * 68);
        const uint4 c = *reinterpret_cast<const uint4 *>(py + i * 68);
        const uint4 d = *reinterpret_cast<const uint4 *>(py + i * 68 + 4);
        const unsigned yv[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
        for (int y = 0; y < 8; y++) {
          acc[y][0] = add_min(yv[y], a.x, acc[y][0]);
          acc[y][1] = add_min(yv[y], a.y, acc[y][1]);
          acc[y][2] = add_min(yv[y], a.z, acc[y][2]);
          acc[y][3] = add_min(yv[y], a.w, acc[y][3]);
        }
      }
      const int64_t pso = s_pso, puo = s_puo;
      const int pm = s_pm, pRp = s_pRp;
#pragma unroll
      for (int y = 0; y < 8; y++) {
        const int yy = y0 + y;
        if (yy >= m) break;
        const int cy = s_up[1][8 * yg + y];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const int xx = x0 + x;
          if (xx >= yy) break;
          const unsigned v = acc[y][x];
          if (v >= kInf) continue;
          const int cx = s_up[0][4 * xg + x];
          unsigned *dst;
          if (cy < 0)  // y is the parent's own node, eliminated before x
            dst = B.direct + pso + (int64_t)(cx < 0 ? pm + ~cx : cx) * pRp + ~cy;
          else
            dst = A.upd + puo + (int64_t)cy * (cy - 1) / 2 + cx;
          atomicMin(dst, v);
        }
      }
    }
    __syncthreads();
    if (p >= 0 && tid == 0) {
      __threadfence();
      atomicSub(A.pending + p, 1);
    }
    // what only later kernels read
    if (sub == 0)
      for (int i = tid; i < R * Rp; i += 128) {
        const int c = i / Rp, r = i - c * Rp;
        if (r > c && r < R) cells[(int64_t)(m + c) * Rp + r] = s_L[r * 36 + c + kRows - 1 - r];
      }
    if (diag && solve && k < m) {
      uint4 *dst = reinterpret_cast<uint4 *>(cells + (int64_t)k * Rp);
      uint4 *cls = reinterpret_cast<uint4 *>(B.closed + so + (int64_t)k * Rp);
#pragma unroll
      for (int i = 0; i < kRows; i++) col[i] = mine[i * 68];
#pragma unroll
      for (int q = 0; q < kRows / 4; q++)
        if (4 * q < Rp) dst[q] = make_uint4(col[4 * q], col[4 * q + 1], col[4 * q + 2], col[4 * q + 3]);
#pragma unroll 1
      for (int u = 0; u < R - 1; u++) {
        const unsigned x = mine[u * 68];
#pragma unroll
        for (int q = 0; q < kRows / 4; q++) {
          const uint4 y = *reinterpret_cast<const uint4 *>(s_Ct + u * 36 + 4 * q);
          col[4 * q] = add_min(y.x, x, col[4 * q]);
          col[4 * q + 1] = add_min(y.y, x, col[4 * q + 1]);
          col[4 * q + 2] = add_min(y.z, x, col[4 * q + 2]);
          col[4 * q + 3] = add_min(y.w, x, col[4 * q + 3]);
        }
      }
#pragma unroll
      for (int q = 0; q < kRows / 4; q++)
        if (4 * q < Rp) cls[q] = make_uint4(col[4 * q], col[4 * q + 1], col[4 * q + 2], col[4 * q + 3]);
    }
  }
}

// Every list entry's weight, in the lists and in the position arrays.  One
// warp per vertex.
__global__ void list_weights_kernel(BlockArgs B, const int *pos_src, const int64_t *list_off, int *list_w, int *pos_w,
                                    int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; v < n;
       v += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int b = B.blk_of[v], i = B.loc_of[v];
    const int64_t m0 = B.moff[b], so = B.soff[b];
    const int m = (int)(B.moff[b + 1] - m0), Rp = ((int)(B.boff[b + 1] - B.boff[b]) + 3) & ~3;
    const int dt = B.depth[B.blk_top[b]] - 1;
    const int64_t pb = B.pos_hash[v], pe = B.pos_hash[v + 1];
    for (int64_t e = pb + lane; e < pe; e += 32) {
      const int src = pos_src[e];
      if (src < 0) {
        pos_w[e] = 0;
        continue;
      }
      const int p = B.pos_pos[e];
      int c;
      if (p >= dt) {
        c = m + B.loc_of[B.pos_id[e]];
      } else {
        int lo = 0, hi = m - 1;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (__ldg(B.bm_p + m0 + mid) < p) lo = mid + 1; else hi = mid;
        }
        c = lo;
      }
      const int w = (int)B.direct[so + (int64_t)c * Rp + i];
      pos_w[e] = w;
      list_w[list_off[v] + src] = w;
    }
  }
}

// ------------------------------------------------------------ the product

struct FillKernelArgs {
  BlockArgs B;
  int *dis;
  const int64_t *hld_row;  // heavy paths, top to bottom: the row offset of the node at each position
  const int64_t *seg_off;  // root-path segments per node
  const int *seg_top, *seg_pos;
  const int *task_blk;
  const int64_t *task0;
  const int *tcols;
  int ntasks;
  int *done, *count, *next;
  const int *mslot;  // blocks of several tasks: their in-block matrix in mbuf, combined by atomicMin
  unsigned *mbuf;
  long long spin_limit;
  int max_segs;
  unsigned long long *trace_t;  // non-null (GPUH2H_TRACE): each node's publish time, ns
};

// A CTA of four warps takes tasks (a block, a range of columns) in block
// order, waits for the father block's flag, and sweeps its
// columns 64 at a time and the top's members 32 at a time: the second factor
// E goes through registers into shared memory one step ahead (so a step's
// loads overlap the product before it), every thread owns a 4 x 4 patch of
// the 32 x 64 result.  A completed tile adds its columns' part of the matrix
// inside the block, whose weights came to shared memory with the tile; the last
// task of a block to finish writes that matrix and publishes the block.  Rows produced in the launch are
// read through L2 (ld.global.cg).  A member at or below a tile is a row of it,
// 16 columns of eight members to a warp request; of a member above it, column
// p_u of each of the tile's ancestors, where lanes along the members read one
// ancestor's row at neighbouring positions.  The product holds the next
// member's operands while it sums: with 57 clocks a member for 32 of sums it
// was the longest part of a narrow step.  1M-vertex graph: 12.9 ms with one
// mapping of loads and without the operands ahead, 12.1 with both (with the tasks
// and the block order of the time); each alone
// gains nothing.
// Five CTAs per SM (four: 12.3 ms; six hold 80 registers and spill).  Loads two
// or three steps ahead, with 128 registers, gain nothing: a step waits 270
// clocks of 4,000 for them.
__global__ void __launch_bounds__(128, 5) block_fill_kernel(FillKernelArgs A) {
  extern __shared__ __align__(16) int s_seg[];
  __shared__ __align__(16) unsigned s_E[(kMembers + 1) * kEStride];  // + 1: the product reads a row ahead
  __shared__ __align__(16) unsigned s_S[(kMembers + 1) * kRows];
  __shared__ __align__(16) int64_t s_arow[2][kCols];
  __shared__ __align__(16) unsigned s_O[kCols * 36];   // a finished tile, [column][row]
  __shared__ int64_t s_mrow[2][kMembers];  // a step's members: rows and positions (-1: none)
  __shared__ int s_mp[2][kMembers];
  __shared__ int64_t s_rowoff[kRows];
  __shared__ int s_kb[kMaxTiles + 1];  // first member at or after each tile's first column
  __shared__ __align__(16) unsigned s_D[kCols * kRows];  // a tile's members: S and positions
  __shared__ int s_pd[kCols];
  __shared__ int s_dcol[kRows];
  __shared__ unsigned s_anc[kRows];
  __shared__ int s_t, s_flag;
  const BlockArgs &B = A.B;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int *const s_top = s_seg, *const s_pos = s_seg + A.max_segs;
  const int em = lane >> 2, ec = 16 * wid + 4 * (lane & 3);  // loads members em, em + 8, .. at columns ec .. ec + 3
  const int ry = tid >> 4, cx = tid & 15;               // its patch of the result
  for (;;) {
    __syncthreads();  // the last task's shared memory is free
    if (tid == 0) s_t = atomicAdd(A.next, 1);
    __syncthreads();
    const int t = s_t;
    if (t >= A.ntasks) return;
    const int b = __ldg(A.task_blk + t);
    const int64_t task0 = __ldg(A.task0 + b);
    const int ntask = (int)(__ldg(A.task0 + b + 1) - task0);
    const int tc = __ldg(A.tcols + b);
    const int top = __ldg(B.blk_top + b);
    const int dt = __ldg(B.depth + top) - 1;  // columns above the block
    const int64_t bo = __ldg(B.boff + b), m0 = __ldg(B.moff + b), so = __ldg(B.soff + b);
    const int R = (int)(__ldg(B.boff + b + 1) - bo), Rp = (R + 3) & ~3;
    const int m = (int)(__ldg(B.moff + b + 1) - m0);
    const int c0 = (int)(t - task0) * tc, c1 = min(dt, c0 + tc);
    const int64_t sb = __ldg(A.seg_off + top);
    const int ns = (int)(__ldg(A.seg_off + top + 1) - sb);
    for (int i = tid; i < ns; i += 128) {
      s_top[i] = __ldg(A.seg_top + sb + i);
      s_pos[i] = __ldg(A.seg_pos + sb + i);
    }
    if (tid < R) {
      const int v = __ldg(B.bnode + bo + tid);
      s_rowoff[tid] = __ldg(B.drow + v);
      s_dcol[tid] = __ldg(B.depth + v) - 1;
      s_anc[tid] = B.anc[bo + tid];
    }
    const int my = tid >> 3, mx = tid & 7;  // this thread's 2 x 4 patch of the in-block matrix
    if (tid <= (c1 - c0 + kCols - 1) / kCols) {
      const int j = min(c0 + kCols * tid, c1);
      int lo = 0, hi = m;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(B.bm_p + m0 + mid) < j) lo = mid + 1; else hi = mid;
      }
      s_kb[tid] = lo;
    }
    __syncthreads();
    int seg = 0;  // the root-path segment of this thread's last column: they only move on
    {
      int hi = ns - 1;
      while (seg < hi) {
        const int mid = (seg + hi + 1) >> 1;
        if (s_top[mid] <= c0 + tid + 1) seg = mid; else hi = mid - 1;
      }
    }
    auto ancestor_row = [&](int j) -> int64_t {  // row offset of the ancestor at depth j + 1
      if (j >= c1) return 0;
      while (seg + 1 < ns && s_top[seg + 1] <= j + 1) seg++;
      return __ldg(A.hld_row + s_pos[seg] + (j + 1 - s_top[seg]));
    };
    s_arow[tid >> 6][tid & 63] = ancestor_row(c0 + tid);
    const int nchunk = (m + kMembers - 1) / kMembers, ntile = (c1 - c0 + kCols - 1) / kCols;
    const int nsteps = c1 > c0 ? nchunk * ntile : 0;
    uint4 eb[4], sbuf[2];
    auto issue_s = [&](const unsigned *src, int k0) {
      const int nq = min(kMembers, m - k0) * (Rp >> 2);
      const uint4 *p = reinterpret_cast<const uint4 *>(src + so + (int64_t)k0 * Rp);
      sbuf[0] = tid < nq ? __ldg(p + tid) : make_uint4(kInf, kInf, kInf, kInf);
      sbuf[1] = tid + 128 < nq ? __ldg(p + tid + 128) : make_uint4(kInf, kInf, kInf, kInf);
    };
    auto store_s = [&]() {
      reinterpret_cast<uint4 *>(s_S)[tid] = sbuf[0];
      reinterpret_cast<uint4 *>(s_S)[tid + 128] = sbuf[1];
    };
    int p2 = -1;  // warp 0: a member of the step after the next
    int64_t row2 = 0;
    auto load_member = [&](int k0) {
      const int k = k0 + lane;
      p2 = k < m ? __ldg(B.bm_p + m0 + k) : -1;
      row2 = k < m ? __ldg(B.bm_row + m0 + k) : 0;
    };
    // members k0 .. k0 + kn of a step, in buffer `mb`, at the columns of tile T.
    // All above the tile (p_u before its columns): a lane per member, so that a
    // request reads one ancestor's row at consecutive positions.  Otherwise a
    // warp takes 16 columns of eight members at a time, rows of 64 bytes.
    bool along = false;  // eb holds a member per lane
    auto issue_e = [&](int T, int mb, int k0, int kn) {
      const int J0 = c0 + T * kCols;
      along = k0 + kn <= s_kb[T];
      if (along) {
        const int *col = A.dis + (lane < kn ? s_mp[mb][lane] : 0);
        const int64_t *ar = s_arow[T & 1] + 16 * wid;
#pragma unroll
        for (int g = 0; g < 4; g++) {
          if (J0 + 16 * wid + 4 * g < c1) {  // past column c1 the ancestor's row is 0: a read that counts for nothing
            eb[g].x = (unsigned)__ldcg(col + ar[4 * g]);
            eb[g].y = (unsigned)__ldcg(col + ar[4 * g + 1]);
            eb[g].z = (unsigned)__ldcg(col + ar[4 * g + 2]);
            eb[g].w = (unsigned)__ldcg(col + ar[4 * g + 3]);
          }
        }
        return;
      }
      const int J = J0 + ec;
      if (k0 >= s_kb[T + 1]) {  // all below it
#pragma unroll
        for (int g = 0; g < 4; g++)
          if (8 * g + em < kn && J < c1) eb[g] = __ldcg(reinterpret_cast<const uint4 *>(A.dis + s_mrow[mb][8 * g + em] + J));
        return;
      }
      const int64_t *ar = s_arow[T & 1] + ec;
#pragma unroll
      for (int g = 0; g < 4; g++) {
        uint4 e = make_uint4(kInf, kInf, kInf, kInf);
        if (8 * g < kn && J < c1) {
          const int k = 8 * g + em, p = s_mp[mb][k];
          const int *row = A.dis + s_mrow[mb][k];
          if (p >= J + 4) {
            e = __ldcg(reinterpret_cast<const uint4 *>(row + J));
          } else if (p >= 0) {
            const int *col = A.dis + p;
            unsigned x[4];
#pragma unroll
            for (int c = 0; c < 4; c++)
              x[c] = (unsigned)(J + c > p ? __ldcg(col + ar[c]) : J + c == p ? 0 : __ldcg(row + J + c));
            e = make_uint4(x[0], x[1], x[2], x[3]);
          }
        }
        eb[g] = e;
      }
    };
    // the members whose positions lie inside a tile: their rows of S go to
    // shared memory beside the tile's product (one chunk: they are in s_S)
    auto issue_d = [&](int T) {
      const int kb = s_kb[T], nd = s_kb[T + 1] - kb;
      const unsigned *src = B.closed + so + (int64_t)kb * Rp;
      for (int i = tid; i < nd * (Rp >> 2); i += 128) cp_async16(s_D + 4 * i, src + 4 * i);
      if (tid < nd) cp_async4(s_pd + tid, B.bm_p + m0 + kb + tid);
    };
    unsigned mm[2][4];  // in-block matrix: W, then the part over members above the block
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int a = 4 * mx + c;
      const uint2 w = t == task0 && a < R && 2 * my < Rp
                          ? *reinterpret_cast<const uint2 *>(B.closed + so + (int64_t)(m + a) * Rp + 2 * my)
                          : make_uint2(kInf, kInf);
      mm[0][c] = w.x;
      mm[1][c] = w.y;
    }
    if (nsteps > 0) {
      issue_s(B.closed, 0);
      if (nchunk > 1 && R > 1) issue_d(0);
      if (wid < 2 && wid < nchunk) {  // the first two steps' members
        load_member(wid * kMembers);
        s_mp[wid][lane] = p2;
        s_mrow[wid][lane] = row2;
      }
    }
    if (tid == 0) {
      int ok = 1;
      const int f = __ldg(B.father + top);
      if (f >= 0) {
        const int *flag = A.done + __ldg(B.blk_of + f);
        const long long t0 = clock64();
        while (ld_acquire(flag) == 0) {
          if (ld_relaxed(B.err) != 0 || clock64() - t0 > A.spin_limit) {
            atomicCAS(B.err, 0, kErrWait);
            ok = 0;
            break;
          }
          __nanosleep(32);
        }
      }
      s_flag = ok;
    }
    __syncthreads();
    if (!s_flag) return;
    if (nsteps > 0) {
      issue_e(0, 0, 0, min(kMembers, m));
    }
    unsigned acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) acc[r][c] = kInf;
    int64_t arow_next = 0;  // threads below 64: the column's ancestor row two tiles ahead
    for (int s = 0, T = 0, ch = 0, ch2 = 2 % max(nchunk, 1); s < nsteps; s++) {
#pragma unroll
      for (int g = 0; g < 4; g++)
        *reinterpret_cast<uint4 *>(along ? s_E + lane * kEStride + 16 * wid + 4 * g : s_E + (8 * g + em) * kEStride + ec) = eb[g];
      if (nchunk > 1 || s == 0) store_s();
      if (nchunk > 1 && s > 0 && wid == 0) {
        s_mp[(s + 1) & 1][lane] = p2;
        s_mrow[(s + 1) & 1][lane] = row2;
      }
      if (ch == 0 && T > 0 && tid < kCols) s_arow[(T + 1) & 1][tid] = arow_next;
      __syncthreads();
      const int kn = min(kMembers, m - ch * kMembers);
      int nT = T, nch = ch + 1;
      if (nch == nchunk) {
        nch = 0;
        nT++;
      }
      if (s + 1 < nsteps) {
        issue_e(nT, nchunk > 1 ? (s + 1) & 1 : 0, nch * kMembers, min(kMembers, m - nch * kMembers));
        if (nchunk > 1) {
          issue_s(B.closed, nch * kMembers);
          if (wid == 0) load_member(ch2 * kMembers);
          if (++ch2 == nchunk) ch2 = 0;
        }
      }
      if (ch == 0 && T > 0 && nchunk > 1 && R > 1) issue_d(T);
      if (ch == 0 && tid < kCols) arow_next = ancestor_row(c0 + (T + 2) * kCols + tid);
      if (4 * ry < Rp) {
        const unsigned *pe = s_E + 4 * cx, *ps = s_S + 4 * ry;
        uint4 e = *reinterpret_cast<const uint4 *>(pe), w = *reinterpret_cast<const uint4 *>(ps);
#pragma unroll 4
        for (int k = 0; k < kn; k++) {  // the next member's row is on its way during this one's sums
          pe += kEStride;
          ps += Rp;
          const uint4 en = *reinterpret_cast<const uint4 *>(pe), wn = *reinterpret_cast<const uint4 *>(ps);
          const unsigned wr[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int r = 0; r < 4; r++) {
            acc[r][0] = add_min(wr[r], e.x, acc[r][0]);
            acc[r][1] = add_min(wr[r], e.y, acc[r][1]);
            acc[r][2] = add_min(wr[r], e.z, acc[r][2]);
            acc[r][3] = add_min(wr[r], e.w, acc[r][3]);
          }
          e = en;
          w = wn;
        }
      }
      const int kb = s_kb[T], ke = nch == 0 ? s_kb[T + 1] : kb;  // members inside a completed tile
      if (nch == 0) {  // the tile is complete
        const int j = c0 + T * kCols + 4 * cx;
        if (kb < ke && R > 1) {
#pragma unroll
          for (int c = 0; c < 4; c++)
            *reinterpret_cast<uint4 *>(s_O + (4 * cx + c) * 36 + 4 * ry) =
                make_uint4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int i = 4 * ry + r;
          if (i < R && j < c1) {
            int *out = A.dis + s_rowoff[i] + j;
            if (j + 4 <= c1) {
              *reinterpret_cast<uint4 *>(out) = make_uint4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
            } else {
#pragma unroll
              for (int c = 0; c < 4; c++)
                if (j + c < c1) out[c] = (int)acc[r][c];
            }
          }
#pragma unroll
          for (int c = 0; c < 4; c++) acc[r][c] = kInf;
        }
        cp_async_wait();
      }
      __syncthreads();
      // columns inside the block, for nodes i below a (both in the block): the
      // way over a member u takes column p_u of row a, which this tile has just
      // completed (the next tile is not written before the next barrier)
      if (R > 1 && 2 * my < Rp) {
        const int J = c0 + T * kCols;
        const unsigned *pd = (nchunk > 1 ? s_D : s_S + kb * Rp) + 2 * my;
        const int *pp = nchunk > 1 ? s_pd : s_mp[0] + kb;
#pragma unroll 4
        for (int k = 0; k < ke - kb; k++) {
          const uint2 w = *reinterpret_cast<const uint2 *>(pd + k * Rp);
          const uint4 e = *reinterpret_cast<const uint4 *>(s_O + (pp[k] - J) * 36 + 4 * mx);
          const unsigned wr[2] = {w.x, w.y};
#pragma unroll
          for (int r = 0; r < 2; r++) {
            mm[r][0] = add_min(wr[r], e.x, mm[r][0]);
            mm[r][1] = add_min(wr[r], e.y, mm[r][1]);
            mm[r][2] = add_min(wr[r], e.z, mm[r][2]);
            mm[r][3] = add_min(wr[r], e.w, mm[r][3]);
          }
        }
      }
      T = nT;
      ch = nch;
    }
    // ---- the last task of the block finishes it
    unsigned *const mb = ntask > 1 ? A.mbuf + (int64_t)__ldg(A.mslot + b) * (kRows * kRows) : nullptr;
    if (mb) {
#pragma unroll
      for (int r = 0; r < 2; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int i = 2 * my + r, a = 4 * mx + c;
          if (i < R && ((s_anc[i] >> a) & 1u) && mm[r][c] < kInf) atomicMin(mb + i * kRows + a, mm[r][c]);
        }
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        s_flag = atomicAdd(A.count + b, 1) == ntask - 1;
        __threadfence();
      }
      __syncthreads();
      if (!s_flag) continue;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(mb + (2 * my + r) * kRows + 4 * mx));
        mm[r][0] = x.x;
        mm[r][1] = x.y;
        mm[r][2] = x.z;
        mm[r][3] = x.w;
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int i = 2 * my + r;
      if (i < R) {
        int *row = A.dis + s_rowoff[i];
        const unsigned anc = s_anc[i] >> (4 * mx);
#pragma unroll
        for (int c = 0; c < 4; c++)
          if ((anc >> c) & 1u) row[s_dcol[4 * mx + c]] = (int)mm[r][c];
        if (mx < 4) {  // 0 for the node itself, INT_MAX in the row's padding
          const int own = s_dcol[i], j = own + mx;
          if (mx == 0) row[j] = 0;
          else if (j < ((own + 4) & ~3)) row[j] = INT_MAX;
        }
      }
    }
    __syncthreads();
    if (A.trace_t && tid < R) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      A.trace_t[__ldg(B.bnode + bo + tid)] = now;
    }
    if (tid == 0) {
      __threadfence();
      st_release(A.done + b, 1);
    }
  }
}

// Shortcut weights of every pos entry, read from the contraction's lists:
// entry k of v takes list index pos_src[k] of v's list, or 0 for v itself.
// One warp per vertex.
__global__ void gather_pos_weights_kernel(const int64_t *pos_hash, const int *pos_src, const int64_t *list_off,
                                          const int *list_w, int *pos_w, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; v < n;
       v += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int64_t b = pos_hash[v], e = pos_hash[v + 1], so = list_off[v];
    for (int64_t k = b + lane; k < e; k += 32) {
      const int src = pos_src[k];
      pos_w[k] = src < 0 ? 0 : list_w[so + src];
    }
  }
}

int grid_for(int64_t n, int nsm) { return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)nsm * 16, (n + 255) / 256)); }

template <typename T>
T read_one(const T *p) {
  T x{};
  GH_CUDA(cudaMemcpy(&x, p, sizeof(T), cudaMemcpyDeviceToHost));
  return x;
}

}  // namespace

// Cuts the forest into blocks and lays out their tables (weights come later,
// with enqueue).
void FillPlan::build_blocks() {
  const int grid = grid_for(N, nsm);
  Workspace ws;
  int *size = ws.get<int>(N), *weight = ws.get<int>(N), *block_top = ws.get<int>(N), *top_of = ws.get<int>(N);
  int *count = ws.get<int>(N), *blk_of_top = ws.get<int>(N);
  int *lvl = ws.get<int>(3 * (int64_t)nlev + 1);  // block tops, width, next free per level
  int *lvl_tops = lvl, *lvl_width = lvl + nlev + 1, *lvl_next = lvl_width + nlev;
  unsigned long long *lvl_work = ws.get<unsigned long long>(nlev);
  int64_t *lvl_first = ws.get<int64_t>(nlev + 1);
  GH_CUDA(cudaMemset(count, 0, sizeof(int) * N));
  GH_CUDA(cudaMemset(lvl, 0, sizeof(int) * (3 * (int64_t)nlev + 1)));
  GH_CUDA(cudaMemset(lvl_work, 0, sizeof(unsigned long long) * nlev));
  GH_CUDA(cudaMemset(block_top, 0, sizeof(int) * N));
  small_size_kernel<<<grid, 256>>>(hld, depth, size, weight, N);
  hang_weight_kernel<<<grid, 256>>>(father, htop, hpos, size, weight, N);
  cut_paths_kernel<<<grid, 256>>>(father, htop, hpos, hld, size, weight, block_top, N);
  node_block_kernel<<<grid, 256>>>(father, htop, hpos, depth, pos_hash, size, weight, block_top, top_of, count,
                                   lvl_tops, lvl_width, lvl_work, N);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(lvl_tops, lvl_first, nlev + 1, ws, 0);
  nblk = (int)read_one(lvl_first + nlev);
  GH_CHECK(nblk >= 1 && nblk <= N, H2H_ERR_STATE, "fill blocks do not cover the tree");
  blk_top = work.get<int>(nblk);
  blk_mem = work.get<int>(nblk + 1);
  blk_boff = work.get<int64_t>(nblk + 1);
  blk_moff = work.get<int64_t>(nblk + 1);
  blk_soff = work.get<int64_t>(nblk + 1);
  bnode = work.get<int>(N);
  blk_of = work.get<int>(N);
  blk_anc = work.get<unsigned>(N);
  loc_of = work.get<unsigned char>(N);
  lvl_cls = work.get<int>(nlev);
  done = work.get<int>(2 * (int64_t)nblk);  // done flags, then finished tasks per block
  unsigned long long per_node = 1ull << 18;
  if (const char *e = std::getenv("GPUH2H_HEAVY_LEVEL_WORK")) per_node = (unsigned long long)std::max(1LL, std::atoll(e));
  level_class_kernel<<<grid_for(nlev, nsm), 256>>>(lvl_width, lvl_work, nlev, nsm, per_node, lvl_cls);
  order_blocks_kernel<<<grid, 256>>>(top_of, depth, lvl_first, lvl_next, blk_top, blk_of_top, N);
  // the longest chain first where the chains set the fill's time (depth order in
  // parentheses): 11k blocks 2.13 ms (2.31), 43k 11.1 (11.4); 1k blocks the same.
  // With more, depth order keeps what it reads in L2: 154k 60.0 (58.5), 270k 121
  // (118.7).
  if (nblk >= 4096 && nblk <= 65536) {
    const int gb = grid_for(nblk, nsm);
    int *deep = ws.get<int>(nblk), *up = ws.get<int>(nblk), *up_next = ws.get<int>(nblk), *tops = ws.get<int>(nblk);
    GH_CUDA(cudaMemset(deep, 0, sizeof(int) * nblk));
    block_depth_kernel<<<grid, 256>>>(top_of, blk_of_top, depth, deep, N);
    father_block_kernel<<<gb, 256>>>(blk_top, father, top_of, blk_of_top, up, nblk);
    for (int r = 1; r <= std::min(nblk, nlev); r <<= 1) {
      deepest_round_kernel<<<gb, 256>>>(up, up_next, deep, nblk);
      std::swap(up, up_next);
    }
    GH_CUDA(cudaMemsetAsync(lvl_tops, 0, sizeof(int) * (nlev + 1)));
    GH_CUDA(cudaMemsetAsync(lvl_next, 0, sizeof(int) * nlev));
    GH_CUDA(cudaMemcpyAsync(tops, blk_top, sizeof(int) * nblk, cudaMemcpyDeviceToDevice));
    chain_count_kernel<<<gb, 256>>>(blk_top, depth, deep, lvl_tops, nlev, nblk);
    GH_CUDA(cudaGetLastError());
    exclusive_scan<int>(lvl_tops, lvl_first, nlev + 1, ws, 0);
    chain_order_kernel<<<gb, 256>>>(tops, deep, lvl_first, lvl_next, blk_top, blk_of_top, nblk);
    GH_CUDA(cudaGetLastError());
  }
  int *rows = ws.get<int>(nblk + 1), *cells = ws.get<int>(nblk + 1), *filled = ws.get<int>(nblk);
  GH_CUDA(cudaMemset(filled, 0, sizeof(int) * nblk));
  block_sizes_kernel<<<grid_for(nblk + 1, nsm), 256>>>(blk_top, count, pos_hash, rows, blk_mem, cells, nblk);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(rows, blk_boff, nblk + 1, ws, 0);
  exclusive_scan<int>(blk_mem, blk_moff, nblk + 1, ws, 0);
  exclusive_scan<int>(cells, blk_soff, nblk + 1, ws, 0);
  GH_CHECK(read_one(blk_boff + nblk) == N, H2H_ERR_STATE, "fill blocks do not cover the tree");
  const int64_t members = read_one(blk_moff + nblk);
  cell_total = read_one(blk_soff + nblk);
  bm_p = work.get<int>(members);
  bm_row = work.get<int64_t>(members);
  closed = work.get<unsigned>(cell_total);
  scatter_nodes_kernel<<<grid, 256>>>(top_of, blk_of_top, blk_boff, filled, bnode, N);
  block_nodes_kernel<<<grid_for((int64_t)nblk * 32, nsm), 256>>>(blk_top, blk_boff, blk_moff, hpos, pos_hash, pos_pos,
                                                                 pos_id, drow, bnode, blk_of, loc_of, bm_p, bm_row,
                                                                 nblk);
  GH_CUDA(cudaGetLastError());
}

namespace {

BlockArgs block_args(const FillPlan &P) {
  BlockArgs B{};
  B.blk_top = P.blk_top;
  B.boff = P.blk_boff;
  B.moff = P.blk_moff;
  B.soff = P.blk_soff;
  B.bnode = P.bnode;
  B.blk_of = P.blk_of;
  B.loc_of = P.loc_of;
  B.bm_p = P.bm_p;
  B.bm_row = P.bm_row;
  B.father = P.father;
  B.depth = P.depth;
  B.drow = P.drow;
  B.pos_hash = P.pos_hash;
  B.pos_pos = P.pos_pos;
  B.pos_id = P.pos_id;
  B.pos_w = P.pos_w;
  B.direct = P.direct;
  B.closed = P.closed;
  B.anc = P.blk_anc;
  B.nblk = P.nblk;
  B.err = P.werr;  // the fill's own word is set where it is launched
  return B;
}

}  // namespace

// Where the weights come from when the order was made on bit rows: every
// arc's cell, the tasks of the block elimination and the blocks' places in
// their parents.  The update triangles of very wide separators (a dense graph
// of many thousand vertices) can outgrow the memory; weights_fit then tells
// the caller to use the list kernels.  A plan that keeps its weights for
// rebuilds has the label rows beside them; otherwise drop_weights frees what
// only the weights need before the rows are allocated (of a 1M-vertex graph
// 0.81 GB; small tables share the plan's memory and stay).
void FillPlan::build_weights_plan(const ElimPlan &from, bool keep) {
  arcs = &from;
  Workspace ws;
  int *ntask = ws.get<int>(nblk + 1);
  int64_t *ucells = ws.get<int64_t>(nblk + 1);
  unsigned char *global = ws.get<unsigned char>(N);
  const int64_t members = read_one(blk_moff + nblk);
  // arrays of 8 MiB or more, which are allocations of their own in any arena
  auto own = [&](int64_t bytes) -> DeviceArena & { return bytes >= (int64_t(8) << 20) ? weights_mem : work; };
  direct = own(4 * cell_total).get<unsigned>(cell_total);
  wtask0 = work.get<int64_t>(nblk + 1);
  blk_up = work.get<int>(nblk);
  blk_uoff = work.get<int64_t>(nblk + 1);
  pending = work.get<int>(nblk);
  pend_init = work.get<int>(nblk);
  bm_up = own(4 * members).get<int>(members);
  arc_cell = own(8 * from.M).get<int64_t>(from.M);
  const BlockArgs B = block_args(*this);
  const int gb = grid_for(nblk + 1, nsm), gw = grid_for((int64_t)nblk * 32, nsm);
  weight_tasks_kernel<<<gb, 256>>>(blk_mem, ntask, nblk);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(ntask, wtask0, nblk + 1, ws, 0);
  wtasks = read_one(wtask0 + nblk);
  GH_CHECK(wtasks < INT32_MAX, H2H_ERR_ARG, "too many weight tasks");
  wtask_blk = own(4 * wtasks).get<int>(wtasks);
  expand_tasks_kernel<<<gw, 256>>>(wtask0, wtask_blk, nblk);
  GH_CUDA(cudaMemset(werr, 0, sizeof(int)));
  GH_CUDA(cudaMemset(pend_init, 0, sizeof(int) * nblk));
  parent_columns_kernel<<<gw, 256>>>(B, wtask0, blk_up, bm_up, pend_init);
  update_sizes_kernel<<<gb, 256>>>(blk_mem, pend_init, ucells, nblk);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int64_t>(ucells, blk_uoff, nblk + 1, ws, 0);
  upd_total = read_one(blk_uoff + nblk);
  size_t fr = 0, tot = 0;
  GH_CUDA(cudaMemGetInfo(&fr, &tot));
  const int64_t rows = keep ? dis_total + (int64_t)nblk * kRows * kRows : 0;  // label rows, in-block matrices
  weights_fit = (uint64_t)(upd_total + rows) * 4 <= fr;
  if (!weights_fit) return;
  try {
    upd = own(4 * upd_total).get<unsigned>(upd_total);
  } catch (const Error &e) {
    if (e.code != H2H_ERR_NOMEM) throw;
    weights_fit = false;
    return;
  }
  GH_CUDA(cudaMemset(global, 0, N));
  if (from.heap_total) {
    mark_kernel<<<grid_for(from.heap_total, nsm), 256>>>(from.heap_verts, from.heap_total, global);
    GH_CUDA(cudaGetLastError());
  }
  if (from.M) {
    const int ga = grid_for(from.M, nsm);
    arc_cells_kernel<<<ga, 256>>>(B, from.adj_off, from.adj_v, global, arc_cell, direct, N, from.M);
    if (from.heap_total) {  // the weights' cells are not in use yet
      first_arcs_kernel<<<ga, 256>>>(arc_cell, direct, from.M);
      drop_arcs_kernel<<<ga, 256>>>(arc_cell, direct, from.M);
    }
    GH_CUDA(cudaGetLastError());
  }
  GH_CHECK(read_one(werr) == 0, H2H_ERR_STATE, "an upper neighbour is missing from its block's separator");
}

void FillPlan::drop_weights() {
  arcs = nullptr;
  weights_mem.release();
  direct = upd = nullptr;
  blk_up = bm_up = wtask_blk = pending = pend_init = nullptr;
  blk_uoff = wtask0 = arc_cell = nullptr;
}

void FillPlan::enqueue_weights(cudaStream_t s) {
  const BlockArgs B = block_args(*this);
  const int gn = std::max(1, std::min(8192, (N + 7) / 8));  // a warp per vertex
  GH_CUDA(cudaMemsetAsync(werr, 0, sizeof(int), s));
  const int gi = (nblk + kClosureWarps - 1) / kClosureWarps;
  if (!arcs) {  // the lists carry the weights
    gather_pos_weights_kernel<<<gn, 256, 0, s>>>(pos_hash, pos_src, lists.off, lists.w, pos_w, N);
    GH_CUDA(cudaGetLastError());
    closure_kernel<<<dim3(gi, 4), 32 * kClosureWarps, 0, s>>>(B);
    inner_closure_kernel<<<gi, 32 * kClosureWarps, 0, s>>>(B);
    GH_CUDA(cudaGetLastError());
    return;
  }
  fill_inf_kernel<<<grid_for(cell_total >> 2, nsm), 256, 0, s>>>(direct, cell_total);
  fill_inf_kernel<<<grid_for(upd_total >> 2, nsm), 256, 0, s>>>(upd, upd_total);
  GH_CUDA(cudaMemcpyAsync(pending, pend_init, sizeof(int) * nblk, cudaMemcpyDeviceToDevice, s));
  GH_CUDA(cudaMemsetAsync(next, 0, sizeof(int), s));
  scatter_arcs_kernel<<<grid_for(arcs->M, nsm), 256, 0, s>>>(arc_cell, arcs->adj_w, direct, arcs->M);
  GH_CUDA(cudaGetLastError());
  WeightArgs A{};
  A.B = B;
  A.blk_up = blk_up;
  A.bm_up = bm_up;
  A.uoff = blk_uoff;
  A.upd = upd;
  A.task_blk = wtask_blk;
  A.task0 = wtask0;
  A.ntasks = (int)wtasks;
  A.pending = pending;
  A.next = next;
  A.spin_limit = spin_limit_cycles();
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  GH_CUDA(cudaStreamIsCapturing(s, &cs));
  const bool trace = std::getenv("GPUH2H_TRACE") && cs == cudaStreamCaptureStatusNone;
  if (trace) GH_CUDA(cudaStreamSynchronize(s));
  Clock clk;
  int per_sm = 0;
  GH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, weights_kernel, 128, 0));
  weights_kernel<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)nsm * std::max(1, per_sm), wtasks)), 128, 0,
                   s>>>(A);
  if (trace) {
    GH_CUDA(cudaStreamSynchronize(s));
    std::fprintf(stderr, "[gpuh2h] weights: %d blocks, %lld tiles, %.1f MB of update triangles, %.3f ms\n", nblk,
                 (long long)wtasks, upd_total * 4e-6, clk.us() / 1e3);
  }
  list_weights_kernel<<<gn, 256, 0, s>>>(B, pos_src, lists.off, lists.w, pos_w, N);
  inner_closure_kernel<<<gi, 32 * kClosureWarps, 0, s>>>(B);
  GH_CUDA(cudaGetLastError());
}

std::vector<int> FillPlan::level_classes() const {
  std::vector<int> cls(nlev);
  GH_CUDA(cudaMemcpy(cls.data(), lvl_cls, sizeof(int) * nlev, cudaMemcpyDeviceToHost));
  return cls;
}

// Tasks in block order, cut as the policy says.  The new tables are made beside
// the old ones and take their place once nothing can fail any more: without room
// the plan keeps its policy and its tasks.
void FillPlan::build_tiles(const TilePolicy &pol) {
  Workspace ws;
  int *ntask = ws.get<int>(nblk + 1), *pieces = ws.get<int>(nblk + 1), *several = ws.get<int>(nblk + 1);
  int64_t *piece0 = ws.get<int64_t>(nblk + 1), *slot0 = ws.get<int64_t>(nblk + 1);
  // the first table is made in place: there is none to keep
  const bool again = ntasks > 0;
  if (!task0) {
    int64_t *t0 = work.get<int64_t>(nblk + 1);
    tcols = work.get<int>(nblk + 1);
    mslot = work.get<int>(nblk + 1);
    task0 = t0;
  }
  int64_t *new_task0 = again ? ws.get<int64_t>(nblk + 1) : task0;
  int *new_tcols = again ? ws.get<int>(nblk + 1) : tcols;
  block_tasks_kernel<<<grid_for(nblk + 1, nsm), 256>>>(blk_top, depth, blk_mem, blk_boff, lvl_cls, pol, ntask, pieces,
                                                            new_tcols, several, nblk);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(ntask, new_task0, nblk + 1, ws, 0);
  exclusive_scan<int>(pieces, piece0, nblk + 1, ws, 0);
  exclusive_scan<int>(several, slot0, nblk + 1, ws, 0);
  const int64_t new_ntasks = read_one(new_task0 + nblk), new_mslots = read_one(slot0 + nblk),
                new_ntiles = read_one(piece0 + nblk);
  GH_CHECK(new_ntasks >= nblk && new_ntasks < INT32_MAX, H2H_ERR_ARG, "too many fill tasks");
  const int smem_dyn = enable_max_dynamic_smem(block_fill_kernel);
  const size_t new_smem = 2 * sizeof(int) * (size_t)std::max(max_segs, 1);
  GH_CHECK(new_smem <= (size_t)smem_dyn, H2H_ERR_DEVICE, "tree too large for the fill staging");
  int per_sm = 0;
  GH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, block_fill_kernel, 128, new_smem));
  // the buffers that grow: all of them before any is replaced
  struct Grown {
    void *p = nullptr;
    ~Grown() { cudaFree(p); }
  } new_mbuf, new_tasks;
  if (new_mslots > mslots_cap) new_mbuf.p = device_array<unsigned>(new_mslots * kRows * kRows);
  if (new_ntasks > tasks_cap) new_tasks.p = device_array<int>(new_ntasks);
  if (new_mbuf.p) {
    grown_bytes += (new_mslots - mslots_cap) * kRows * kRows * 4;
    mslots_cap = new_mslots;
    new_mbuf.p = std::exchange(mbuf, static_cast<unsigned *>(new_mbuf.p));
  }
  if (new_tasks.p) {
    grown_bytes += (new_ntasks - tasks_cap) * 4;
    tasks_cap = new_ntasks;
    new_tasks.p = std::exchange(tasks, static_cast<int *>(new_tasks.p));
  }
  if (again) {
    GH_CUDA(cudaMemcpyAsync(task0, new_task0, sizeof(int64_t) * (nblk + 1), cudaMemcpyDeviceToDevice));
    GH_CUDA(cudaMemcpyAsync(tcols, new_tcols, sizeof(int) * (nblk + 1), cudaMemcpyDeviceToDevice));
  }
  narrow_kernel<<<grid_for(nblk + 1, nsm), 256>>>(slot0, mslot, nblk + 1);
  expand_tasks_kernel<<<grid_for((int64_t)nblk * 32, nsm), 256>>>(task0, tasks, nblk);
  GH_CUDA(cudaGetLastError());
  policy = pol;
  ntasks = new_ntasks;
  mslots = new_mslots;
  ntiles = new_ntiles;
  smem = new_smem;
  blocks = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)nsm * std::max(1, per_sm), ntasks));
}

void FillPlan::enqueue(cudaStream_t s, cudaEvent_t *fill_ev) {
  GH_CHECK(ntasks > 0 && tasks && (mbuf || !mslots), H2H_ERR_STATE, "the fill's tasks are not laid out");
  GH_CUDA(cudaMemsetAsync(done, 0, sizeof(int) * 2 * (int64_t)nblk, s));
  GH_CUDA(cudaMemsetAsync(next, 0, sizeof(int), s));
  GH_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
  FillKernelArgs A{};
  A.B = block_args(*this);
  A.B.err = err;
  A.dis = dis;
  A.hld_row = hld_row;
  A.seg_off = seg_off;
  A.seg_top = seg_top;
  A.seg_pos = seg_pos;
  A.task_blk = tasks;
  A.task0 = task0;
  A.tcols = tcols;
  A.ntasks = (int)ntasks;
  A.done = done;
  A.count = done + nblk;
  A.next = next;
  A.mslot = mslot;
  A.mbuf = mbuf;
  A.spin_limit = spin_limit_cycles();
  A.max_segs = std::max(max_segs, 1);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  GH_CUDA(cudaStreamIsCapturing(s, &cs));
  const bool capturing = cs != cudaStreamCaptureStatusNone;
  if (std::getenv("GPUH2H_TRACE") && !capturing) {
    if (!trace_t) GH_CUDA(cudaMalloc(&trace_t, sizeof(unsigned long long) * std::max(N, 1)));
    GH_CUDA(cudaMemsetAsync(trace_t, 0, sizeof(unsigned long long) * std::max(N, 1), s));
    A.trace_t = trace_t;
  }
  // inside a capture an event record becomes a graph node only when external
  auto record = [&](cudaEvent_t e) {
    GH_CUDA(capturing ? cudaEventRecordWithFlags(e, s, cudaEventRecordExternal) : cudaEventRecord(e, s));
  };
  if (fill_ev) record(fill_ev[0]);
  if (mslots) fill_inf_kernel<<<grid_for(mslots * 256, nsm), 256, 0, s>>>(mbuf, mslots * kRows * kRows);
  block_fill_kernel<<<blocks, 128, smem, s>>>(A);
  GH_CUDA(cudaGetLastError());
  if (fill_ev) record(fill_ev[1]);
}

}  // namespace gh
