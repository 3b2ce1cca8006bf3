// labels.cu -- no-hub H2H label fill on the GPU, the work of
// makeH2HLabel_noHub_noComm_3 / makeH2HLabel_noCommunication_D_noHub_3
// (tanslate.cu:511-617, kernel_functions.cu:717-796), with the L4 block
// (kernel_functions.cu:738-743, H2HConsturction.cu:850-857) enabled.
//
// Row v holds dis[v][j] = distance from v to its ancestor at depth j+1.  For
// every u in X(v)\{v}, in descending position p (H2HConsturction.cu:840):
//   t = dis[v][p]
//   dis[v][j] = min(dis[v][j], t + dis[u][j])            j < p   (ancestors above u)
//   dis[v][j] = min(dis[v][j], t + dis[anc_j(v)][p])     p < j < d-1 (L4: below u)
//
// The L4 fill is in fill_blocks.cu; here are its plan's forest arrays and
// position lists, the exports, and two more fills:
//   * fill_level_kernel, level-synchronous, one warp per node in the
//     reference's update order: L3 rows (order-dependent) and L4 on request;
//     the node's row stays in shared memory, and its ancestors' row offsets
//     are staged from the father's, which the previous level wrote to a
//     ping-pong buffer;
//   * plain_fill_level_kernel and plain_node_fill_kernel, the reference's own
//     two GPU mappings (one thread per (v, u) pair, or one per node; a launch
//     per level), kept as measurement baselines.
//
// Rows are padded to 16-byte starts (drow[v] is a multiple of 4 ints) so the
// u-row reads are 128-bit vector loads.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <sstream>

#include "graph.h"

namespace gh {

void DeviceIndex::release_labels() {
  for (void *p : owned) cudaFree(p);
  owned.clear();
  keep.reset();
  depth = pos_pos = pos_id = dis = father = err = nullptr;
  pos_hash = drow = nullptr;
  bytes = rmq_bytes;
}

void DeviceIndex::release() {
  release_labels();
  lists = ListStore();
  x_base = pos_base = 0;
  id_base = 0;
  owned_rmq.reset();
  first = rmq_id = nullptr;
  rmq_hash = nullptr;
  bytes = rmq_bytes = 0;
}

namespace {

template <typename T>
T *dalloc(size_t n, int64_t &bytes) {
  T *p = device_array<T>((int64_t)n);
  bytes += (int64_t)(std::max<size_t>(n, 1) * sizeof(T));
  return p;
}

// An allocation the handle's DeviceIndex owns.
template <typename T>
T *dalloc_owned(size_t n, DeviceIndex &D) {
  T *p = dalloc<T>(n, D.bytes);
  D.owned.push_back(p);
  return p;
}

// Initial rows (mallocH2HLabel_noHub, H2HConsturction.cu:636-654): INT_MAX,
// shortcut weights at the positions of X(v), 0 at the own position.
__global__ void init_rows_kernel(const int64_t *drow, const int *depth, const int64_t *pos_hash, const int *pos_pos,
                                 const int *pos_w, int *dis, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; v < n;
       v += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int64_t b = drow[v];
    const int64_t e = drow[v + 1];
    for (int64_t j = b + lane; j < e; j += 32) dis[j] = INT_MAX;
    __syncwarp();
    for (int64_t t = pos_hash[v] + lane; t < pos_hash[v + 1]; t += 32) dis[b + pos_pos[t]] = pos_w[t];
  }
}

struct FillArgs {
  const int *nodes;      // tree_bfs slice of this level
  int count;             // nodes in the level
  int level;             // 0-based; depth d = level + 1
  const int *father;
  const int *lvl_idx;    // position of a node within its level
  const int64_t *drow;
  int *dis;
  const int64_t *pos_hash;
  const int *pos_id;
  const int *pos_pos;
  const int64_t *chain_prev;  // father chains: per node of level-1, (level-1) row offsets
  int64_t *chain_cur;         // chains of this level: per node, level row offsets
  int l4;
};

__global__ void fill_level_kernel(FillArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int d = A.level + 1;
  // per-warp staging: row (d ints, rounded to 4) then chain (d-1 int64)
  const int row_cap = (d + 3) & ~3;
  unsigned char *mine = smem + (size_t)wid * ((size_t)row_cap * 4 + (size_t)d * 8);
  int *row = (int *)mine;
  int64_t *anc = (int64_t *)(mine + (size_t)row_cap * 4);
  for (int w = blockIdx.x * wpb + wid; w < A.count; w += gridDim.x * wpb) {
    const int v = A.nodes[w];
    const int f = A.father[v];
    const int64_t base = A.drow[v];
    // ancestor chain: father's chain + father
    if (d >= 2) {
      const int64_t *fc = A.chain_prev + (int64_t)A.lvl_idx[f] * (d - 2);
      for (int j = lane; j < d - 2; j += 32) anc[j] = fc[j];
      if (lane == 0) anc[d - 2] = A.drow[f];
    }
    for (int j = lane; j < d; j += 32) row[j] = A.dis[base + j];
    __syncwarp();
    if (A.chain_cur) {
      int64_t *mc = A.chain_cur + (int64_t)w * (d - 1);
      for (int j = lane; j < d - 1; j += 32) mc[j] = anc[j];
    }
    const int64_t pb = A.pos_hash[v], pe = A.pos_hash[v + 1];
    for (int64_t t = pe - 2; t >= pb; t--) {      // X(v)\{v} in descending position
      const int p = A.pos_pos[t];
      const int u = A.pos_id[t];
      const int tv = row[p];
      const int *urow = A.dis + A.drow[u];
      // j < p: 128-bit loads of u's row (16-byte aligned), 4 columns per lane
      const int p4 = p >> 2;
      for (int q = lane; q < p4; q += 32) {
        int4 x = __ldg(reinterpret_cast<const int4 *>(urow) + q);
        int j = q << 2;
        row[j] = min(row[j], tv + x.x);
        row[j + 1] = min(row[j + 1], tv + x.y);
        row[j + 2] = min(row[j + 2], tv + x.z);
        row[j + 3] = min(row[j + 3], tv + x.w);
      }
      for (int j = (p4 << 2) + lane; j < p; j += 32) row[j] = min(row[j], tv + __ldg(urow + j));
      if (A.l4) {
        for (int j = p + 1 + lane; j < d - 1; j += 32) row[j] = min(row[j], tv + __ldg(A.dis + anc[j] + p));
      }
      __syncwarp();
    }
    for (int j = lane; j < d; j += 32) A.dis[base + j] = row[j];
    __syncwarp();
  }
}

// The reference's GPU label fill mapping, kept as a measurement baseline
// (makeH2HLabel_noCommunication_D_noHub_3, kernel_functions.cu:717-744, with
// the L4 block :738-743 enabled): one thread per (v, u) pair of one tree
// level; the thread min-updates the columns above u directly and walks
// father pointers for the columns below u.  Launched once per level with a
// device synchronisation in between, as the reference does.
__global__ void plain_fill_level_kernel(const int *pair_v, const int64_t *pair_k, int npairs, const int64_t *drow,
                                        const int *depth, const int *father, const int *pos_pos, const int *pos_id,
                                        const int *pos_w, int *dis) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npairs; i += gridDim.x * blockDim.x) {
    const int v = pair_v[i];
    const int64_t k = pair_k[i];
    const int p = pos_pos[k], u = pos_id[k], t = pos_w[k], d = depth[v];
    const int64_t base = drow[v], ub = drow[u];
    for (int j = 0; j < p; j++) atomicMin(dis + base + j, t + __ldcg(dis + ub + j));
    int a = father[v];
    for (int j = d - 2; j > p && a >= 0; j--) {
      atomicMin(dis + base + j, t + __ldcg(dis + drow[a] + p));
      a = father[a];
    }
  }
}

// The reference's other GPU fill mapping (parallelFine = 1:
// makeH2HLabel_noCommunication_D_noHub, kernel_functions.cu:802-837, with its
// commented L4 block enabled), kept as a measurement baseline: one thread per
// node of one tree level, walking the node's position list from the highest
// position down (its own entry, the last, excluded); each entry u at position
// p min-updates the columns below p from u's row and, for L4, the columns
// above p from the ancestors' column p along the father chain.  The thread
// owns its row: no atomics.
__global__ void plain_node_fill_kernel(const int *nodes, int cnt, const int64_t *drow, const int *depth,
                                       const int *father, const int64_t *pos_hash, const int *pos_pos,
                                       const int *pos_id, const int *pos_w, int *dis) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    const int v = nodes[i];
    const int64_t base = drow[v];
    const int d = depth[v];
    for (int64_t k = pos_hash[v + 1] - 1; k >= pos_hash[v]; k--) {
      const int u = pos_id[k];
      if (u == v) continue;
      const int p = pos_pos[k];
      const int t = dis[base + p];
      const int64_t ub = drow[u];
      for (int j = p - 1; j >= 0; j--) dis[base + j] = min(dis[base + j], t + __ldcg(dis + ub + j));
      int a = v;
      for (int j = d - 2; j > p; j--) {
        a = father[a];
        if (a < 0) break;
        dis[base + j] = min(dis[base + j], t + __ldcg(dis + drow[a] + p));
      }
    }
  }
}

__global__ void count_mismatch_kernel(const int *a, const int *b, int64_t n, unsigned long long *bad) {
  unsigned long long c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += a[i] != b[i];
  if (c) atomicAdd(bad, c);
}

// Row offset of the node at every heavy-path position (the fill reads an
// ancestor's row offset with one load instead of two dependent ones).
__global__ void hld_row_kernel(const int *hld, const int64_t *drow, int64_t *hld_row, int n) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) hld_row[k] = drow[hld[k]];
}

// Root-path segments of every node, shallowest first: walking up from v,
// each heavy path met contributes (depth of its top, index of its top in
// hld).  One thread per node; the walk crosses O(log n) light edges.
__global__ void root_path_segments_kernel(const int *father, const int *depth, const int *htop, const int *hpos,
                                          const int64_t *seg_off, int *seg_top, int *seg_pos, int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int64_t b = seg_off[v];
    int64_t k = seg_off[v + 1];
    for (int u = v; u >= 0 && k > b;) {
      const int t = htop[u];
      --k;
      seg_top[k] = depth[t];
      seg_pos[k] = hpos[t];
      u = father[t];
    }
  }
}

__global__ void max_label_kernel(const int *dis, int64_t n, int *out) {
  int m = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int x = dis[i];
    if (x != INT_MAX && x > m) m = x;
  }
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Position lists (mallocH2HLabel_noHub, H2HConsturction.cu:656-700): X(v)
// and v itself ordered by position (depth - 1 of the member).  Positions of
// one list are distinct, so an entry's slot is the number of smaller
// positions in the list.  A member that is not a proper ancestor (position >=
// d - 1) sets *err = 5.  list_w: nullptr where the weights come later.
//
// Lists that fit a warp's lanes (nine in ten of a road graph's) take a warp
// each, positions compared through shuffles; the others go to a second kernel,
// a block per list that ranks positions in a bit map of the depth (comparing
// every pair costs m * m, and the global order's lists are thousands long).  Bound: the
// loads of the members' depths; 20M entries of 1M lists take 0.5 ms (1.2 with a
// block per list and every pair compared).
struct PosArgs {
  const int64_t *list_off;
  const int *list_id, *list_w, *depth;
  const int64_t *pos_hash;
  int *pos_pos, *pos_id, *pos_w, *pos_src;
  int *large, *count;  // vertices with longer lists
  int *err;
};

__device__ __forceinline__ int member_position(const PosArgs &A, int u, int d) {
  const int key = A.depth[u] - 1;
  if (key < 0 || key >= d - 1) atomicCAS(A.err, 0, 5);
  return key;
}

__device__ __forceinline__ void put_position(const PosArgs &A, int64_t at, int key, int id, int w, int src) {
  A.pos_pos[at] = key;
  A.pos_id[at] = id;
  if (A.list_w) A.pos_w[at] = w;
  A.pos_src[at] = src;
}

__global__ void short_positions_kernel(PosArgs A, int n) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; v < n;
       v += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const int64_t b = A.list_off[v];
    const int m = (int)(A.list_off[v + 1] - b), d = A.depth[v];
    if (m > 31) {
      if (lane == 0) A.large[atomicAdd(A.count, 1)] = (int)v;
      continue;
    }
    const int id = lane < m ? A.list_id[b + lane] : (int)v;
    const int key = lane < m ? member_position(A, id, d) : d - 1;
    int r = 0;
    for (int j = 0; j <= m; j++) r += __shfl_sync(0xffffffffu, key, j) < key;
    if (lane <= m)
      put_position(A, A.pos_hash[v] + r, key, id, A.list_w && lane < m ? A.list_w[b + lane] : 0, lane < m ? lane : -1);
  }
}

__global__ void long_positions_kernel(PosArgs A, int room) {
  extern __shared__ int words[];
  __shared__ int s_total;
  const int tid = threadIdx.x, T = blockDim.x;
  for (int q = blockIdx.x; q < *A.count; q += gridDim.x) {
    const int v = A.large[q];
    const int64_t b = A.list_off[v], pb = A.pos_hash[v];
    const int m = (int)(A.list_off[v + 1] - b), d = A.depth[v];
    const int W = (d + 31) >> 5;
    if (2 * W <= room) {  // a bit per position, then the bits before each word
      unsigned *bits = reinterpret_cast<unsigned *>(words);
      int *before = words + W;
      for (int w = tid; w < W; w += T) bits[w] = 0;
      __syncthreads();
      for (int i = tid; i <= m; i += T) {
        const int key = i < m ? member_position(A, A.list_id[b + i], d) : d - 1;
        if (key >= 0 && key < d) atomicOr(bits + (key >> 5), 1u << (key & 31));
      }
      __syncthreads();
      if (tid < 32) {
        int run = 0;
        for (int w0 = 0; w0 < W; w0 += 32) {
          const int c = w0 + tid < W ? __popc(bits[w0 + tid]) : 0;
          int incl = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += y;
          }
          if (w0 + tid < W) before[w0 + tid] = run + incl - c;
          run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (tid == 0) s_total = run;
      }
      __syncthreads();
      for (int i = tid; i <= m; i += T) {
        const int id = i < m ? A.list_id[b + i] : v, key = A.depth[id] - 1;
        if (s_total != m + 1 || key < 0 || key >= d) {  // a position out of range, or twice
          atomicCAS(A.err, 0, 5);
          continue;
        }
        put_position(A, pb + before[key >> 5] + __popc(bits[key >> 5] & ((1u << (key & 31)) - 1u)), key, id,
                     A.list_w && i < m ? A.list_w[b + i] : 0, i < m ? i : -1);
      }
    } else {  // deep for its length: the number of smaller positions in the list
      for (int i = tid; i <= m; i += T) words[i] = i < m ? member_position(A, A.list_id[b + i], d) : d - 1;
      __syncthreads();
      for (int i = tid; i <= m; i += T) {
        const int key = words[i];
        int r = 0;
        for (int j = 0; j <= m; j++) r += words[j] < key;
        put_position(A, pb + r, key, i < m ? A.list_id[b + i] : v, A.list_w && i < m ? A.list_w[b + i] : 0,
                     i < m ? i : -1);
      }
    }
    __syncthreads();
  }
}

}  // namespace

// A narrow level's blocks are the chain the fill waits for and are cut finely;
// elsewhere a task's own start (tables, members, ancestors) costs as much as two
// or three steps, so small separators keep whole rows, but wide ones, whose
// tasks of 512 columns ran for 200 us each on the critical path, are cut too.
// Columns by separator up to 16 / 64 / 256 / more, 264k, 1M and 6.26M vertices: 4096 /
// 4096 / 512 / 128 2.56, 12.2 and 118.8 ms; 4096 / 512 / 128 / 64 2.25, 11.4,
// 120.3; 4096 / 768 / 192 / 128 2.27, 11.3, 118.3; 1024 / 512 / 128 / 64 2.36, 12.0.
TilePolicy::TilePolicy() {
  static const int cb[kWidth][kSep] = {{64, 64, 64, 64}, {4096, 768, 192, 128}, {4096, 768, 192, 128}};
  for (int w = 0; w < kWidth; w++)
    for (int b = 0; b < kSep; b++) {
      small_work[w][b] = 1024;
      col_block[w][b] = cb[w][b];
      sep_chunk[w][b] = 32;
    }
}

std::string TilePolicy::str() const {
  std::ostringstream o;
  for (int w = 0; w < kWidth; w++)
    for (int b = 0; b < kSep; b++)
      o << (w || b ? " " : "") << small_work[w][b] << "/" << col_block[w][b] << "/" << sep_chunk[w][b];
  return o.str();
}

bool TilePolicy::parse(const std::string &text) {
  TilePolicy t;
  std::istringstream in(text);
  for (int w = 0; w < kWidth; w++)
    for (int b = 0; b < kSep; b++) {
      long long sw, cb, sc;
      char s1, s2;
      if (!(in >> sw >> s1 >> cb >> s2 >> sc) || s1 != '/' || s2 != '/') return false;
      if (sw < 0 || sw > (1LL << 30) || cb < 1 || cb > 4096 || sc < 1 || sc > 1024) return false;
      t.small_work[w][b] = (int)sw;
      t.col_block[w][b] = (int)cb;
      t.sep_chunk[w][b] = (int)sc;
    }
  std::string rest;
  if (in >> rest) return false;
  *this = t;
  return true;
}

FillPlan::FillPlan(const std::vector<Graph *> &graphs, const ListStore &lst, const ElimPlan *from, bool keep)
    : gs(graphs), lists(lst) {
  const bool trace = std::getenv("GPUH2H_TRACE") != nullptr;
  Clock tclk;
  auto mark = [&](const char *what) {
    if (!trace) return;
    cudaDeviceSynchronize();
    std::fprintf(stderr, "[gpuh2h] fill plan: %s %.3f ms\n", what, tclk.us() / 1e3);
    tclk.reset();
  };
  GH_CHECK(!gs.empty(), H2H_ERR_ARG, "no graph to label");
  const std::shared_ptr<TreeStore> tree = gs[0]->tree;
  GH_CHECK(tree && tree->gs == gs && tree->layout, H2H_ERR_STATE, "tree not built");
  vbase = tree->vbase;
  vbase.pop_back();
  N = tree->n;
  pos_total = tree->pos_total;
  dis_total = tree->dis_total;
  max_segs = std::max(max_segs, tree->max_segs);
  nlev = tree->height;
  layout = tree->layout;
  int dev = 0;
  GH_CUDA(cudaGetDevice(&dev));
  GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  storage = std::make_shared<LabelStore>();
  storage->tree = tree;
  drow = tree->drow;
  pos_hash = tree->pos_hash;
  father = tree->father;
  depth = tree->depth;
  hld = tree->hld;
  htop = tree->htop;
  hpos = tree->hpos;
  seg_off = tree->seg_off;
  const int64_t seg_total = tree->seg_total;
  const int max_m = tree->max_list;
  pos_pos = storage->mem.get<int>(pos_total);
  pos_id = storage->mem.get<int>(pos_total);
  try {
    pos_w = work.get<int>(pos_total);
    pos_src = work.get<int>(pos_total);
    seg_top = work.get<int>(std::max<int64_t>(seg_total, 1));
    seg_pos = work.get<int>(std::max<int64_t>(seg_total, 1));
    next = work.get<int>(1);
    err = work.get<int>(2);
    werr = err + 1;
    GH_CUDA(cudaMemset(err, 0, 2 * sizeof(int)));
    hld_row = work.get<int64_t>(N);
    hld_row_kernel<<<std::max(1, std::min(8192, (N + 255) / 256)), 256>>>(hld, drow, hld_row, N);
    GH_CUDA(cudaGetLastError());
    mark("allocations");
    {
      const int room = std::max(max_m + 1, 1024);  // ints of staging: a list, or the bits of 16,384 positions
      const size_t ksmem = (size_t)room * sizeof(int);
      const int kdyn = enable_max_dynamic_smem(long_positions_kernel);
      GH_CHECK(ksmem <= (size_t)kdyn, H2H_ERR_DEVICE, "separator too large for the position-list staging");
      DeviceArena ws;
      PosArgs A{lists.off, lists.id, from && from->bits ? nullptr : lists.w, depth, pos_hash, pos_pos, pos_id, pos_w,
                pos_src, ws.get<int>(N), ws.get<int>(1), err};
      GH_CUDA(cudaMemset(A.count, 0, sizeof(int)));
      short_positions_kernel<<<std::max(1, std::min(nsm * 8, (N + 7) / 8)), 256>>>(A, N);
      if (max_m > 31) long_positions_kernel<<<std::max(1, std::min(N, nsm * 16)), 128, ksmem>>>(A, room);
      GH_CUDA(cudaGetLastError());
      int e = 0;
      GH_CUDA(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
      GH_CHECK(e == 0, H2H_ERR_STATE, "an upper neighbour is not an ancestor in the tree");
    }
    mark("position lists");
    root_path_segments_kernel<<<std::max(1, std::min(8192, (N + 255) / 256)), 256>>>(father, depth, htop, hpos,
                                                                                     seg_off, seg_top, seg_pos, N);
    GH_CUDA(cudaGetLastError());
    mark("root-path segments");
    build_blocks();
    mark("blocks");
    if (from && from->bits) {
      build_weights_plan(*from, keep);
      mark("weights plan");
    }
  } catch (...) {
    release_work();
    throw;
  }
}

FillPlan::~FillPlan() { release_work(); }

void FillPlan::prepare(const TilePolicy &pol) {
  if (!dis) dis = storage->mem.get<int>(dis_total);  // a second attempt has them already
  build_tiles(pol);
}

void FillPlan::release_work() {
  work.release();
  weights_mem.release();
  layout.reset();
  for (void *p : {(void *)tasks, (void *)mbuf, (void *)trace_t}) cudaFree(p);
  grown_bytes = tasks_cap = mslots_cap = ntasks = mslots = 0;
  trace_t = nullptr;
  pos_w = pos_src = hld = htop = hpos = seg_top = seg_pos = done = next = err = werr = tasks = nullptr;
  blk_top = blk_mem = bnode = blk_of = lvl_cls = bm_p = tcols = nullptr;
  hld_row = seg_off = blk_boff = blk_moff = blk_soff = bm_row = task0 = nullptr;
  loc_of = nullptr;
  direct = closed = blk_anc = upd = mbuf = nullptr;
  mslot = nullptr;
  blk_up = bm_up = wtask_blk = pending = pend_init = nullptr;
  blk_uoff = wtask0 = arc_cell = nullptr;
}

// With GPUH2H_TRACE: where the last fill's time went, from the nodes'
// publish times -- per forest level the time from the previous level's last
// publish to its own (levels overlap; the spans add up to the fill), summed per tile class, and the ten longest levels.
void FillPlan::trace_report() {
  if (!trace_t) return;
  GH_CUDA(cudaDeviceSynchronize());
  std::vector<unsigned long long> t(N);
  std::vector<int> dep(N);
  GH_CUDA(cudaMemcpy(t.data(), trace_t, sizeof(unsigned long long) * N, cudaMemcpyDeviceToHost));
  GH_CUDA(cudaMemcpy(dep.data(), depth, sizeof(int) * N, cudaMemcpyDeviceToHost));
  const std::vector<int> cls = level_classes();
  const int nlev = (int)cls.size();
  std::vector<unsigned long long> last(nlev, 0);
  std::vector<int64_t> width(nlev, 0);
  unsigned long long t0 = ~0ull;
  for (int v = 0; v < N; v++) {
    const int l = dep[v] - 1;
    if (l < 0 || l >= nlev || t[v] == 0) continue;
    last[l] = std::max(last[l], t[v]);
    width[l]++;
    t0 = std::min(t0, t[v]);
  }
  if (t0 == ~0ull) return;
  double by_cls[3] = {0, 0, 0};
  std::vector<std::pair<double, int>> spans;
  unsigned long long prev = t0;
  for (int l = 0; l < nlev; l++) {
    if (!last[l]) continue;
    const double us = last[l] > prev ? (last[l] - prev) / 1e3 : 0.0;
    by_cls[cls[l]] += us;
    spans.push_back({us, l});
    prev = std::max(prev, last[l]);
  }
  std::fprintf(stderr, "[gpuh2h] fill trace: first to last publish %.3f ms; narrow levels %.3f, wide %.3f, heavy %.3f ms\n",
               (prev - t0) / 1e6, by_cls[0] / 1e3, by_cls[1] / 1e3, by_cls[2] / 1e3);
  std::sort(spans.rbegin(), spans.rend());
  for (size_t k = 0; k < spans.size() && k < 10; k++)
    std::fprintf(stderr, "[gpuh2h] fill trace: level %d (class %d, %lld nodes): %.1f us\n", spans[k].second,
                 cls[spans[k].second], (long long)width[spans[k].second], spans[k].first);
}

void FillPlan::check_error() {
  GH_CUDA(cudaDeviceSynchronize());
  int e[2] = {0, 0};  // err, werr
  GH_CUDA(cudaMemcpy(e, err, sizeof(e), cudaMemcpyDeviceToHost));
  GH_CHECK(e[1] == 0, H2H_ERR_DEVICE, "block weights: a dependency wait ran out (error code " + std::to_string(e[1]) + ")");
  GH_CHECK(e[0] == 0, H2H_ERR_DEVICE, "label fill: a dependency wait ran out (error code " + std::to_string(e[0]) + ")");
}

void FillPlan::attach(bool first) {
  for (size_t i = 0; i < gs.size(); i++) {
    Graph &g = *gs[i];
    DeviceIndex &D = g.dev;
    const int vb = vbase[i];
    if (first) {
      D.release_labels();
      D.n = g.n;
      D.keep = storage;
      D.depth = depth + vb;
      D.father = father + vb;
      D.drow = drow + vb;
      D.pos_hash = pos_hash + vb;
      D.pos_pos = pos_pos;
      D.pos_id = pos_id;
      D.dis = dis;
      D.pos = g.pos_n;
      D.pos_base = D.x_base + vb;
      D.dis_padded = g.row1 - g.row0;
      D.err = dalloc_owned<int>(1, D);
      D.bytes += (int64_t)(g.n + 1) * 16 + (int64_t)g.n * 8 + D.pos * 8 + D.dis_padded * 4;
    }
    g.max_label = -1;  // the largest label is computed when it is first asked for (label_max)
  }
  if (first) storage->tree->layout.reset();  // the plan's own reference is the last
}

// The largest finite label of g's rows, computed on first request (a pass
// over the labels, about 20 ms for the 6.26M-vertex graph's 115 GB) and
// kept; a rebuild resets it.
int64_t label_max(const Graph &gc) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  Graph &g = const_cast<Graph &>(gc);
  if (g.max_label >= 0 || !g.dev.dis || !g.dev.err) return std::max<int64_t>(g.max_label, 0);
  const int64_t r0 = g.row0, r1 = g.row1;
  int dev = 0, nsm = 1;
  GH_CUDA(cudaGetDevice(&dev));
  GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  GH_CUDA(cudaMemset(g.dev.err, 0, sizeof(int)));
  max_label_kernel<<<std::max(1, std::min<int>(nsm * 4, (int)((r1 - r0 + 255) / 256))), 256>>>(
      g.dev.dis + r0, r1 - r0, g.dev.err);
  GH_CUDA(cudaGetLastError());
  int mx = 0;
  GH_CUDA(cudaMemcpy(&mx, g.dev.err, sizeof(int), cudaMemcpyDeviceToHost));
  GH_CUDA(cudaMemset(g.dev.err, 0, sizeof(int)));
  g.max_label = mx;
  return mx;
}

// Autotuner of the forest fill's tile shapes.  Coordinate descent over the
// (level width x separator size) buckets that hold nodes: for each bucket in
// turn, first the one-task threshold, then the columns of a task, each
// candidate timed as a whole fill (best of two runs) with the
// other buckets held; a candidate replaces the incumbent only when it is 2%
// faster.  Any policy gives the same labels: only the schedule changes.
std::string tile_policy_tune(FillPlan &plan, cudaStream_t s, int rounds) {
  bool used[TilePolicy::kWidth][TilePolicy::kSep] = {};
  {
    const std::vector<int> lcls = plan.level_classes();
    for (const Graph *g : plan.gs) {
      host_tree(*g);
      for (int l = 0; l + 1 < (int)g->tree_hash.size(); l++)
        for (int q = g->tree_hash[l]; q < g->tree_hash[l + 1]; q++) {
          const int v = g->tree_bfs[q];
          used[lcls[l]][TilePolicy::sep_bucket((int)(g->pos_hash[v + 1] - g->pos_hash[v]) - 1)] = true;
        }
    }
  }
  cudaEvent_t ev[2];
  GH_CUDA(cudaEventCreate(&ev[0]));
  GH_CUDA(cudaEventCreate(&ev[1]));
  auto time_fill = [&]() -> float {
    float best = 1e30f;
    for (int rep = 0; rep < 2; rep++) {
      plan.enqueue(s, ev);
      plan.check_error();
      float ms = 0;
      GH_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      best = std::min(best, ms);
    }
    return best;
  };
  auto time_policy = [&](const TilePolicy &p) -> float {
    try {
      plan.build_tiles(p);
    } catch (const Error &) {
      return 1e30f;  // no room for its tasks: not a candidate
    }
    return time_fill();
  };
  static const int kSmall[] = {0, 1 << 10, 1 << 12, 1 << 14, 1 << 16, 1 << 20};
  static const int kCols[] = {64, 128, 256, 512, 1024, 4096};
  TilePolicy best = plan.policy;
  float best_ms = 0;
  try {
    plan.build_tiles(best);
    best_ms = time_fill();
    for (int r = 0; r < rounds; r++)
      for (int wb = 0; wb < TilePolicy::kWidth; wb++)
        for (int sb = 0; sb < TilePolicy::kSep; sb++) {
          if (!used[wb][sb]) continue;
          for (int sw : kSmall) {
            if (sw == best.small_work[wb][sb]) continue;
            TilePolicy p = best;
            p.small_work[wb][sb] = sw;
            const float t = time_policy(p);
            if (t < best_ms * 0.98f) { best = p; best_ms = t; }
          }
          for (int cols : kCols) {
            if (cols == best.col_block[wb][sb]) continue;
            TilePolicy p = best;
            p.col_block[wb][sb] = cols;
            const float t = time_policy(p);
            if (t < best_ms * 0.98f) { best = p; best_ms = t; }
          }
        }
    plan.build_tiles(best);  // leaves the tasks and the labels of the chosen policy
    time_fill();
  } catch (...) {
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    throw;
  }
  cudaEventDestroy(ev[0]);
  cudaEventDestroy(ev[1]);
  return best.str();
}

void fill_labels_gpu(Graph &g) {
  Clock clk;
  const int n = g.n;
  DeviceIndex &D = g.dev;
  // L4 runs over blocks of the tree; L3 (order-dependent, as shipped)
  // keeps the level-synchronous kernel that applies the reference's order.
  const bool flow = !uses_level_fill(g);
  if (flow) {
    TilePolicy pol = TilePolicy();
    if (const char *e = std::getenv("GPUH2H_TILE_POLICY"))
      GH_CHECK(pol.parse(e), H2H_ERR_ARG, "GPUH2H_TILE_POLICY: expected 12 entries small_work/col_block/sep_chunk");
    if (!g.plan) {  // contracted by the list kernels
      g.plan = std::make_shared<FillPlan>(std::vector<Graph *>{&g}, D.lists, nullptr, false);
      g.plan->enqueue_weights(0);
    }
    FillPlan &plan = *g.plan;
    plan.prepare(pol);
    GH_CUDA(cudaDeviceSynchronize());
    g.t.translate_labels = clk.us();
    clk.reset();
    cudaEvent_t ev[2];
    GH_CUDA(cudaEventCreate(&ev[0]));
    GH_CUDA(cudaEventCreate(&ev[1]));
    float ms = 0;
    try {
      plan.enqueue(0, ev);
      plan.check_error();
      plan.trace_report();
      GH_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
    } catch (...) {
      cudaEventDestroy(ev[0]);
      cudaEventDestroy(ev[1]);
      throw;
    }
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    g.t.fill_gpu = (long long)(ms * 1000.0f);
    Clock tail;  // the per-graph view and the plan's work buffers count with the plan's host time
    plan.attach(true);
    g.plan.reset();
    g.t.translate_labels += tail.us();
    return;
  }
  g.plan.reset();
  D.release_labels();
  struct Undo {  // what a fill that fails had allocated; the tree stays for another
    DeviceIndex *d;
    ~Undo() {
      if (d) d->release_labels();
    }
  } undo{&D};
  D.n = n;
  D.pos_base = 0;
  // padded row offsets
  std::vector<int64_t> drow(n + 1, 0);
  for (int v = 0; v < n; v++) drow[v + 1] = drow[v] + ((g.depth[v] + 3) & ~3);
  D.dis_padded = drow[n];
  D.pos = g.pos_hash[n];
  const int nlev = (int)g.tree_hash.size() - 1;
  int64_t tmp_bytes = 0;
  D.drow = dalloc_owned<int64_t>(n + 1, D);
  D.dis = dalloc_owned<int>(D.dis_padded, D);
  D.pos_hash = dalloc_owned<int64_t>(n + 1, D);
  D.pos_pos = dalloc_owned<int>(D.pos, D);
  D.pos_id = dalloc_owned<int>(D.pos, D);
  D.father = dalloc_owned<int>(n, D);
  D.depth = dalloc_owned<int>(n, D);
  D.err = dalloc_owned<int>(1, D);
  int *d_pos_w = nullptr, *d_nodes = nullptr, *d_aux = nullptr;
  int64_t *d_chain[2] = {nullptr, nullptr};
  auto cleanup = [&]() {
    cudaFree(d_pos_w); cudaFree(d_nodes); cudaFree(d_aux); cudaFree(d_chain[0]); cudaFree(d_chain[1]);
  };
  try {
    d_pos_w = dalloc<int>(D.pos, tmp_bytes);
    d_nodes = dalloc<int>(n, tmp_bytes);
    d_aux = dalloc<int>(n, tmp_bytes);  // index of the node within its level
    std::vector<int> aux(n, 0);
    int64_t chain_max = 1;
    for (int l = 0; l < nlev; l++)
      for (int i = g.tree_hash[l]; i < g.tree_hash[l + 1]; i++) aux[g.tree_bfs[i]] = i - g.tree_hash[l];
    for (int l = 0; l < nlev; l++)
      chain_max = std::max<int64_t>(chain_max, (int64_t)(g.tree_hash[l + 1] - g.tree_hash[l]) * l);
    d_chain[0] = dalloc<int64_t>(chain_max, tmp_bytes);
    d_chain[1] = dalloc<int64_t>(chain_max, tmp_bytes);
    GH_CUDA(cudaMemcpy(D.drow, drow.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.pos_hash, g.pos_hash.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.pos_pos, g.pos_pos.data(), sizeof(int) * D.pos, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.pos_id, g.pos_id.data(), sizeof(int) * D.pos, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_pos_w, g.pos_w.data(), sizeof(int) * D.pos, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.father, g.father.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.depth, g.depth.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_nodes, g.tree_bfs.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_aux, aux.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemset(D.err, 0, sizeof(int)));
    init_rows_kernel<<<std::max(1, std::min(65535, (n * 32 + 255) / 256)), 256>>>(D.drow, D.depth, D.pos_hash,
                                                                                  D.pos_pos, d_pos_w, D.dis, n);
    GH_CUDA(cudaGetLastError());
    GH_CUDA(cudaDeviceSynchronize());
    g.t.translate_labels = clk.us();
    clk.reset();
    int dev = 0, nsm = 0;
    GH_CUDA(cudaGetDevice(&dev));
    GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    cudaEvent_t e0, e1;
    GH_CUDA(cudaEventCreate(&e0));
    GH_CUDA(cudaEventCreate(&e1));
    GH_CUDA(cudaEventRecord(e0));
    const int smem_dyn = enable_max_dynamic_smem(fill_level_kernel);
    for (int l = 1; l < nlev; l++) {
      const int d = l + 1;
      const size_t per_warp = (size_t)((d + 3) & ~3) * 4 + (size_t)d * 8;
      int wpb = (int)std::min<size_t>(8, (size_t)smem_dyn / per_warp);
      GH_CHECK(wpb >= 1, H2H_ERR_DEVICE, "tree too deep for the shared-memory row staging");
      const int count = g.tree_hash[l + 1] - g.tree_hash[l];
      FillArgs A;
      A.nodes = d_nodes + g.tree_hash[l];
      A.count = count;
      A.level = l;
      A.father = D.father;
      A.lvl_idx = d_aux;
      A.drow = D.drow;
      A.dis = D.dis;
      A.pos_hash = D.pos_hash;
      A.pos_id = D.pos_id;
      A.pos_pos = D.pos_pos;
      A.chain_prev = d_chain[(l + 1) & 1];
      A.chain_cur = (l + 1 < nlev) ? d_chain[l & 1] : nullptr;
      A.l4 = g.label_mode == H2H_LABEL_L4;
      int blocks = (int)std::min<int64_t>((count + wpb - 1) / wpb, (int64_t)nsm * 16);
      fill_level_kernel<<<std::max(1, blocks), wpb * 32, per_warp * wpb>>>(A);
      GH_CUDA(cudaGetLastError());
    }
    GH_CUDA(cudaEventRecord(e1));
    GH_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    GH_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    g.t.fill_gpu = (long long)(ms * 1000.0f);
    g.max_label = -1;  // computed on first request (label_max)
  } catch (...) {
    cleanup();
    throw;
  }
  cleanup();
  undo.d = nullptr;
  g.tree.reset();  // its host copies are made (allocate_labels_and_bfs)
  g.drow_host.swap(drow);
  g.row0 = 0;
  g.row1 = D.dis_padded;
}

// Copies the filled labels back into the reference's unpadded layout.
void upload_labels(Graph &g, const std::vector<int> &dis, const std::vector<int> &pos_id,
                   const std::vector<int> &pos_pos) {
  const int n = g.n;
  DeviceIndex &D = g.dev;
  D.release_labels();
  D.n = n;
  D.pos_base = 0;
  std::vector<int64_t> drow(n + 1, 0);
  for (int v = 0; v < n; v++) drow[v + 1] = drow[v] + ((g.depth[v] + 3) & ~3);
  D.dis_padded = drow[n];
  D.pos = g.pos_hash[n];
  D.drow = dalloc_owned<int64_t>(n + 1, D);
  D.dis = dalloc_owned<int>(D.dis_padded, D);
  D.pos_hash = dalloc_owned<int64_t>(n + 1, D);
  D.pos_pos = dalloc_owned<int>(D.pos, D);
  D.pos_id = dalloc_owned<int>(D.pos, D);
  D.father = dalloc_owned<int>(n, D);
  D.depth = dalloc_owned<int>(n, D);
  D.err = dalloc_owned<int>(1, D);
  GH_CUDA(cudaMemcpy(D.drow, drow.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
  GH_CUDA(cudaMemcpy(D.pos_hash, g.pos_hash.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
  if (D.pos) {
    GH_CUDA(cudaMemcpy(D.pos_pos, pos_pos.data(), sizeof(int) * D.pos, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(D.pos_id, pos_id.data(), sizeof(int) * D.pos, cudaMemcpyHostToDevice));
  }
  GH_CUDA(cudaMemcpy(D.father, g.father.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  GH_CUDA(cudaMemcpy(D.depth, g.depth.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  GH_CUDA(cudaMemset(D.err, 0, sizeof(int)));
  // rows into the padded layout through a page-locked staging buffer of at
  // most 64 Mi entries (padding entries are INT_MAX, as the fill leaves them)
  const int64_t kStage = int64_t(1) << 26;
  int *stage = nullptr;
  GH_CUDA(cudaMallocHost(&stage, sizeof(int) * std::min<int64_t>(std::max<int64_t>(D.dis_padded, 1), kStage)));
  try {
    int v = 0;
    while (v < n) {
      const int64_t p0 = drow[v];
      int w = v;
      while (w < n && drow[w + 1] - p0 <= kStage) w++;
      GH_CHECK(w > v, H2H_ERR_ARG, "a label row longer than the upload staging");
      for (int u = v; u < w; u++) {
        int *row = stage + (drow[u] - p0);
        std::copy(dis.begin() + g.dis_hash[u], dis.begin() + g.dis_hash[u] + g.depth[u], row);
        for (int64_t j = g.depth[u]; j < drow[u + 1] - drow[u]; j++) row[j] = INT_MAX;
      }
      GH_CUDA(cudaMemcpy(D.dis + p0, stage, sizeof(int) * (drow[w] - p0), cudaMemcpyHostToDevice));
      v = w;
    }
  } catch (...) {
    cudaFreeHost(stage);
    throw;
  }
  cudaFreeHost(stage);
  g.drow_host.swap(drow);
  g.row0 = 0;
  g.row1 = D.dis_padded;
}

// Runs one of the reference's GPU fill mappings (mapping 0: a thread per
// (v, u) pair, plain_fill_level_kernel; 1: a thread per node,
// plain_node_fill_kernel) on the built graph into a scratch copy of the rows
// and compares it with the built labels.  The device time of the per-level
// launches and synchronisations goes to *ms; *mismatches receives the number
// of differing entries.
void fill_labels_plain(const Graph &g, int mapping, double *ms, int64_t *mismatches) {
  GH_CHECK(mapping == 0 || mapping == 1, H2H_ERR_ARG, "mapping must be 0 (pair per thread) or 1 (node per thread)");
  GH_CHECK(g.labelled && g.label_mode == H2H_LABEL_L4, H2H_ERR_STATE, "needs built L4 labels");
  const DeviceIndex &D = g.dev;
  const int n = g.n;
  host_tree(g);
  const int64_t np = g.pos_n;
  std::vector<int> pid(np), ppos(np);
  download_positions(g, pid.data(), ppos.data());
  // (v, k) pairs per tree level, k over v's entries other than v itself
  std::vector<int> pv;
  std::vector<int64_t> pk;
  std::vector<int64_t> lvl_off{0};
  const int nlev = (int)g.tree_hash.size() - 1;
  for (int l = 0; l < nlev; l++) {
    for (int q = g.tree_hash[l]; q < g.tree_hash[l + 1]; q++) {
      const int v = g.tree_bfs[q];
      for (int64_t k = g.pos_hash[v]; k < g.pos_hash[v + 1]; k++)
        if (pid[k] != v) { pv.push_back(v); pk.push_back(k); }
    }
    lvl_off.push_back((int64_t)pv.size());
  }
  int64_t tmp = 0;
  int *d_dis = nullptr, *d_pv = nullptr, *d_w = nullptr;
  int64_t *d_pk = nullptr, *d_drow = nullptr;
  int *d_depth = nullptr, *d_father = nullptr, *d_pos_pos = nullptr, *d_pos_id = nullptr, *d_bfs = nullptr;
  int64_t *d_pos_hash = nullptr;
  unsigned long long *d_bad = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto cleanup = [&]() {
    cudaFree(d_dis); cudaFree(d_pv); cudaFree(d_w); cudaFree(d_pk); cudaFree(d_drow); cudaFree(d_depth);
    cudaFree(d_father); cudaFree(d_pos_pos); cudaFree(d_pos_id); cudaFree(d_pos_hash); cudaFree(d_bad);
    cudaFree(d_bfs);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  };
  try {
    const int64_t rows = g.drow_host[n] - g.drow_host[0];
    std::vector<int64_t> drow(n + 1);
    for (int v = 0; v <= n; v++) drow[v] = g.drow_host[v] - g.drow_host[0];
    std::vector<int> pw(np);
    {
      // shortcut weights per position entry from the device lists
      std::vector<int> xid(g.x_off[n]), xw(g.x_off[n]);
      if (g.x_off[n]) {
        GH_CUDA(cudaMemcpy(xid.data(), D.lists.id + D.x_base, sizeof(int) * g.x_off[n], cudaMemcpyDeviceToHost));
        GH_CUDA(cudaMemcpy(xw.data(), D.lists.w + D.x_base, sizeof(int) * g.x_off[n], cudaMemcpyDeviceToHost));
      }
      for (int v = 0; v < n; v++)  // lists are sorted by id: binary search
        for (int64_t k = g.pos_hash[v]; k < g.pos_hash[v + 1]; k++) {
          pw[k] = 0;
          if (pid[k] == v) continue;
          const auto b = xid.begin() + g.x_off[v], e = xid.begin() + g.x_off[v + 1];
          const auto it = std::lower_bound(b, e, pid[k] + D.id_base);
          if (it != e && *it == pid[k] + D.id_base) pw[k] = xw[it - xid.begin()];
        }
    }
    d_dis = dalloc<int>(rows, tmp);
    d_pv = dalloc<int>(std::max<size_t>(pv.size(), 1), tmp);
    d_pk = dalloc<int64_t>(std::max<size_t>(pk.size(), 1), tmp);
    d_drow = dalloc<int64_t>(n + 1, tmp);
    d_depth = dalloc<int>(n, tmp);
    d_father = dalloc<int>(n, tmp);
    d_pos_pos = dalloc<int>(std::max<int64_t>(np, 1), tmp);
    d_pos_id = dalloc<int>(std::max<int64_t>(np, 1), tmp);
    d_w = dalloc<int>(std::max<int64_t>(np, 1), tmp);
    d_pos_hash = dalloc<int64_t>(n + 1, tmp);
    d_bad = dalloc<unsigned long long>(1, tmp);
    d_bfs = dalloc<int>(std::max<size_t>(g.tree_bfs.size(), 1), tmp);
    if (!g.tree_bfs.empty())
      GH_CUDA(cudaMemcpy(d_bfs, g.tree_bfs.data(), sizeof(int) * g.tree_bfs.size(), cudaMemcpyHostToDevice));
    if (!pv.empty()) {
      GH_CUDA(cudaMemcpy(d_pv, pv.data(), sizeof(int) * pv.size(), cudaMemcpyHostToDevice));
      GH_CUDA(cudaMemcpy(d_pk, pk.data(), sizeof(int64_t) * pk.size(), cudaMemcpyHostToDevice));
    }
    GH_CUDA(cudaMemcpy(d_drow, drow.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_depth, g.depth.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_father, g.father.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_pos_pos, ppos.data(), sizeof(int) * np, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_pos_id, pid.data(), sizeof(int) * np, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_w, pw.data(), sizeof(int) * np, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_pos_hash, g.pos_hash.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemset(d_bad, 0, sizeof(unsigned long long)));
    GH_CUDA(cudaEventCreate(&e0));
    GH_CUDA(cudaEventCreate(&e1));
    GH_CUDA(cudaEventRecord(e0));
    // mallocH2HLabel_noHub's initial rows, then the levels in order
    init_rows_kernel<<<std::max(1, std::min(65535, (n * 32 + 255) / 256)), 256>>>(d_drow, d_depth, d_pos_hash,
                                                                                  d_pos_pos, d_w, d_dis, n);
    GH_CUDA(cudaGetLastError());
    GH_CUDA(cudaDeviceSynchronize());
    for (int l = 1; l < nlev; l++) {
      if (mapping == 1) {
        const int cnt = g.tree_hash[l + 1] - g.tree_hash[l];
        if (cnt == 0) continue;
        plain_node_fill_kernel<<<(cnt + 255) / 256, 256>>>(d_bfs + g.tree_hash[l], cnt, d_drow, d_depth, d_father,
                                                            d_pos_hash, d_pos_pos, d_pos_id, d_w, d_dis);
      } else {
        const int64_t a = lvl_off[l], b = lvl_off[l + 1];
        if (b == a) continue;
        const int cnt = (int)(b - a);
        plain_fill_level_kernel<<<(cnt + 255) / 256, 256>>>(d_pv + a, d_pk + a, cnt, d_drow, d_depth, d_father,
                                                             d_pos_pos, d_pos_id, d_w, d_dis);
      }
      GH_CUDA(cudaGetLastError());
      GH_CUDA(cudaDeviceSynchronize());
    }
    GH_CUDA(cudaEventRecord(e1));
    GH_CUDA(cudaEventSynchronize(e1));
    float t = 0;
    GH_CUDA(cudaEventElapsedTime(&t, e0, e1));
    if (ms) *ms = t;
    count_mismatch_kernel<<<1024, 256>>>(d_dis, D.dis + g.drow_host[0], rows, d_bad);
    GH_CUDA(cudaGetLastError());
    unsigned long long bad = 0;
    GH_CUDA(cudaMemcpy(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost));
    if (mismatches) *mismatches = (int64_t)bad;
  } catch (...) {
    cleanup();
    throw;
  }
  cleanup();
}

// Position lists in the reference layout with graph-local ids: the host
// copies (L3) or the graph's range of the device arrays (L4).
void download_positions(const Graph &g, int *pos_id, int *pos_pos) {
  const int64_t np = g.pos_n;
  if ((int64_t)g.pos_id.size() == np && np) {
    if (pos_id) std::copy(g.pos_id.begin(), g.pos_id.end(), pos_id);
    if (pos_pos) std::copy(g.pos_pos.begin(), g.pos_pos.end(), pos_pos);
    return;
  }
  GH_CHECK(g.dev.pos_id && g.dev.pos_pos && g.dev.pos == np, H2H_ERR_STATE, "position lists not on the device");
  if (!np) return;
  if (pos_pos) GH_CUDA(cudaMemcpy(pos_pos, g.dev.pos_pos + g.dev.pos_base, sizeof(int) * np, cudaMemcpyDeviceToHost));
  if (pos_id) {
    GH_CUDA(cudaMemcpy(pos_id, g.dev.pos_id + g.dev.pos_base, sizeof(int) * np, cudaMemcpyDeviceToHost));
    if (g.dev.id_base)
      for (int64_t k = 0; k < np; k++) pos_id[k] -= g.dev.id_base;
  }
}

// The graph's rows are [row0, row1) of the device array
// (a batch's forest array holds other graphs' rows around them).
void download_labels(const Graph &g, int *dis_out) {
  const int n = g.n;
  host_tree(g);
  const int64_t r0 = g.row0, r1 = g.row1;
  GH_CHECK(r1 - r0 == g.dev.dis_padded, H2H_ERR_STATE, "label rows and device index disagree");
  std::vector<int> tmp(r1 - r0);
  GH_CUDA(cudaMemcpy(tmp.data(), g.dev.dis + r0, sizeof(int) * (r1 - r0), cudaMemcpyDeviceToHost));
  for (int v = 0; v < n; v++)
    std::copy(tmp.begin() + (g.drow_host[v] - r0), tmp.begin() + (g.drow_host[v] - r0) + g.depth[v],
              dis_out + g.dis_hash[v]);
}

}  // namespace gh
