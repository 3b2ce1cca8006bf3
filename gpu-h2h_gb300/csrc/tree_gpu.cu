// tree_gpu.cu -- the tree decomposition's structure and the fill's layout on
// the GPU, from the fathers the contraction picked:
//   getTreeStructure / OULADFS / makeOULAAndRMQ's tour (TreeStructure.cu:
//     102-262, 500-572): children in increasing id order (Childs), depths
//     (H2H_TreeHeight_Hash), firstAppeare and the Euler tour OULA_DFS_;
//   the heavy-path layout and root-path segments the L4 fill reads its
//     ancestors from, label row and position offsets (labels.cu).
// Several graphs' trees are built together, one root per graph, in the
// contraction's numbering.
//
// The reference walks the tree recursively on the host.  Here every quantity
// is a closed form over subtree sizes and sums along root paths:
//   * children: a stable radix sort of (father, v) pairs, v ascending;
//   * subtree sizes: by doubling, every node's count added to its ancestor 2^k
//     levels up;
//   * a child c of p is entered in the tour at first(p) + 1 + 2 * (sizes of
//     the siblings before c), and p follows c's subtree at first(c) +
//     2 * size(c) - 1; the preorder index is (first + depth - 1) / 2;
//   * depth, first, heavy-path position and the count of heavy-path tops on
//     the root path are sums of per-node offsets along the root path:
//     pointer jumping, about log2(height) synchronous rounds;
// The arrays stay on the device and the host waits once, for a few numbers per
// graph; the accessors download copies on request (host_tree).  On one GB300 a
// 1M-vertex graph's tree, table and fill layout took 15 ms with every array going through
// the host, 3 ms now.
// Every index a kernel writes through is checked against its array's size;
// a violation (only possible if the fathers are not one tree) sets an error
// word instead of writing.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "graph.h"
#include "quiet.h"
#include "sort.h"

namespace gh {

namespace {

// ------------------------------------------------------------ tree kernels

__device__ __forceinline__ void flag_err(int *err) { *err = 1; }

// The graph of a vertex: vbase holds the first vertex of every graph.
__device__ __forceinline__ int graph_of(const int *vbase, int K, int v) {
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (vbase[mid] <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void child_key_kernel(const int *father, int n, unsigned *key, int *val, int *cnt) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int f = father[v];
    key[v] = f >= 0 && f < n ? (unsigned)f : (unsigned)n;  // roots sort last
    val[v] = v;
    if (f >= 0 && f < n) atomicAdd(cnt + f, 1);
  }
}

// Subtree sizes by doubling: after k rounds size[v] counts v's descendants
// less than 2^k levels below it, and a round adds every node's count to the
// ancestor 2^k levels up: `in` holds what the last round sent to v, `out` takes
// what this one sends.  12 rounds of independent adds on a 2,588-deep tree of 1M
// nodes take 0.3 ms; climbing from the leaves is a chain of that many steps (1.7
// ms with an atomic at every step, 1.3 with atomics only where siblings meet).
// more: as in jump_kernel.
__global__ void size_round_kernel(const int *anc, int *anc_next, int *in, int *out, int *size, int n, int *more) {
  if (more[0] == 0 && more[1] == 0) return;
  bool m = false;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int u = anc[v], add = in[v], sz = size[v] + add;
    int up = -1;
    if (add) {
      size[v] = sz;
      in[v] = 0;  // the next round's out
    }
    if (u >= 0 && u < n) {
      atomicAdd(out + u, sz);
      up = anc[u];
      m |= up >= 0;
    }
    anc_next[v] = up;
  }
  if (__syncthreads_or(m) && threadIdx.x == 0) more[2] = 1;
}

// Per father, over its children in id order: the heavy child (largest
// subtree, the first one on ties), each child's tour offset 1 + 2 * (sizes of
// earlier siblings), its heavy-path offset (1 for the heavy child, else 1 +
// size(heavy) + sizes of earlier light siblings), whether it starts a heavy
// path, and its link up a heavy edge (the father when heavy, else itself).
__global__ void child_offsets_kernel(const int64_t *child_off, const int *childs, const int *size, const int *father,
                                     const int *vbase, int K, int n, int *off_first, int *off_hpos, int *seg_flag,
                                     int *hlink) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int64_t b = child_off[p], e = child_off[p + 1];
    int best = -1, bs = 0;
    for (int64_t k = b; k < e; k++) {
      const int c = childs[k];
      if (size[c] > bs) { bs = size[c]; best = c; }
    }
    int64_t S = 0, L = 0;
    for (int64_t k = b; k < e; k++) {
      const int c = childs[k];
      off_first[c] = (int)(1 + 2 * S);
      S += size[c];
      if (c == best) {
        off_hpos[c] = 1;
      } else {
        off_hpos[c] = (int)(1 + bs + L);
        L += size[c];
      }
      seg_flag[c] = c != best;
      hlink[c] = c == best ? p : c;
    }
    if (father[p] < 0) {
      off_first[p] = 0;
      off_hpos[p] = vbase[graph_of(vbase, K, p)];
      seg_flag[p] = 1;
      hlink[p] = p;
    }
  }
}

struct Jump {
  int *anc, *dep, *fst, *hp, *sg, *tl;
};

// One synchronous round of pointer jumping: every node adds its current
// ancestor's partial sums and jumps to that ancestor's ancestor; the heavy
// links jump likewise.  more[2] is set while any chain has not reached its top.
// Two rounds after none is left both buffers hold the result and the remaining
// rounds (enqueued for a chain of n nodes) return at once.
__global__ void jump_kernel(Jump a, Jump b, int n, int *more) {
  if (more[0] == 0 && more[1] == 0) return;
  bool m = false;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int u = a.anc[v];
    if (u >= 0 && u < n) {
      b.dep[v] = a.dep[v] + a.dep[u];
      b.fst[v] = a.fst[v] + a.fst[u];
      b.hp[v] = a.hp[v] + a.hp[u];
      b.sg[v] = a.sg[v] + a.sg[u];
      b.anc[v] = a.anc[u];
      m |= b.anc[v] >= 0;
    } else {
      b.dep[v] = a.dep[v];
      b.fst[v] = a.fst[v];
      b.hp[v] = a.hp[v];
      b.sg[v] = a.sg[v];
      b.anc[v] = -1;
    }
    const int t = a.tl[v];
    const int tt = t >= 0 && t < n ? a.tl[t] : t;
    b.tl[v] = tt;
    m |= tt != t;
  }
  if (__syncthreads_or(m) && threadIdx.x == 0) more[2] = 1;
}

// Euler tour (graph-local vertices, graph i's from 2 * vbase[i] - i) and
// heavy-path order; every write index range-checked.
__global__ void place_kernel(const int *father, const int *size, const int *dep, const int *fst, const int *hp,
                             const int *vbase, int K, int n, int *euler, int *hld, int *err) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int g = graph_of(vbase, K, v), vb = vbase[g], ng = vbase[g + 1] - vb;
    const int64_t L = 2 * (int64_t)ng - 1, f0 = fst[v], eb = 2 * (int64_t)vb - g;
    if (f0 < 0 || f0 >= L || dep[v] < 1 || dep[v] > ng || hp[v] < vb || hp[v] >= vb + ng) { flag_err(err); continue; }
    euler[eb + f0] = v - vb;
    const int p = father[v];
    if (p >= 0) {
      const int64_t back = f0 + 2 * (int64_t)size[v] - 1;
      if (back < 0 || back >= L || p < vb || p >= vb + ng) { flag_err(err); continue; }
      euler[eb + back] = p - vb;
    }
    hld[hp[v]] = v;
  }
}

// Position-list starts (a vertex's list and itself) and padded row lengths.
__global__ void row_sizes_kernel(const int64_t *list_off, const int *dep, int64_t *pos_hash, int *row, int n) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x) {
    pos_hash[v] = list_off[v] + v;
    row[v] = v < n ? (dep[v] + 3) & ~3 : 0;
  }
}

// What the host learns of a graph's tree; entry K only holds the ends of the
// last graph's arrays and the flags.
struct TreeSums {
  unsigned long long labels, updates;  // sum of depths; min-plus updates of the fill
  int64_t list0, row0, seg0;           // where the graph's lists, rows and segments start
  int height, max_segs, max_list, roots, head, head_size;
  int err, more;
};

__global__ void tree_sums_kernel(const int *father, const int *dep, const int *sg, const int64_t *list_off,
                                 const int *vbase, int K, int n, TreeSums *out) {
  int g = -1, height = 0, segs = 0, list = 0, roots = 0;
  unsigned long long labels = 0, updates = 0;
  auto flush = [&](bool whole) {
    if (whole) {  // the warp's lanes hold one graph's sums
      for (int o = 16; o > 0; o >>= 1) {
        labels += __shfl_xor_sync(0xffffffffu, labels, o);
        updates += __shfl_xor_sync(0xffffffffu, updates, o);
      }
      height = __reduce_max_sync(0xffffffffu, height);
      segs = __reduce_max_sync(0xffffffffu, segs);
      list = __reduce_max_sync(0xffffffffu, list);
      roots = __reduce_add_sync(0xffffffffu, roots);
      if (threadIdx.x & 31) return;
    }
    if (g < 0) return;
    atomicAdd(&out[g].labels, labels);
    atomicAdd(&out[g].updates, updates);
    atomicMax(&out[g].height, height);
    atomicMax(&out[g].max_segs, segs);
    atomicMax(&out[g].max_list, list);
    if (roots) atomicAdd(&out[g].roots, roots);
    labels = updates = 0;
    height = segs = list = roots = 0;
  };
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int gv = graph_of(vbase, K, v);
    if (gv != g) {
      flush(false);
      g = gv;
    }
    const int d = dep[v], m = (int)(list_off[v + 1] - list_off[v]);
    labels += d;
    updates += (unsigned long long)m * max(d - 2, 0);
    height = max(height, d);
    segs = max(segs, sg[v]);
    list = max(list, m);
    roots += father[v] < 0;
  }
  flush(__reduce_min_sync(0xffffffffu, g) == __reduce_max_sync(0xffffffffu, g));
}

__global__ void tree_ends_kernel(const int *elim, const int *father, const int *size, const int64_t *list_off,
                                 const int64_t *drow, const int64_t *seg_off, const int *vbase, int K,
                                 const int *err, const int *more, TreeSums *out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= K; i += gridDim.x * blockDim.x) {
    const int vb = vbase[i];
    out[i].list0 = list_off[vb];
    out[i].row0 = drow[vb];
    out[i].seg0 = seg_off[vb];
    if (i < K) {
      const int h = elim[vbase[i + 1] - 1];
      const bool ok = h >= vb && h < vbase[i + 1] && father[h] < 0;
      out[i].head = h - vb;
      out[i].head_size = ok ? size[h] : -1;
    } else {
      out[i].err = *err;
      out[i].more = *more;
    }
  }
}

__global__ void fill_value_kernel(int *a, int n, int value) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = value;
}

}  // namespace

void build_tree_gpu(const std::vector<Graph *> &gs) {
  Clock clk;
  const std::shared_ptr<TreeStore> tree = gs[0]->tree;
  GH_CHECK(tree && tree->gs == gs, H2H_ERR_STATE, "fathers missing");
  TreeStore &T = *tree;
  const int K = (int)gs.size(), n = T.n;
  const ListStore &lists = gs[0]->dev.lists;
  int dev = 0, nsm = 0;
  GH_CUDA(cudaGetDevice(&dev));
  GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int grid = std::max(1, std::min(nsm * 8, (n + 255) / 256));
  cudaStream_t s = 0;
  Workspace ws;
  T.layout = std::make_shared<DeviceArena>();
  T.tour = std::make_unique<DeviceArena>();
  T.depth = T.mem.get<int>(n);
  T.drow = T.mem.get<int64_t>(n + 1);
  T.pos_hash = T.mem.get<int64_t>(n + 1);
  T.hld = T.layout->get<int>(n);
  T.htop = T.layout->get<int>(n);
  T.hpos = T.layout->get<int>(n);
  T.seg_off = T.layout->get<int64_t>(n + 1);
  T.first = T.tour->get<int>(n);
  T.euler = T.tour->get<int>(2 * (int64_t)n - K);
  const int rounds = bits_for(n) + 3;
  const bool trace = std::getenv("GPUH2H_TRACE") != nullptr;
  Clock tclk;
  auto mark = [&](const char *what) {
    if (!trace) return;
    cudaDeviceSynchronize();
    std::fprintf(stderr, "[gpuh2h] tree: %s %.3f ms\n", what, tclk.us() / 1e3);
    tclk.reset();
  };
  const int *father = T.father;
  int *vbase = ws.get<int>(K + 1), *cnt = ws.get<int>(n + 1), *flags = ws.get<int>(rounds + 3);  // err, then more
  int *err = flags, *more = flags + 1;
  GH_CUDA(cudaMemcpyAsync(vbase, T.vbase.data(), sizeof(int) * (K + 1), cudaMemcpyHostToDevice, s));
  GH_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * (n + 1), s));
  GH_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * (rounds + 3), s));
  fill_value_kernel<<<1, 32, 0, s>>>(more, 2, 1);
  // children in id order
  unsigned *key = ws.get<unsigned>(n);
  int *val = ws.get<int>(n);
  child_key_kernel<<<grid, 256, 0, s>>>(father, n, key, val, cnt);
  GH_CUDA(cudaGetLastError());
  radix_sort_pairs(key, val, n, bits_for(n), ws, s);
  const int *childs = val;
  int64_t *child_off = ws.get<int64_t>(n + 1);
  exclusive_scan<int>(cnt, child_off, n + 1, ws, s);
  mark("children");
  // subtree sizes
  int *size = ws.get<int>(n), *anc = ws.get<int>(n), *anc_next = ws.get<int>(n);
  int *arrived = ws.get<int>(n), *sent = ws.get<int>(n), *more_sizes = ws.get<int>(rounds + 2);
  GH_CUDA(cudaMemsetAsync(arrived, 0, sizeof(int) * n, s));
  GH_CUDA(cudaMemsetAsync(sent, 0, sizeof(int) * n, s));
  GH_CUDA(cudaMemsetAsync(more_sizes, 0, sizeof(int) * (rounds + 2), s));
  fill_value_kernel<<<1, 32, 0, s>>>(more_sizes, 2, 1);
  fill_value_kernel<<<grid, 256, 0, s>>>(size, n, 1);
  GH_CUDA(cudaMemcpyAsync(anc, father, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  for (int r = 0; r < rounds; r++) {
    size_round_kernel<<<grid, 256, 0, s>>>(anc, anc_next, arrived, sent, size, n, more_sizes + r);
    GH_CUDA(cudaGetLastError());
    std::swap(anc, anc_next);
    std::swap(arrived, sent);
  }
  mark("sizes");
  // per-child offsets, then root-path sums by pointer jumping
  Jump A, B;
  for (Jump *J : {&A, &B}) {
    J->anc = ws.get<int>(n);
    J->dep = ws.get<int>(n);
    J->fst = ws.get<int>(n);
    J->hp = ws.get<int>(n);
    J->sg = ws.get<int>(n + 1);
    J->tl = ws.get<int>(n);
    GH_CUDA(cudaMemsetAsync(J->sg + n, 0, sizeof(int), s));
  }
  child_offsets_kernel<<<grid, 256, 0, s>>>(child_off, childs, size, father, vbase, K, n, A.fst, A.hp, A.sg, A.tl);
  GH_CUDA(cudaMemcpyAsync(A.anc, father, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  fill_value_kernel<<<grid, 256, 0, s>>>(A.dep, n, 1);  // every depth starts at one step
  GH_CUDA(cudaGetLastError());
  for (int r = 0; r < rounds; r++) {
    jump_kernel<<<grid, 256, 0, s>>>(A, B, n, more + r);
    GH_CUDA(cudaGetLastError());
    std::swap(A, B);
  }
  const std::pair<int *, const int *> copies[] = {{T.depth, A.dep}, {T.first, A.fst}, {T.hpos, A.hp}, {T.htop, A.tl}};
  for (const auto &c : copies) GH_CUDA(cudaMemcpyAsync(c.first, c.second, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  mark("root paths");
  // tour, heavy-path order, segment, row and position offsets
  place_kernel<<<grid, 256, 0, s>>>(father, size, T.depth, T.first, T.hpos, vbase, K, n, T.euler, T.hld, err);
  exclusive_scan<int>(A.sg, T.seg_off, n + 1, ws, s);
  row_sizes_kernel<<<grid, 256, 0, s>>>(lists.off, T.depth, T.pos_hash, cnt, n);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(cnt, T.drow, n + 1, ws, s);
  TreeSums *d_sums = ws.get<TreeSums>(K + 1);
  GH_CUDA(cudaMemsetAsync(d_sums, 0, sizeof(TreeSums) * (K + 1), s));
  tree_sums_kernel<<<grid, 256, 0, s>>>(father, T.depth, A.sg, lists.off, vbase, K, n, d_sums);
  tree_ends_kernel<<<1, 256, 0, s>>>(T.elim, father, size, lists.off, T.drow, T.seg_off, vbase, K, err,
                                     more + rounds + 1, d_sums);
  GH_CUDA(cudaGetLastError());
  std::vector<TreeSums> sums(K + 1);
  GH_CUDA(cudaMemcpy(sums.data(), d_sums, sizeof(TreeSums) * (K + 1), cudaMemcpyDeviceToHost));
  mark("tour and offsets");
  GH_CHECK(!sums[K].err && !sums[K].more, H2H_ERR_STATE, "decomposition is not a single tree");
  T.height = T.max_segs = T.max_list = 0;
  T.dis_total = sums[K].row0;
  T.seg_total = sums[K].seg0;
  T.pos_total = sums[K].list0 + n;
  const long long us = clk.us();
  for (int i = 0; i < K; i++) {
    Graph &g = *gs[i];
    const TreeSums &S = sums[i];
    GH_CHECK(S.roots == 1 && S.head_size == g.n, H2H_ERR_STATE, "decomposition is not a single tree");
    T.height = std::max(T.height, S.height);
    T.max_segs = std::max(T.max_segs, S.max_segs);
    T.max_list = std::max(T.max_list, S.max_list);
    g.head = S.head;
    g.tree_height = g.n_levels = S.height;
    g.h2h_size = (int64_t)S.labels;
    g.x_total = sums[i + 1].list0 - S.list0;
    g.decomposition_size = g.x_total + g.n;
    g.updates = (int64_t)S.updates;
    g.row0 = S.row0;
    g.row1 = sums[i + 1].row0;
    g.euler_n = 2 * (int64_t)g.n - 1;
    g.dev.x_base = S.list0;
    g.dev.id_base = T.vbase[i];
    g.t.tree = us / K;
  }
}

// The order, the tree and the list offsets from the device (nullptr: not asked for).
static void read_tree(const Graph &g, int *order, int *father, int *depth, int *first, int64_t *x_off) {
  const TreeStore &T = *g.tree;
  const int n = g.n, vb = g.dev.id_base;
  GH_CHECK(T.depth && g.dev.first, H2H_ERR_STATE, "tree not built");
  RelaxedCapture relaxed;
  QuietStream q;
  auto down = [&](auto *to, const auto *from, int64_t count) {
    if (to) q.read(to, from, sizeof(*to) * (size_t)count);
  };
  down(order, T.elim + vb, n);
  down(father, T.father + vb, n);
  down(depth, T.depth + vb, n);
  down(first, g.dev.first, n);
  down(x_off, g.dev.lists.off + vb, (int64_t)n + 1);
  for (int v = 0; v < n && vb && order; v++) order[v] -= vb;
  for (int v = 0; v < n && vb && father; v++)
    if (father[v] >= 0) father[v] -= vb;
  for (int v = 0; v <= n && g.dev.x_base && x_off; v++) x_off[v] -= g.dev.x_base;
}

// The same into a caller's arrays, from the host copies where there are some.
void download_tree(const Graph &g, int *order, int *father, int *depth, int *first, int64_t *x_off) {
  std::unique_lock<std::mutex> lock(g.host_lock);
  if (g.tree && (int)g.elim.size() != g.n) {
    lock.unlock();
    read_tree(g, order, father, depth, first, x_off);
    return;
  }
  if (order) std::copy(g.elim.begin(), g.elim.end(), order);
  if (father) std::copy(g.father.begin(), g.father.end(), father);
  if (depth) std::copy(g.depth.begin(), g.depth.end(), depth);
  if (first) std::copy(g.first.begin(), g.first.end(), first);
  if (x_off) std::copy(g.x_off.begin(), g.x_off.end(), x_off);
}

// Host copies of the order, the tree and the offsets, made when they are first
// asked for: the level order is the preorder (the order of first appearances)
// sorted stably by depth, since a breadth-first walk reaches the nodes of one
// depth in the order a depth-first walk with the same child order does.
const Graph &host_tree(const Graph &gc) {
  std::lock_guard<std::mutex> lock(gc.host_lock);
  if (!gc.tree || (int)gc.elim.size() == gc.n) return gc;
  Graph &g = const_cast<Graph &>(gc);
  const int n = g.n;
  std::vector<int> order(n);
  g.father.resize(n);
  g.depth.resize(n);
  g.first.resize(n);
  g.x_off.resize((size_t)n + 1);
  g.drow_host.resize((size_t)n + 1);
  read_tree(g, order.data(), g.father.data(), g.depth.data(), g.first.data(), g.x_off.data());
  {
    RelaxedCapture relaxed;
    QuietStream q;
    q.read(g.drow_host.data(), g.tree->drow + g.dev.id_base, sizeof(int64_t) * ((size_t)n + 1));
  }
  g.pos_hash.resize((size_t)n + 1);
  g.dis_hash.assign((size_t)n + 1, 0);
  std::vector<int> pre(n);
  g.tree_hash.assign((size_t)g.tree_height + 1, 0);
  for (int v = 0; v < n; v++) {
    g.dis_hash[v + 1] = g.dis_hash[v] + g.depth[v];
    pre[(g.first[v] + g.depth[v] - 1) / 2] = v;
    g.tree_hash[g.depth[v]]++;
  }
  for (int v = 0; v <= n; v++) g.pos_hash[v] = g.x_off[v] + v;
  for (int l = 0; l < g.tree_height; l++) g.tree_hash[l + 1] += g.tree_hash[l];
  std::vector<int> at(g.tree_hash.begin(), g.tree_hash.end() - 1);
  g.tree_bfs.resize(n);
  for (int v : pre) g.tree_bfs[at[g.depth[v] - 1]++] = v;
  g.elim.swap(order);
  return gc;
}

}  // namespace gh
