// elim_sets.cu -- the per-cell elimination sets, the LUB capacities and the
// per-cell list bounds, Graph::makeAdjcentNode(0) (GraphPartition.cu:178-308),
// on the GPU for one graph or a batch of graphs.
//
// Bottom-up over partition levels h = H..1: a vertex of a level-h cell that
// has no alive neighbour outside the cell is interior and joins the cell's
// candidate range of `elim`; the others stay alive for the parent level.
// The capacity of a vertex's adjacency slot range is the largest (alive cell
// size + alive out-of-cell arcs) over the levels it takes part in, at least
// its input degree: it bounds every list the partition-level contraction
// builds, so the device lists never move.  The same pass gives every cell its
// list bound -- alive cell size - 1 + alive out-of-cell arcs + parallel arcs,
// maximised over its alive members -- which sizes the elimination kernels'
// staging.
//
// Cell ranges of `elim` are laid out as the reference lays them (levels
// bottom-up, a level's cells from the highest index down).  Inside a range
// the reference keeps std::map order (by id); the elimination kernels pick by
// a strict key over the whole range, so that order reaches no result, and a
// range here holds its vertices in partition-array order.
//
// Work unit: a chunk of at most kChunk partition positions of one cell.  Per
// level: alive members per cell (atomic count); per member the out-of-cell
// arcs, interior flag, capacity and cell bound, interior count per chunk; a
// one-block segmented scan over the level's chunks (per graph, continuing
// from the levels below) gives every chunk and cell its offset; each chunk
// writes its interior vertices in position order and retires them.  The list
// ranges follow from a scan of the capacities in partition-array order
// (GraphPartition.cu:270-292).  The sets stay on the device: the host reads the
// per-cell tables and a few sums (with the arrays going through the host the
// sets and the elimination's tables of a 1M-vertex graph took 8.7 ms, now 2.5).
#include <algorithm>

#include "graph.h"
#include "scan.h"

namespace gh {

namespace {

constexpr int kChunk = 1024;   // partition positions per work unit
constexpr int kThreads = 256;

struct Chunk {
  int cell;    // global cell id (graph's cell base + cell index)
  int graph;
  int start;   // forest partition positions [start, end)
  int end;
};

struct SetsGraph {
  const int *off, *nbr;    // n + 1 offsets, local neighbour ids
  const int *part, *pos;   // local vertex per local position and its inverse
  int vbase;               // the graph's first forest vertex and position
};

struct SetsArgs {
  const Chunk *chunks;     // this level's chunks, graph-major, cells from the highest index down
  int nchunks;
  const SetsGraph *graphs;
  int ngraphs;
  int *dup;                // parallel arcs per vertex (forest)
  const int *cut_l, *cut_r;  // per global cell, local positions
  unsigned char *alive;    // per forest vertex
  unsigned char *flag;     // per forest position: interior at this level
  int *cap, *deg;          // per forest vertex
  int *cap_max;
  int *cell_sz, *cell_bound, *cell_start, *cell_count;  // per global cell
  int *chunk_cnt, *chunk_out;  // per chunk of the level
  int *gfill;              // per graph: elim entries written so far
  int *elim;               // forest vertices, graph i's from its vbase
};

__device__ __forceinline__ int block_sum(int v, int *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  int t = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
  return t;  // valid in thread 0
}

// The graph of a forest vertex.
__device__ __forceinline__ const SetsGraph &graph_of(const SetsArgs &A, int V) {
  int lo = 0, hi = A.ngraphs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (A.graphs[mid].vbase <= V) lo = mid;
    else hi = mid - 1;
  }
  return A.graphs[lo];
}

// Degree of every vertex, which its capacity starts from, and its parallel
// arcs: entries whose neighbour id appeared earlier in the same input list.
// One warp per vertex.
__global__ void dup_kernel(SetsArgs A, int N) {
  const int lane = threadIdx.x & 31;
  for (int64_t V = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; V < N;
       V += (gridDim.x * (int64_t)blockDim.x) >> 5) {
    const SetsGraph &G = graph_of(A, (int)V);
    const int v = (int)V - G.vbase;
    const int *nb = G.nbr;
    const int b = G.off[v], e = G.off[v + 1];
    int d = 0;
    for (int i = b + lane; i < e; i += 32) {
      const int x = nb[i];
      bool seen = false;
      for (int j = b; j < i && !seen; j++) seen = nb[j] == x;
      d += seen;
    }
    for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
    if (lane == 0) {
      A.dup[V] = d;
      A.deg[V] = A.cap[V] = e - b;
      A.alive[V] = 1;
    }
  }
}

// Alive members per cell.
__global__ void __launch_bounds__(kThreads) count_alive_kernel(SetsArgs A) {
  __shared__ int red[32];
  for (int k = blockIdx.x; k < A.nchunks; k += gridDim.x) {
    const Chunk c = A.chunks[k];
    const SetsGraph G = A.graphs[c.graph];
    int n = 0;
    for (int j = c.start + threadIdx.x; j < c.end; j += blockDim.x) n += A.alive[G.vbase + G.part[j - G.vbase]];
    const int t = block_sum(n, red);
    if (threadIdx.x == 0 && t) atomicAdd(A.cell_sz + c.cell, t);
  }
}

// Per alive member: alive out-of-cell arcs, interior flag, capacity, bound.
__global__ void __launch_bounds__(kThreads) classify_kernel(SetsArgs A) {
  __shared__ int red[32];
  for (int k = blockIdx.x; k < A.nchunks; k += gridDim.x) {
    const Chunk c = A.chunks[k];
    const SetsGraph G = A.graphs[c.graph];
    const int vb = G.vbase;
    const int *off = G.off, *nb = G.nbr;
    const int cl = A.cut_l[c.cell], cr = A.cut_r[c.cell];  // local positions
    const int sz = A.cell_sz[c.cell];
    int interior = 0, bound = 0;
    for (int j = c.start + threadIdx.x; j < c.end; j += blockDim.x) {
      const int v = G.part[j - vb];  // local
      unsigned char f = 0;
      if (A.alive[vb + v]) {
        int out = 0;
        for (int e = off[v]; e < off[v + 1]; e++) {
          const int u = nb[e];
          const int pu = G.pos[u];
          out += A.alive[vb + u] && (pu < cl || pu >= cr);
        }
        f = out == 0;
        interior += f;
        A.cap[vb + v] = max(A.cap[vb + v], sz + out);
        bound = max(bound, sz - 1 + out + A.dup[vb + v]);
      }
      A.flag[j] = f;
    }
    const int t = block_sum(interior, red);
    if (threadIdx.x == 0) A.chunk_cnt[k] = t;
    for (int o = 16; o > 0; o >>= 1) bound = max(bound, __shfl_down_sync(0xffffffffu, bound, o));
    if ((threadIdx.x & 31) == 0 && bound > 0) atomicMax(A.cell_bound + c.cell, bound);
  }
}

// One block: offsets of the level's chunks, graph by graph in chunk order,
// continuing each graph's range from its earlier levels; cell starts and
// counts; the graphs' running totals.
__global__ void __launch_bounds__(1024) scan_kernel(SetsArgs A) {
  __shared__ int s_val[1024], s_flag[1024];
  __shared__ int s_carry, s_graph;
  if (threadIdx.x == 0) {
    s_carry = 0;
    s_graph = -1;
  }
  __syncthreads();
  for (int base = 0; base < A.nchunks; base += blockDim.x) {
    const int k = base + threadIdx.x;
    const bool in = k < A.nchunks;
    const Chunk c = in ? A.chunks[k] : Chunk{0, -1, 0, 0};
    const int cnt = in ? A.chunk_cnt[k] : 0;
    // inclusive scan of cnt with a reset at every graph boundary
    const bool head = in && (k == 0 || A.chunks[k - 1].graph != c.graph);
    int v = cnt, hd = head;
    s_val[threadIdx.x] = v;
    __syncthreads();
    // segmented Hillis-Steele: flags travel with the values
    s_flag[threadIdx.x] = hd;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {
      int pv = 0, pf = 0;
      if ((int)threadIdx.x >= o) { pv = s_val[threadIdx.x - o]; pf = s_flag[threadIdx.x - o]; }
      __syncthreads();
      if ((int)threadIdx.x >= o && !hd) { v += pv; hd |= pf; }
      s_val[threadIdx.x] = v;
      s_flag[threadIdx.x] = hd;
      __syncthreads();
    }
    // exclusive offset inside the graph's level: the carry applies to the
    // leading segment when it continues the previous tile's graph
    const int carry = (!hd && in && c.graph == s_graph) ? s_carry : 0;
    if (in) {
      const int excl = v - cnt + carry;
      A.chunk_out[k] = A.gfill[c.graph] + excl;
      const bool first_of_cell = k == 0 || A.chunks[k - 1].cell != c.cell;
      if (first_of_cell) A.cell_start[c.cell] = A.gfill[c.graph] + excl;
    }
    __syncthreads();
    // the last chunk of a graph in this level closes the graph's total
    if (in) {
      const bool last_of_graph = k == A.nchunks - 1 || A.chunks[k + 1].graph != c.graph;
      if (last_of_graph) A.gfill[c.graph] += v + carry;
    }
    __syncthreads();
    if (k == min(base + (int)blockDim.x, A.nchunks) - 1) {  // the tile's last chunk carries on
      s_carry = v + carry;
      s_graph = c.graph;
    }
    __syncthreads();
  }
}

// Cell counts from the chunk offsets (the chunks of a cell are consecutive).
__global__ void cell_count_kernel(SetsArgs A) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < A.nchunks; k += gridDim.x * blockDim.x) {
    const Chunk c = A.chunks[k];
    const bool last_of_cell = k == A.nchunks - 1 || A.chunks[k + 1].cell != c.cell;
    if (last_of_cell) A.cell_count[c.cell] = A.chunk_out[k] + A.chunk_cnt[k] - A.cell_start[c.cell];
  }
}

// Each chunk writes its interior vertices in position order and retires them.
__global__ void __launch_bounds__(kThreads) write_kernel(SetsArgs A) {
  __shared__ int s_warp[kThreads / 32];
  __shared__ int s_base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = blockIdx.x; k < A.nchunks; k += gridDim.x) {
    const Chunk c = A.chunks[k];
    const SetsGraph G = A.graphs[c.graph];
    const int vb = G.vbase;
    if (threadIdx.x == 0) s_base = A.chunk_out[k];
    __syncthreads();
    for (int j0 = c.start; j0 < c.end; j0 += blockDim.x) {
      const int j = j0 + threadIdx.x;
      const bool f = j < c.end && A.flag[j];
      const unsigned bal = __ballot_sync(0xffffffffu, f);
      if (lane == 0) s_warp[wid] = __popc(bal);
      __syncthreads();
      int before = 0, total = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        if (w < wid) before += s_warp[w];
        total += s_warp[w];
      }
      if (f) {
        const int V = vb + G.part[j - vb];
        A.elim[vb + s_base + before + __popc(bal & ((1u << lane) - 1u))] = V;
        A.alive[V] = 0;
      }
      __syncthreads();
      if (threadIdx.x == 0) s_base += total;
      __syncthreads();
    }
  }
}

// Capacities in partition-array order (len[N] = 0) and the largest.
__global__ void capacity_order_kernel(SetsArgs A, int *len, int N) {
  int most = 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j <= N; j += gridDim.x * blockDim.x) {
    int c = 0;
    if (j < N) {
      const SetsGraph &G = graph_of(A, j);
      c = A.cap[G.vbase + G.part[j - G.vbase]];
    }
    len[j] = c;
    most = max(most, c);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(A.cap_max, most);
}

// List starts per vertex, and where every graph's lists end.
__global__ void slot_kernel(SetsArgs A, const int64_t *start, int64_t *slot, int64_t *graph_end, int N) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < N; j += gridDim.x * blockDim.x) {
    const SetsGraph &G = graph_of(A, j);
    slot[G.vbase + G.part[j - G.vbase]] = start[j];
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.ngraphs; i += gridDim.x * blockDim.x)
    graph_end[i] = start[i + 1 < A.ngraphs ? A.graphs[i + 1].vbase : N];
}

}  // namespace

void build_elimination_sets(const std::vector<Graph *> &gs) {
  Clock clk;
  const int K = (int)gs.size();
  GH_CHECK(K >= 1, H2H_ERR_ARG, "no graph");
  std::vector<int> vbase(K), cbase(K);
  int64_t N = 0, M = 0, CELLS = 0;
  int Hmax = 0;
  for (int i = 0; i < K; i++) {
    const Graph &g = *gs[i];
    vbase[i] = (int)N;
    cbase[i] = (int)CELLS;
    N += g.n;
    M += g.m;
    CELLS += (int64_t(1) << g.H) - 1;
    Hmax = std::max(Hmax, g.H);
    GH_CHECK((int64_t)g.cut_l.size() >= (int64_t(1) << g.H) - 1, H2H_ERR_FORMAT, "cut table shorter than 2^H - 1");
  }
  GH_CHECK(N + K < INT32_MAX && M < INT32_MAX && CELLS < INT32_MAX, H2H_ERR_ARG, "batch too large");
  // ---- chunks per level (graph-major, cells from the highest index down),
  // with the reference's checks on the cut rows
  std::vector<std::vector<Chunk>> lv(Hmax + 1);
  std::vector<int> f_cut_l(CELLS), f_cut_r(CELLS);
  for (int i = 0; i < K; i++) {
    const Graph &g = *gs[i];
    for (int h = g.H; h > 0; h--) {
      const int64_t lo = (int64_t(1) << (h - 1)) - 1, hi = (int64_t(1) << h) - 2;
      std::vector<std::pair<int, int>> rs;
      for (int64_t c = lo; c <= hi; c++) {
        const int cl = std::max(0, g.cut_l[c]), cr = std::min(g.n, g.cut_r[c]);
        f_cut_l[cbase[i] + c] = cl;
        f_cut_r[cbase[i] + c] = std::max(cl, cr);
        if (cr > cl) rs.push_back({cl, cr});
      }
      std::sort(rs.begin(), rs.end());
      for (size_t r = 1; r < rs.size(); r++)
        GH_CHECK(rs[r].first >= rs[r - 1].second, H2H_ERR_FORMAT, "partition cells of one level overlap");
      for (int64_t c = hi; c >= lo; c--) {
        const int cl = f_cut_l[cbase[i] + c], cr = f_cut_r[cbase[i] + c];
        const int cell = cbase[i] + (int)c;
        if (cr <= cl) {
          lv[h].push_back({cell, i, vbase[i] + cl, vbase[i] + cl});  // empty: still gets a start
          continue;
        }
        for (int s = cl; s < cr; s += kChunk)
          lv[h].push_back({cell, i, vbase[i] + s, vbase[i] + std::min(cr, s + kChunk)});
      }
    }
  }
  int64_t nchunk_max = 1, nchunk_total = 0;
  for (int h = 1; h <= Hmax; h++) {
    nchunk_max = std::max<int64_t>(nchunk_max, (int64_t)lv[h].size());
    nchunk_total += (int64_t)lv[h].size();
  }
  // ---- device state
  Workspace ws;
  auto sets = std::make_shared<SetsStore>();
  sets->gs = gs;
  std::vector<int> f_cell(4 * CELLS), f_fill(K + 1);  // size, bound, start, count; placed per graph, largest capacity
  std::vector<int64_t> graph_end(K);
  {
    SetsArgs S{};
    sets->elim = sets->mem.get<int>(N);
    sets->cap = sets->mem.get<int>(N);
    sets->deg = sets->mem.get<int>(N);
    sets->slot = sets->mem.get<int64_t>(N);
    SetsGraph *d_graphs = ws.get<SetsGraph>(K);
    int *d_dup = ws.get<int>(N), *d_len = ws.get<int>(N + 1);
    int64_t *d_start = ws.get<int64_t>(N + 1), *d_end = ws.get<int64_t>(K);
    int *d_cut_l = ws.get<int>(CELLS), *d_cut_r = ws.get<int>(CELLS);
    unsigned char *d_alive = ws.get<unsigned char>(N), *d_flag = ws.get<unsigned char>(N);
    int *d_cell = ws.get<int>(4 * CELLS);
    int *d_chunk_cnt = ws.get<int>(nchunk_max), *d_chunk_out = ws.get<int>(nchunk_max);
    Chunk *d_chunks = ws.get<Chunk>(std::max<int64_t>(nchunk_total, 1));
    int *d_fill = ws.get<int>(K + 1);
    std::vector<SetsGraph> table(K);
    for (int i = 0; i < K; i++) {
      const DeviceInput &in = input_device(*gs[i]);
      table[i] = {in.off, in.v, in.part, in.pos, vbase[i]};
    }
    GH_CUDA(cudaMemcpy(d_graphs, table.data(), sizeof(SetsGraph) * K, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_cut_l, f_cut_l.data(), sizeof(int) * CELLS, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_cut_r, f_cut_r.data(), sizeof(int) * CELLS, cudaMemcpyHostToDevice));
    {
      int64_t at = 0;
      for (int h = Hmax; h >= 1; h--) {
        if (!lv[h].empty())
          GH_CUDA(cudaMemcpy(d_chunks + at, lv[h].data(), sizeof(Chunk) * lv[h].size(), cudaMemcpyHostToDevice));
        at += (int64_t)lv[h].size();
      }
    }
    GH_CUDA(cudaMemset(d_cell, 0, sizeof(int) * 4 * CELLS));
    GH_CUDA(cudaMemset(d_fill, 0, sizeof(int) * (K + 1)));
    S.graphs = d_graphs;
    S.ngraphs = K;
    S.dup = d_dup;
    S.cut_l = d_cut_l;
    S.cut_r = d_cut_r;
    S.alive = d_alive;
    S.flag = d_flag;
    S.cap = sets->cap;
    S.deg = sets->deg;
    S.cap_max = d_fill + K;
    S.cell_sz = d_cell;
    S.cell_bound = d_cell + CELLS;
    S.cell_start = d_cell + 2 * CELLS;
    S.cell_count = d_cell + 3 * CELLS;
    S.chunk_cnt = d_chunk_cnt;
    S.chunk_out = d_chunk_out;
    S.gfill = d_fill;
    S.elim = sets->elim;
    int dev = 0, nsm = 0;
    GH_CUDA(cudaGetDevice(&dev));
    GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    if (N) {
      dup_kernel<<<std::max(1, std::min<int>(nsm * 16, (int)((N * 32 + 255) / 256))), 256>>>(S, (int)N);
      GH_CUDA(cudaGetLastError());
    }
    int64_t at = 0;
    for (int h = Hmax; h >= 1; h--) {
      const int nc = (int)lv[h].size();
      if (nc == 0) continue;
      S.chunks = d_chunks + at;
      S.nchunks = nc;
      at += nc;
      const int grid = std::max(1, std::min(nc, nsm * 8));
      count_alive_kernel<<<grid, kThreads>>>(S);
      classify_kernel<<<grid, kThreads>>>(S);
      scan_kernel<<<1, 1024>>>(S);
      cell_count_kernel<<<std::max(1, std::min(nsm * 4, (nc + 255) / 256)), 256>>>(S);
      write_kernel<<<grid, kThreads>>>(S);
      GH_CUDA(cudaGetLastError());
    }
    const int grid = std::max(1, std::min<int>(nsm * 8, (int)((N + 256) / 256)));
    capacity_order_kernel<<<grid, 256>>>(S, d_len, (int)N);
    GH_CUDA(cudaGetLastError());
    exclusive_scan<int>(d_len, d_start, N + 1, ws, 0);
    slot_kernel<<<grid, 256>>>(S, d_start, sets->slot, d_end, (int)N);
    GH_CUDA(cudaGetLastError());
    GH_CUDA(cudaMemcpy(f_fill.data(), d_fill, sizeof(int) * (K + 1), cudaMemcpyDeviceToHost));
    GH_CUDA(cudaMemcpy(graph_end.data(), d_end, sizeof(int64_t) * K, cudaMemcpyDeviceToHost));
    GH_CUDA(cudaMemcpy(f_cell.data(), d_cell, sizeof(int) * 4 * CELLS, cudaMemcpyDeviceToHost));
  }
  ws.release();
  sets->cap_max = f_fill[K];
  const long long t_sets = clk.us();
  // ---- per graph: tables, LUB layout (GraphPartition.cu:270-292), level rates
  for (int i = 0; i < K; i++) {
    Graph &g = *gs[i];
    clk.reset();
    GH_CHECK(f_fill[i] == g.n, H2H_ERR_FORMAT,
             "partition does not cover every vertex (root cut row must span all vertices)");
    const int64_t cells = (int64_t(1) << g.H) - 1;
    const int *bound = f_cell.data() + CELLS + cbase[i], *start = bound + CELLS, *count = start + CELLS;
    g.cell_start.assign(start, start + cells);
    g.cell_count.assign(count, count + cells);
    g.cell_bound.resize(cells);
    for (int64_t c = 0; c < cells; c++) g.cell_bound[c] = std::max(1, bound[c]);
    g.layer_rate.assign(g.H + 1, 0.0);
    int64_t done = 0;
    for (int h = g.H; h > 0; h--) {
      const int64_t lo = (int64_t(1) << (h - 1)) - 1, hi = (int64_t(1) << h) - 2;
      for (int64_t c = lo; c <= hi; c++) done += g.cell_count[c];
      g.layer_rate[h] = g.n ? (double)done / g.n : 0.0;
    }
    g.lub = graph_end[i] - (i ? graph_end[i - 1] : 0);
    g.sets = sets;
    g.t.rank_tree = t_sets;
    g.t.lub = clk.us();
  }
}

}  // namespace gh
