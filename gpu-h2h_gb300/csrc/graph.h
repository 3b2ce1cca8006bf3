// graph.h -- the handle behind h2h_graph: host arrays of one road graph, its
// tree decomposition and its no-hub labels, plus the device-resident index.
#pragma once

#include <cstdint>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "arena.h"
#include "common.h"

namespace gh {

struct Graph;

// X(v)\{v} lists after contraction, on the device, in the numbering of the
// contraction that produced them (a batch's forest, or one graph): list of
// vertex v is id[off[v] .. off[v+1]) (neighbour ids, sorted) with shortcut
// weights w.  `keep` owns the arrays.
struct ListStore {
  int64_t *off = nullptr;
  int *id = nullptr, *w = nullptr;
  int64_t total = 0;
  std::shared_ptr<void> keep;
};

// A loaded graph's input on the device (input_gpu.cu): stored arcs in CSR
// order, the vertex at every partition position and its inverse.
struct DeviceInput {
  DeviceArena mem;
  int *off = nullptr, *v = nullptr, *w = nullptr, *part = nullptr, *pos = nullptr;
  int device = 0;
  ~DeviceInput();
};

// The same on the host.
struct HostInput {
  std::vector<int> adj_off;        // CSR offsets of adjList in file order [n+1]
  std::vector<int> adj_v, adj_w;   // arcs, self loops dropped, parallel arcs kept
  std::vector<int> part_ids;       // NE_P[idx].NodeID (partition array)
  std::vector<int> id_hash;        // ID_hash[vertex] = idx
};

// The elimination sets of the graphs built together, on the device
// (elim_sets.cu) until they are contracted, in one numbering (graph i's
// vertices from the sum of the sizes before it): vertices by elimination
// range, list capacities, input degrees, list starts in partition-array order
// and the largest capacity.
struct SetsStore {
  DeviceArena mem;
  std::vector<Graph *> gs;
  int *elim = nullptr, *cap = nullptr, *deg = nullptr;
  int64_t *slot = nullptr;
  int cap_max = 0;
};

// The trees of the graphs contracted together, on the device in the
// contraction's numbering (tree_gpu.cu): graph i's vertices are vbase[i] ..
// vbase[i + 1] - 1.
struct TreeStore {
  DeviceArena mem;                // of the arrays that live as long as the labels
  std::vector<Graph *> gs;
  std::vector<int> vbase;         // [graphs + 1]
  int n = 0;
  int *elim = nullptr, *father = nullptr, *depth = nullptr;  // order; father (-1: a root); depth, roots 1
  int64_t *drow = nullptr, *pos_hash = nullptr;              // padded row and position-list offsets [n + 1]
  int64_t pos_total = 0, dis_total = 0, seg_total = 0;
  int height = 0, max_segs = 0, max_list = 0;
  // until the sparse tables are built: first appearance (per graph) and the
  // Euler tours (graph-local vertices), graph i's from 2 * vbase[i] - i
  std::unique_ptr<DeviceArena> tour;
  int *first = nullptr, *euler = nullptr;
  // until the labels are built: hld lists the heavy paths one after another,
  // top to bottom (hpos[v] = v's index, htop[v] = the top of v's path); node
  // v's root path is the segments seg_off[v] .. seg_off[v+1]-1, shallowest
  // first, one per heavy path it crosses (written by FillPlan)
  std::shared_ptr<DeviceArena> layout;
  int *hld = nullptr, *htop = nullptr, *hpos = nullptr;
  int64_t *seg_off = nullptr;
};

// Device-resident index used by the label fill and the query kernels.
// Label rows are padded so every row starts on a 16-byte boundary
// (drow[v] is a multiple of 4 ints); the reference layout is restored on
// export.  Pointers in `owned` belong to the handle.  A graph labelled in a
// batch points into the batch's forest arrays instead (`keep` holds them):
// depth, pos_hash, drow and father are then offset to the graph's first
// vertex, while drow and pos_hash values stay absolute offsets into the
// shared dis and pos_pos / pos_id arrays.
struct DeviceIndex {
  int n = 0;
  int64_t euler = 0, rmq = 0, pos = 0, dis_padded = 0;
  bool rmq_closed = true;     // RMQHash is the closed form of build_rmq_gpu
  int *first = nullptr;       // firstAppeare           [n]
  int *depth = nullptr;       // H2H_TreeHeight_Hash    [n]
  int64_t *rmq_hash = nullptr;// RMQHash                [euler]
  int *rmq_id = nullptr;      // RMQ_ID                 [rmq]
  int64_t *pos_hash = nullptr;// H2H_pos_hash           [n+1]
  int *pos_pos = nullptr;     // H2H_pos_POS            [pos]
  int *pos_id = nullptr;      // H2H_pos_ID             [pos]
  int64_t *drow = nullptr;    // padded row offsets     [n+1]
  int *dis = nullptr;         // padded labels          [dis_padded]
  int *father = nullptr;      // father                 [n]
  int *err = nullptr;         // kernel error word      [1]
  // views into the contraction's device lists and the fill's position
  // arrays: the graph's entries start at x_base / pos_base, its vertex ids
  // at id_base (non-zero in a batch)
  ListStore lists;
  int64_t x_base = 0, pos_base = 0;
  int id_base = 0;
  int64_t bytes = 0, rmq_bytes = 0;
  std::vector<void *> owned;      // label-side allocations of this handle
  std::shared_ptr<DeviceArena> owned_rmq;  // first, rmq_hash, rmq_id (built with the trees)
  std::shared_ptr<void> keep;
  void release();
  void release_labels();  // everything but the sparse table
};

struct Timings {
  long long load = 0, rank_tree = 0, lub = 0, translate_lub = 0, td_gpu = 0, translate_back = 0, td_cpu = 0,
            tree = 0, malloc_labels = 0, bfs = 0, translate_labels = 0, fill_gpu = 0;
};

struct Graph : HostInput {
  // configuration (the G2H command line, main.cu:252-260)
  std::string name;
  int H_cli = 0, H = 0, C = 0, threads = 1, method = 1;
  int contract_device = 1, parallel_fine = 2, construct_device = 1, label_mode = H2H_LABEL_L4;
  // input (Graph_Fundamental.cu:4-95): on the device, in HostInput's arrays,
  // or both (input_device / input_host)
  int n = 0;
  int64_t m = 0;
  std::shared_ptr<DeviceInput> input;
  mutable std::mutex host_lock;
  std::vector<int> cut_l, cut_r;   // partition_Tree rows [2^H-1]
  // elimination sets (GraphPartition.cu:178-308)
  std::vector<int> cell_start, cell_count;  // NANHash first / NodeID per cell
  std::vector<int> elim;                    // elimination order (host_tree)
  std::vector<int> cell_bound;              // per partition cell: bound on a list while its level runs
  std::shared_ptr<SetsStore> sets;          // until the graph is contracted
  int64_t lub = 0;
  std::vector<double> layer_rate;           // afs[h] / n for the PartitionRate CSV
  // contraction results: on the device (tree, dev.lists); the host arrays
  // below are filled by host_tree, the lists by download_lists
  std::shared_ptr<TreeStore> tree;
  std::vector<int64_t> x_off;               // X(v)\{v}: upper neighbours, CSR by vertex [n+1]
  std::vector<int> x_id, x_w;               //   sorted by id, shortcut weights
  int gpu_vertices = 0;                     // vertexesConstructedInGPU
  int64_t x_total = 0;                      // entries of the lists
  int64_t decomposition_size = 0;           // size1 = sum(|X(v)|+1)
  bool contracted = false;
  // tree (TreeStructure.cu)
  int head = -1, tree_height = 0, n_levels = 0;
  std::vector<int> father, depth, first;
  int64_t euler_n = 0, h2h_size = 0, rmq_total = 0;  // rmq_total: RMQ_ID entries (the table is on the GPU)
  // labels (H2HConsturction.cu), reference layout on the host
  std::vector<int64_t> dis_hash, pos_hash;
  int64_t pos_n = 0;                        // entries of the position lists, once the labels are laid out
  int64_t updates = 0;                      // min-plus updates of the fill
  // host position lists: built for L3 labels only (L4 builds them on the GPU;
  // accessors download them)
  std::vector<int> pos_id, pos_pos, pos_w;  // pos_w: shortcut weight per pos entry (0 for v itself)
  std::vector<int64_t> drow_host;           // padded device row offsets (absolute in a batch's forest)
  int64_t row0 = 0, row1 = 0;               // the first and the end
  std::vector<int> tree_bfs, tree_hash;     // TreeBFS / TreeHash
  bool labelled = false;
  int64_t max_label = 0;  // -1: not computed yet (label_max computes it)
  // device
  DeviceIndex dev;
  std::shared_ptr<struct FillPlan> plan;  // blocks and weights made by the contraction, until the labels are built
  Timings t;

  // After a contraction or a batch that failed on the way: what it had made is
  // freed, and the graph is as it was loaded.
  void drop_build();
  ~Graph() { dev.release(); }
};

// The label arrays of graphs filled together.
struct LabelStore {
  DeviceArena mem;
  std::shared_ptr<TreeStore> tree;
};

// Where a graph's global order starts: the vertices of the cells at levels
// C..1 (the tail of elim).
struct GraphLevels {
  int heap_start = 0, heap_n = 0;
};

// Vertex elimination over one or more graphs in one set of launches
// (symbolic.cu; contract.cu where the cells are too large for bit rows).  The graphs' vertices are numbered consecutively (graph i
// starts at vbase[i]); launch s eliminates the cells of level H_i - s of
// every graph i with H_i - s > C_i, and one last launch runs every graph's
// global order (levels <= C_i) as one cell per graph.  The list structure
// and the elimination order depend only on the topology, so enqueue() can be
// replayed (or captured in a CUDA graph) after set_weights().
struct ElimPlan {
  struct Launch {
    int step, level, ncell, kmax, lmax, cs, nw, slots;
    int arena = 0;               // cooperative launches: ints of shared-memory arena per block
    bool arena_merges = false;   // ... that merges take their buffers from
    int64_t lo, smem, pstage_off;
    bool heap, global_stage;
    // cell_grid_kernel: the step's cells in one cooperative launch, `slots`
    // blocks (block -> cell map at grid_map + map_off, cell -> first block
    // after it), one barrier counter per cell at grid_bar + bar_off, at most
    // slice_max candidates owned by one block
    bool grid;
    int slice_max;
    int64_t map_off, bar_off;
  };
  // A launch of symbolic_kernel: cells lo .. lo + ncell of sym_cells, clusters
  // of cs CTAs with nw warps, rows of up to smax members
  struct SymLaunch {
    int step, level, ncell, kmax, smax, npow, cs, nw;
    bool heap, global, grid;  // grid: cs CTAs per cell in one cooperative launch
    int64_t lo, smem, rows_off, best_off;
    int arrived_off;
  };
  // What the list kernels' launches need on the device
  struct ListLaunches {
    std::vector<int> fcs, fcc, gmap;  // cell starts and counts, block maps
    int64_t pstage_ints = 0, partial_max = 0;
  };
  std::vector<Graph *> gs;
  std::vector<int> vbase;
  std::vector<int64_t> mbase;
  // the order and the lists' ids come from bit rows, the weights from
  // FillPlan::enqueue_weights; otherwise the list kernels make all three
  bool bits = false;
  std::vector<SymLaunch> sym;
  int *members = nullptr, *extra = nullptr;
  unsigned char *sym_cells = nullptr;
  // the lists on bit rows, level after level; from 8 MiB an allocation of its
  // own, freed once they are compacted
  int *pool = nullptr;
  bool own_pool = false;
  unsigned *grows = nullptr, *sym_arrived = nullptr;
  unsigned long long *sym_best = nullptr;
  int grid_cells = 0;
  int N = 0, heap_total = 0;
  int64_t M = 0, lub = 0, slots_size = 0, pool_size = 0;
  std::vector<Launch> launches;  // in step order; launches of one step are independent
  int nsm = 0, max_group = 1;
  bool elim_balance = true;  // cooperative steps: merges split over a cell's blocks by work
  int64_t partial_cap = 0;   // blocks the per-block arrays of cooperative launches hold
  std::vector<cudaStream_t> side;  // streams for the second and later launches of a step
  std::vector<cudaEvent_t> ev_join;
  cudaEvent_t ev_fork = nullptr;
  // device state (global vertex ids)
  int *slot_nbr = nullptr, *slot_w = nullptr, *lsize = nullptr, *cap = nullptr, *cap_init = nullptr;
  int *height = nullptr, *elim = nullptr;
  int *deg0 = nullptr, *h0 = nullptr, *cpos = nullptr, *err = nullptr, *ljunk = nullptr, *cell_start = nullptr;
  int *cell_count = nullptr, *adj_off = nullptr, *adj_v = nullptr, *adj_w = nullptr, *pstage = nullptr;
  int *deg_init = nullptr, *elim_init = nullptr, *heap_verts = nullptr;
  int64_t *slot_off = nullptr, *slot_off_init = nullptr;
  unsigned long long *pool_next = nullptr, *pool_first = nullptr;
  ListStore lists;       // compact final lists (forest numbering), after build_lists()
  int *rank = nullptr;
  // cell_grid_kernel state: per-block argmins, block maps, barrier counters
  int *grid_map = nullptr;
  void *hg_partial = nullptr;
  unsigned *grid_bar = nullptr;
  int64_t grid_bar_words = 0;
  DeviceArena mem;          // every array but the pool
  int64_t slot_bytes = 0;
  int64_t bytes() const { return mem.bytes + slot_bytes; }
  explicit ElimPlan(const std::vector<Graph *> &graphs, bool allow_bits = true);
  ~ElimPlan();
  bool plan_bits();
  void plan_lists(const int *f_elim, const std::vector<GraphLevels> &L, ListLaunches &LL);
  void enqueue_bits(cudaStream_t s, cudaEvent_t *heap_ev, bool trace);
  void gather_bits(cudaStream_t s);
  bool grow_pool();
  void free_pool();
  int launch_count() const { return (int)(bits ? sym.size() : launches.size()); }
  void release();
  ElimPlan(const ElimPlan &) = delete;
  ElimPlan &operator=(const ElimPlan &) = delete;
  // Resets the lists from the input arcs and runs every launch on s.  With
  // heap_ev non-null, records heap_ev[0] before the global-order launch and
  // heap_ev[1] after it.
  void enqueue(cudaStream_t s, cudaEvent_t *heap_ev = nullptr, bool trace = false);
  void launch_one(const Launch &Lc, cudaStream_t s, bool trace);
  // The first enqueue, waited for; again with a larger pool where the lists
  // outgrew it.  False: they take more than the list kernels would.
  bool run(cudaStream_t s, cudaEvent_t *heap_ev, bool trace);
  int read_error();    // synchronises
  void check_error();  // synchronises; throws on a kernel error code
  // After the first enqueue: compact the final lists and pick each vertex's
  // father (min elimination rank over its list), all on the device; every
  // graph gets the lists and the tree they start.
  void build_lists();
  // Refreshes the compact lists' entries from the slot arrays (replays).
  void enqueue_gather(cudaStream_t s);
  void set_weights(int gi, const int *w, cudaStream_t s);  // arc weights in the graph's file order
};

// Task shapes of the L4 fill, keyed on a block's top: its tree level --
// class 0: fewer nodes than SMs (the chain-like top, on the critical path);
// class 1: wider; class 2: wider and heavy (its nodes average at least 2^18
// min-plus updates m*d) -- and its separator size m (buckets m <= 16, <= 64,
// <= 256, > 256).  A block whose m * d is at most small_work is one task; a
// larger one is cut into tasks of col_block columns (rounded up to 64).
// sep_chunk belongs to the text form and shapes nothing.
struct TilePolicy {
  static constexpr int kWidth = 3, kSep = 4;
  int small_work[kWidth][kSep], col_block[kWidth][kSep], sep_chunk[kWidth][kSep];
  TilePolicy();
  static int sep_bucket(int m) { return m <= 16 ? 0 : m <= 64 ? 1 : m <= 256 ? 2 : 3; }
  std::string str() const;
  bool parse(const std::string &s);
};

// The L4 label fill over one or more graphs as one forest (labels.cu): the
// graphs' trees are laid side by side (graph i's vertex v is forest vertex
// vbase[i] + v) and filled by one launch.  Each graph's DeviceIndex
// becomes a view into the forest arrays.
struct FillPlan {
  std::vector<Graph *> gs;
  std::vector<int> vbase;
  int N = 0;
  int64_t pos_total = 0, dis_total = 0;
  TilePolicy policy;
  std::shared_ptr<struct LabelStore> storage;  // forest arrays shared with the graphs' views
  int64_t *drow = nullptr, *pos_hash = nullptr;
  int *pos_pos = nullptr, *pos_id = nullptr, *pos_w = nullptr, *pos_src = nullptr, *father = nullptr;
  ListStore lists;
  int *depth = nullptr, *dis = nullptr;
  // workspace
  int *hld = nullptr, *htop = nullptr, *hpos = nullptr, *seg_top = nullptr, *seg_pos = nullptr;
  int64_t *hld_row = nullptr;
  int64_t *seg_off = nullptr;
  int *done = nullptr, *next = nullptr, *tasks = nullptr;  // tasks: task -> block
  // error words of the fill and of the weights, side by side: a rebuild runs
  // both and then looks once, so neither clears the other's
  int *err = nullptr, *werr = nullptr;
  // the blocks (fill_blocks.cu): top, separator size, first node / member /
  // cell of the weight tables per block; node lists and places; members'
  // positions and row offsets; direct and closed weights; first task and
  // columns per task
  int nblk = 0, nlev = 0;
  int *blk_top = nullptr, *blk_mem = nullptr, *bnode = nullptr, *blk_of = nullptr, *lvl_cls = nullptr, *bm_p = nullptr,
      *tcols = nullptr;
  int64_t *blk_boff = nullptr, *blk_moff = nullptr, *blk_soff = nullptr, *bm_row = nullptr, *task0 = nullptr;
  unsigned char *loc_of = nullptr;
  unsigned *direct = nullptr, *closed = nullptr, *blk_anc = nullptr;
  int64_t cell_total = 0;
  // weights from arcs: parent block and the members' places in it, update
  // triangles, task tables, arrivals a block waits for, each arc's cell
  const ElimPlan *arcs = nullptr;
  bool weights_fit = true;  // false: no room for the update triangles
  int *blk_up = nullptr, *bm_up = nullptr, *wtask_blk = nullptr, *pending = nullptr, *pend_init = nullptr;
  int64_t *blk_uoff = nullptr, *wtask0 = nullptr, *arc_cell = nullptr;
  unsigned *upd = nullptr;
  int64_t wtasks = 0, upd_total = 0;
  unsigned long long *trace_t = nullptr;  // publish time per node (GPUH2H_TRACE)
  int *mslot = nullptr;  // blocks of several tasks: their in-block matrix
  unsigned *mbuf = nullptr;
  int64_t mslots = 0, mslots_cap = 0;
  int64_t ntasks = 0, tasks_cap = 0;
  int64_t ntiles = 0;  // row pieces: every node of a block once per task of the block
  int max_segs = 1, blocks = 1;
  size_t smem = 0;
  int nsm = 0;
  DeviceArena work;       // the plan's arrays but tasks and mbuf, which grow with the policy
  DeviceArena weights_mem;  // those that only enqueue_weights reads, where they are large
  std::shared_ptr<DeviceArena> layout;  // the tree's heavy paths and segment offsets
  int64_t grown_bytes = 0;
  int64_t work_bytes() const { return work.bytes + weights_mem.bytes + (layout ? layout->bytes : 0) + grown_bytes; }
  // The blocks and, when `arcs` made the order on bit rows, where each of its
  // arcs enters the blocks' weights.  lists: the graphs' X lists in the same
  // forest numbering.  keep: the weights are made again after the labels (rebuilds).
  FillPlan(const std::vector<Graph *> &graphs, const ListStore &lists, const ElimPlan *arcs, bool keep);
  ~FillPlan();
  void release_work();
  FillPlan(const FillPlan &) = delete;
  FillPlan &operator=(const FillPlan &) = delete;
  void build_blocks();
  void build_weights_plan(const ElimPlan &arcs, bool keep);
  void drop_weights();  // after the weights of a plan that makes them once
  void prepare(const TilePolicy &pol);  // label rows and tasks
  void build_tiles(const TilePolicy &pol);
  std::vector<int> level_classes() const;  // TilePolicy class per forest level
  // The shortcut weights of every list and block on s: eliminated block by
  // block from the arcs' current weights, or gathered from the lists.
  void enqueue_weights(cudaStream_t s);
  // Resets the flags and runs the fill on s.
  void enqueue(cudaStream_t s, cudaEvent_t *fill_ev = nullptr);
  void check_error();            // synchronises; throws if a wait of the weights or of the fill ran out
  void trace_report();           // GPUH2H_TRACE: the last fill's time per level class
  void attach(bool first);       // per-graph views; first: of new arrays
};

// Phases (one translation unit each).
bool load_input_gpu(Graph &g, const char *ids, int64_t ids_size, const char *arcs, int64_t arcs_size,
                    int64_t m);                        // input_gpu.cu
const DeviceInput &input_device(Graph &g);             // input_gpu.cu
const HostInput &input_host(const Graph &g);           // input_gpu.cu
void load_graph(Graph &g, const std::string &edge, const std::string &idf, const std::string &cut);
// elim_sets.cu: elimination sets, LUB capacities and layout, cell list
// bounds and parallel-arc counts of one or more graphs, on the GPU
void build_elimination_sets(const std::vector<Graph *> &gs);
// contract.cu: partition levels H..C+1 and the global heap over levels <= C;
// (then the tree, sparse table and weights of one graph)
void contract_gpu(Graph &g);
// tree_gpu.cu: the tree of every graph contracted together (children, tour,
// depths, heavy paths, offsets) from the fathers, on the GPU
void build_tree_gpu(const std::vector<Graph *> &gs);
const Graph &host_tree(const Graph &g);                // tree_gpu.cu: fills the host arrays of the tree
void download_tree(const Graph &g, int *order, int *father, int *depth, int *first, int64_t *x_off);  // tree_gpu.cu
// query.cu: the compacted sparse tables of the graphs' Euler tours on the
// GPU (first, rmq_hash, rmq_id in each graph's DeviceIndex)
void build_rmq_gpu(const std::vector<Graph *> &gs);
void download_rmq(const Graph &g, int64_t *rmq_hash, int *rmq_id);  // query.cu
void allocate_labels_and_bfs(Graph &g);                // tree.cpp
void fill_labels_gpu(Graph &g);                        // labels.cu
// The level-synchronous fill (L3 labels, or L4 with GPUH2H_LEVEL_FILL set)
// runs from host position lists; the L4 block fill builds them on the GPU.
inline bool uses_level_fill(const Graph &g) {
  return g.label_mode == H2H_LABEL_L3 || std::getenv("GPUH2H_LEVEL_FILL") != nullptr;
}
void download_labels(const Graph &g, int *dis_out);    // labels.cu, reference layout
int64_t label_max(const Graph &g);                     // labels.cu: largest finite label, computed once
// labels.cu: the reference's level-by-level GPU fill mapping on a built L4
// graph (measurement baseline): device ms and mismatches against the labels
void fill_labels_plain(const Graph &g, int mapping, double *ms, int64_t *mismatches);
// labels.cu: the graph's position lists (reference layout, graph-local ids)
void download_positions(const Graph &g, int *pos_id, int *pos_pos);
// contract.cu: host copies of the X lists (graph-local ids) from the device
void download_lists(Graph &g);
// Device copies of a saved index (index_io.cpp loads the file):
ListStore upload_lists(const std::vector<int64_t> &off, const std::vector<int> &id,
                       const std::vector<int> &w);                         // contract.cu
void upload_rmq(Graph &g, const std::vector<int64_t> &rmq_hash, const std::vector<int> &rmq_id);  // query.cu
// labels.cu: rows (reference layout, dis_hash offsets) into padded device
// rows plus the position arrays; sets drow_host and the DeviceIndex
void upload_labels(Graph &g, const std::vector<int> &dis, const std::vector<int> &pos_id,
                   const std::vector<int> &pos_pos);
void upload_query_index(Graph &g);                     // query.cu
// query.cu; bad: the flag word set when a pair holds an id out of range
// (nullptr: the graph's own)
void run_query_batch(const Graph &g, const int *x, const int *y, int *out, int64_t n, int mode, cudaStream_t s,
                     int *bad = nullptr);
void run_query_batch_plain(const Graph &g, const int *x, const int *y, int *out, int64_t n, int mode,
                           cudaStream_t s);                  // query.cu, one thread per query

}  // namespace gh
