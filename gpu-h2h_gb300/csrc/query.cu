// query.cu -- batched H2H distance queries on the device-resident index, the
// work of H2HQuery_UsingLCA_D_noHub / H2HQuery_noLCA_D_noHub
// (kernel_functions.cu:1143-1296) and of the host single-pair queries
// (Query.cu:108-151).
//
// LCA by range minimum over the Euler tour: l, r = sorted firstAppeare,
// k = floor(log2(r - l + 1)) (31 - clz, the integer equal of the reference's
// (int)log2((double)...)), two sparse-table ids, the shallower wins.  Then:
//   LCA mode:   min over p in pos(LCA) of dis[x][p] + dis[y][p]
//   noLCA mode: min over j < depth(LCA) of dis[x][j] + dis[y][j]
// x == y answers 0 as in the reference.
#include <algorithm>
#include <climits>

#include "graph.h"

namespace gh {

namespace {

struct QArgs {
  const int *x, *y;
  int *out;
  int64_t n;
  int nv;  // vertices; ids outside [0, nv) answer -1 without touching the index
  const int *first, *depth;
  const int64_t *rmq_hash;
  const int *rmq_id;
  const int64_t *pos_hash;
  const int *pos_pos;
  const int64_t *drow;
  const int *dis;
  int *bad;  // set to 1 when a pair holds an id outside [0, nv)
  int64_t tiles;             // ceil(n / TILE)
  int64_t euler, rmq_total;  // tour and table lengths; euler 0: row starts are read from rmq_hash
};

// G lanes cooperate on one query.  Every lane of the group resolves the LCA
// (same addresses, one transaction per load), then the lanes split the min.
template <int G, bool LCA_MODE>
__global__ void query_kernel(QArgs A) {
  const int lane = threadIdx.x & (G - 1);
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
  const int64_t groups = ((int64_t)gridDim.x * blockDim.x) / G;
  for (int64_t q = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G; q < A.n; q += groups) {
    const int a = __ldg(A.x + q), b = __ldg(A.y + q);
    const bool valid = (unsigned)a < (unsigned)A.nv && (unsigned)b < (unsigned)A.nv;
    int res = !valid ? -1 : (a == b ? 0 : INT_MAX);
    if (!valid && lane == 0) atomicExch(A.bad, 1);
    if (valid && a != b) {
      const int fa = __ldg(A.first + a), fb = __ldg(A.first + b);
      const int l = min(fa, fb), r = max(fa, fb);
      const int k = 31 - __clz(r - l + 1);
      const int i1 = __ldg(A.rmq_id + __ldg(A.rmq_hash + l) + k);
      const int i2 = __ldg(A.rmq_id + __ldg(A.rmq_hash + r - (1 << k) + 1) + k);
      const int d1 = __ldg(A.depth + i1), d2 = __ldg(A.depth + i2);
      const int *rx = A.dis + __ldg(A.drow + a);
      const int *ry = A.dis + __ldg(A.drow + b);
      if (LCA_MODE) {
        const int lca = d1 <= d2 ? i1 : i2;
        const int64_t pb = __ldg(A.pos_hash + lca), pe = __ldg(A.pos_hash + lca + 1);
        for (int64_t t = pb + lane; t < pe; t += G) {
          const int p = __ldg(A.pos_pos + t);
          res = min(res, __ldg(rx + p) + __ldg(ry + p));
        }
      } else {
        const int dl = min(d1, d2);
        for (int j = lane; j < dl; j += G) res = min(res, __ldg(rx + j) + __ldg(ry + j));
      }
    }
    if (G > 1) {
      for (int o = G >> 1; o > 0; o >>= 1) res = min(res, __shfl_down_sync(gmask, res, o, G));
    }
    if (lane == 0) A.out[q] = res;
  }
}

// Start of row i of the sparse table (see build_rmq_gpu): S(L) - S(L - i).
__host__ __device__ inline int64_t rmq_prefix(int64_t x) {
  if (x <= 0) return 0;
#ifdef __CUDA_ARCH__
  const int k = 63 - __clzll(x);
#else
  int k = 0;
  while ((int64_t(2) << k) <= x) k++;
#endif
  return ((int64_t)(k - 1) << k) + 1 + (x - (int64_t(1) << k) + 1) * (k + 1);
}

__device__ __forceinline__ int64_t rmq_row(const QArgs &A, int i) {
  return A.euler > 0 ? A.rmq_total - rmq_prefix(A.euler - i) : __ldg(A.rmq_hash + i);
}

// A warp owns TILE queries.  Phase 1: lane i < TILE resolves query i (ids, row
// bases, LCA through the sparse table) -- TILE chains of dependent loads in
// flight.  The table's row starts are computed and the position ranges of both
// LCA candidates fetched with their depths, so a chain is five loads long, not
// seven.  Phase 2: the warp walks the queries one after another in pieces of
// 128 entries; while the label entries of a piece are on their way it loads
// the positions (noLCA mode: the entries) of the next one, this query's or
// the next query's, so only one load's latency is left per piece.  The answers
// leave in one store.
//
// Bound: HBM on large batches, the chain of dependent loads on small ones.  On
// one GB300, against loading positions and entries of one query in turn: 2e6
// pairs on a 264k-vertex road graph 812 -> 692 us (0.91 of HBM), 1e5 pairs 72
// -> 61 us, 1e5 pairs in noLCA mode on a 70k-vertex graph 66 -> 45 us, 1e3
// pairs 8 us either way.  Spreading a warp over several queries (8 lanes each)
// took 2,200 us: a row is then read in 128-byte pieces at different times,
// which DRAM serves at a third of its rate.
template <bool LCA_MODE, int TILE>
__global__ void __launch_bounds__(256, 6) query_tile_kernel(QArgs A) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t tile = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; tile < A.tiles; tile += nwarps) {
    // narrow tiles (one wave) take half their queries from each half of the
    // batch: a run of near or far pairs spreads over more warps, and fewer get
    // only long walks
    constexpr int RUN = TILE < 32 && TILE > 1 ? TILE / 2 : TILE;
    const int64_t q = (lane / RUN * A.tiles + tile) * RUN + lane % RUN;
    int res = INT_MAX, len = 0;
    int64_t pb = 0, bx = 0, by = 0;
    if (lane < TILE && q < A.n) {
      const int a = __ldg(A.x + q), b = __ldg(A.y + q);
      const bool valid = (unsigned)a < (unsigned)A.nv && (unsigned)b < (unsigned)A.nv;
      if (!valid) {
        res = -1;
        *(volatile int *)A.bad = 1;
      } else if (a == b) {
        res = 0;
      } else {
        const int fa = __ldg(A.first + a), fb = __ldg(A.first + b);
        bx = __ldg(A.drow + a);
        by = __ldg(A.drow + b);
        const int l = min(fa, fb), r = max(fa, fb);
        const int k = 31 - __clz(r - l + 1);
        const int i1 = __ldg(A.rmq_id + rmq_row(A, l) + k);
        const int i2 = __ldg(A.rmq_id + rmq_row(A, r - (1 << k) + 1) + k);
        const int d1 = __ldg(A.depth + i1), d2 = __ldg(A.depth + i2);
        if (LCA_MODE) {
          const int64_t b1 = __ldg(A.pos_hash + i1), e1 = __ldg(A.pos_hash + i1 + 1);
          const int64_t b2 = __ldg(A.pos_hash + i2), e2 = __ldg(A.pos_hash + i2 + 1);
          pb = d1 <= d2 ? b1 : b2;
          len = (int)(d1 <= d2 ? e1 - b1 : e2 - b2);
        } else {
          len = min(d1, d2);
        }
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, len > 0);
    if (LCA_MODE) {
      if (todo) {
        int s = __ffs(todo) - 1, t0 = 0;
        int L = __shfl_sync(0xffffffffu, len, s);
        int64_t PB = __shfl_sync(0xffffffffu, pb, s);
        int p[U];
#pragma unroll
        for (int u = 0; u < U; u++) p[u] = 32 * u + lane < L ? __ldg(A.pos_pos + PB + 32 * u + lane) : -1;
        const int *rx = A.dis + __shfl_sync(0xffffffffu, bx, s), *ry = A.dis + __shfl_sync(0xffffffffu, by, s);
        int m = INT_MAX;
        for (;;) {
          int xv[U], yv[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            xv[u] = p[u] >= 0 ? __ldg(rx + p[u]) : 0;
            yv[u] = p[u] >= 0 ? __ldg(ry + p[u]) : 0;
          }
          // the positions of the next piece: this query's next 128, or the next query's first
          const int cur = s;
          const bool last = t0 + 32 * U >= L;
          int next[U];
          if (last) {
            todo &= todo - 1;
            s = todo ? __ffs(todo) - 1 : s;
            t0 = 0;
            L = todo ? __shfl_sync(0xffffffffu, len, s) : 0;
            PB = __shfl_sync(0xffffffffu, pb, s);
          } else {
            t0 += 32 * U;
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int t = t0 + 32 * u + lane;
            next[u] = t < L ? __ldg(A.pos_pos + PB + t) : -1;
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            if (p[u] >= 0) m = min(m, xv[u] + yv[u]);
            p[u] = next[u];
          }
          if (last) {
            m = __reduce_min_sync(0xffffffffu, m);
            if (lane == cur) res = m;
            if (!todo) break;
            m = INT_MAX;
            rx = A.dis + __shfl_sync(0xffffffffu, bx, s);
            ry = A.dis + __shfl_sync(0xffffffffu, by, s);
          }
        }
      }
    } else if (todo) {
      // pieces of 128 entries, four per lane (rows start on 16 bytes and are
      // padded to them); the next piece, this query's or the next one's, is
      // loaded before this one is used
      int s = __ffs(todo) - 1, t0 = 0;
      int L = __shfl_sync(0xffffffffu, len, s);
      const int *rx = A.dis + __shfl_sync(0xffffffffu, bx, s), *ry = A.dis + __shfl_sync(0xffffffffu, by, s);
      const int4 none = make_int4(0, 0, 0, 0);
      int4 xv = 4 * lane < L ? __ldg(reinterpret_cast<const int4 *>(rx) + lane) : none;
      int4 yv = 4 * lane < L ? __ldg(reinterpret_cast<const int4 *>(ry) + lane) : none;
      int m = INT_MAX;
      for (;;) {
        const int cur = s, left = L - t0 - 4 * lane;  // entries of this lane's four that count
        const bool last = t0 + 128 >= L;
        if (last) {
          todo &= todo - 1;
          s = todo ? __ffs(todo) - 1 : s;
          t0 = 0;
          L = todo ? __shfl_sync(0xffffffffu, len, s) : 0;
          rx = A.dis + __shfl_sync(0xffffffffu, bx, s);
          ry = A.dis + __shfl_sync(0xffffffffu, by, s);
        } else {
          t0 += 128;
        }
        const int j = t0 + 4 * lane;
        const int4 xn = j < L ? __ldg(reinterpret_cast<const int4 *>(rx + j)) : none;
        const int4 yn = j < L ? __ldg(reinterpret_cast<const int4 *>(ry + j)) : none;
        if (left > 0) m = min(m, xv.x + yv.x);
        if (left > 1) m = min(m, xv.y + yv.y);
        if (left > 2) m = min(m, xv.z + yv.z);
        if (left > 3) m = min(m, xv.w + yv.w);
        xv = xn;
        yv = yn;
        if (last) {
          m = __reduce_min_sync(0xffffffffu, m);
          if (lane == cur) res = m;
          if (!todo) break;
          m = INT_MAX;
        }
      }
    }
    if (lane < TILE && q < A.n) A.out[q] = res;
  }
}

}  // namespace

// ---- compacted sparse table of the Euler tour (makeOULAAndRMQ,
// TreeStructure.cu:500-572), built on the GPU.  Row i of the table holds the
// shallowest-node ids of the windows [i, i + 2^j) for every j with
// i + 2^j - 1 < L, so it has floor(log2(L - i)) + 1 entries and starts at
//   RMQHash[i] = S(L) - S(L - i),  S(x) = sum_{t=1..x} (floor(log2 t) + 1)
//              = (k - 1) 2^k + 1 + (x - 2^k + 1)(k + 1),  k = floor(log2 x).
// Level j combines two level-(j-1) windows, the left one winning ties
// (depth <=, TreeStructure.cu:528); one launch per level covers the Euler
// tours of every graph given.
namespace {

struct RmqJob {
  const int *eid;    // Euler tour, vertex per position
  const int *depth;  // depth per vertex
  int64_t *hash;     // RMQHash [L]
  int *id;           // RMQ_ID  [S(L)]
  int64_t L;
};

__device__ __forceinline__ int job_of(const int64_t *off, int njobs, int64_t p) {
  int lo = 0, hi = njobs - 1;  // last job with off[job] <= p
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void rmq_hash_kernel(const RmqJob *jobs, const int64_t *off, int njobs, int64_t total) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
    const int g = job_of(off, njobs, p);
    const int64_t i = p - off[g], L = jobs[g].L;
    jobs[g].hash[i] = rmq_prefix(L) - rmq_prefix(L - i);
  }
}

__global__ void rmq_level_kernel(const RmqJob *jobs, const int64_t *off, int njobs, int64_t total, int j) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
    const int g = job_of(off, njobs, p);
    const RmqJob J = jobs[g];
    const int64_t i = p - off[g];
    if (j == 0) {
      J.id[J.hash[i]] = J.eid[i];
    } else if (i + (int64_t(1) << j) - 1 < J.L) {
      const int a = J.id[J.hash[i] + j - 1];
      const int c = J.id[J.hash[i + (int64_t(1) << (j - 1))] + j - 1];
      J.id[J.hash[i] + j] = __ldg(J.depth + a) <= __ldg(J.depth + c) ? a : c;
    }
  }
}

// firstAppeare, RMQHash and RMQ_ID on the device, in an arena of their own or
// of the graphs built together (a batch of sixteen spent 1 ms on theirs).
void allocate_rmq(Graph &g, const std::shared_ptr<DeviceArena> &mem) {
  DeviceIndex &D = g.dev;
  D.bytes -= D.rmq_bytes;
  D.owned_rmq = mem;
  D.euler = g.euler_n;
  D.rmq = g.rmq_total;
  D.first = mem->get<int>(g.n);
  D.rmq_hash = mem->get<int64_t>(D.euler);
  D.rmq_id = mem->get<int>(D.rmq);
  D.rmq_bytes = 4 * (int64_t)g.n + 8 * D.euler + 4 * D.rmq;
  D.bytes += D.rmq_bytes;
}

}  // namespace

void build_rmq_gpu(const std::vector<Graph *> &gs) {
  Clock clk;
  const int K = (int)gs.size();
  const std::shared_ptr<TreeStore> tree = gs[0]->tree;
  GH_CHECK(tree && tree->gs == gs && tree->euler, H2H_ERR_STATE, "Euler tour missing");
  std::vector<int64_t> off(K + 1, 0);
  int levels = 0;
  for (int i = 0; i < K; i++) {
    off[i + 1] = off[i] + gs[i]->euler_n;
    levels = std::max(levels, ilog2_floor(gs[i]->euler_n));
  }
  const int64_t total = off[K];
  DeviceArena ws;
  {
    int64_t *d_off = ws.get<int64_t>(K + 1);
    RmqJob *d_jobs = ws.get<RmqJob>(K);
    std::vector<RmqJob> jobs(K);
    auto mem = std::make_shared<DeviceArena>();
    size_t bytes = 0;
    for (const Graph *g : gs)
      bytes += 4 * (size_t)g->n + 8 * (size_t)g->euler_n + 4 * (size_t)rmq_prefix(g->euler_n) + 3 * 256;
    mem->reserve(bytes);
    for (int i = 0; i < K; i++) {
      Graph &g = *gs[i];
      DeviceIndex &D = g.dev;
      const int vb = tree->vbase[i];
      g.rmq_total = rmq_prefix(g.euler_n);
      allocate_rmq(g, mem);
      GH_CUDA(cudaMemcpyAsync(D.first, tree->first + vb, sizeof(int) * g.n, cudaMemcpyDeviceToDevice));
      jobs[i] = RmqJob{tree->euler + off[i], tree->depth + vb, D.rmq_hash, D.rmq_id, g.euler_n};
    }
    GH_CUDA(cudaMemcpy(d_jobs, jobs.data(), sizeof(RmqJob) * K, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(d_off, off.data(), sizeof(int64_t) * (K + 1), cudaMemcpyHostToDevice));
    int dev = 0, nsm = 0;
    GH_CUDA(cudaGetDevice(&dev));
    GH_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)nsm * 8, (total + 255) / 256));
    rmq_hash_kernel<<<blocks, 256>>>(d_jobs, d_off, K, total);
    GH_CUDA(cudaGetLastError());
    for (int j = 0; j <= levels; j++) {
      rmq_level_kernel<<<blocks, 256>>>(d_jobs, d_off, K, total, j);
      GH_CUDA(cudaGetLastError());
    }
    GH_CUDA(cudaDeviceSynchronize());
  }
  ws.release();
  tree->tour.reset();
  tree->first = tree->euler = nullptr;
  const long long us = clk.us();
  for (Graph *g : gs) g->t.tree += us / K;
}

void upload_rmq(Graph &g, const std::vector<int64_t> &rmq_hash, const std::vector<int> &rmq_id) {
  // a file's row starts are usually the closed form's; otherwise the queries read them
  const int64_t total = rmq_prefix(g.euler_n);
  bool closed = total == g.rmq_total;
  for (int64_t i = 0, start = 0; i < g.euler_n && closed; i++) {
    closed = rmq_hash[i] == start;
    start += 64 - __builtin_clzll((unsigned long long)(g.euler_n - i));
  }
  allocate_rmq(g, std::make_shared<DeviceArena>());
  DeviceIndex &D = g.dev;
  D.rmq_closed = closed;
  GH_CUDA(cudaMemcpy(D.first, g.first.data(), sizeof(int) * g.n, cudaMemcpyHostToDevice));
  GH_CUDA(cudaMemcpy(D.rmq_hash, rmq_hash.data(), sizeof(int64_t) * D.euler, cudaMemcpyHostToDevice));
  GH_CUDA(cudaMemcpy(D.rmq_id, rmq_id.data(), sizeof(int) * D.rmq, cudaMemcpyHostToDevice));
}

void download_rmq(const Graph &g, int64_t *rmq_hash, int *rmq_id) {
  GH_CHECK(g.dev.rmq_hash && g.dev.rmq_id, H2H_ERR_STATE, "sparse table not built");
  if (rmq_hash) GH_CUDA(cudaMemcpy(rmq_hash, g.dev.rmq_hash, sizeof(int64_t) * g.euler_n, cudaMemcpyDeviceToHost));
  if (rmq_id) GH_CUDA(cudaMemcpy(rmq_id, g.dev.rmq_id, sizeof(int) * g.rmq_total, cudaMemcpyDeviceToHost));
}

// The sparse table and firstAppeare are on the device since h2h_contract;
// labels since the fill.  Nothing is left to upload.
void upload_query_index(Graph &g) {
  GH_CHECK(g.dev.first && g.dev.rmq_hash && g.dev.rmq_id, H2H_ERR_STATE, "sparse table not built");
}

void run_query_batch(const Graph &g, const int *x, const int *y, int *out, int64_t n, int mode, cudaStream_t s,
                     int *bad) {
  if (n <= 0) return;
  const DeviceIndex &D = g.dev;
  QArgs A{x, y, out, n, g.n, D.first, D.depth, D.rmq_hash, D.rmq_id, D.pos_hash, D.pos_pos, D.drow, D.dis,
          bad ? bad : D.err, 0, D.rmq_closed ? D.euler : 0, D.rmq};
  const int threads = 256;
  const int mi = mode == H2H_QUERY_LCA ? 0 : 1;
  using Kernel = void (*)(QArgs);
  static const Kernel kernels[2][6] = {
      {query_tile_kernel<true, 32>, query_tile_kernel<true, 16>, query_tile_kernel<true, 8>,
       query_tile_kernel<true, 4>, query_tile_kernel<true, 2>, query_tile_kernel<true, 1>},
      {query_tile_kernel<false, 32>, query_tile_kernel<false, 16>, query_tile_kernel<false, 8>,
       query_tile_kernel<false, 4>, query_tile_kernel<false, 2>, query_tile_kernel<false, 1>}};
  // device shape, looked up once (thread-safe static initialisation: the
  // server's worker and callers' threads may arrive together)
  struct Shape {
    int nsm = 1, per_sm[2] = {1, 1};  // resident 256-thread blocks per SM (all tile widths use 40 registers)
  };
  static const Shape shape = [] {
    Shape sh;
    int dev = 0;
    GH_CUDA(cudaGetDevice(&dev));
    GH_CUDA(cudaDeviceGetAttribute(&sh.nsm, cudaDevAttrMultiProcessorCount, dev));
    for (int k = 0; k < 2; k++) {
      GH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sh.per_sm[k], kernels[k][0], 256, 0));
      sh.per_sm[k] = std::max(1, sh.per_sm[k]);
    }
    return sh;
  }();
  const int nsm = shape.nsm;
  const int per_sm[2] = {shape.per_sm[0], shape.per_sm[1]};
  // narrowest tile whose warps still fit one wave of resident warps
  const int64_t resident_warps = (int64_t)nsm * per_sm[mi] * (threads / 32);
  int ti = 0, tile = 32;
  while (ti < 5 && ((n + tile / 2 - 1) / (tile / 2)) <= resident_warps) {
    tile /= 2;
    ti++;
  }
  const int64_t tiles = (n + tile - 1) / tile;
  A.tiles = tiles;
  // one wave of resident blocks, grid-striding over the tiles
  const int blocks = (int)std::min<int64_t>((tiles + 7) / 8, (int64_t)nsm * per_sm[mi]);
  kernels[mi][ti]<<<std::max(1, blocks), threads, 0, s>>>(A);
  GH_CUDA(cudaGetLastError());
}

void run_query_batch_plain(const Graph &g, const int *x, const int *y, int *out, int64_t n, int mode,
                           cudaStream_t s) {
  if (n <= 0) return;
  const DeviceIndex &D = g.dev;
  QArgs A{x, y, out, n, g.n, D.first, D.depth, D.rmq_hash, D.rmq_id, D.pos_hash, D.pos_pos, D.drow, D.dis, D.err,
          0,      0,      0};
  const int threads = 256;
  int blocks = (int)std::min<int64_t>((n + threads - 1) / threads, INT32_MAX);
  if (mode == H2H_QUERY_LCA) query_kernel<1, true><<<blocks, threads, 0, s>>>(A);
  else query_kernel<1, false><<<blocks, threads, 0, s>>>(A);
  GH_CUDA(cudaGetLastError());
}

}  // namespace gh
