// input_gpu.cu -- the Edge and ID files on the GPU: parsing, adjacency offsets
// and the checks of the loader (Graph_Fundamental.cu:4-95).
//
// The files' text goes to the device as it is.  A pass counts the lines that
// start in every 16 KB, a scan numbers them, and a second pass parses each
// line in one thread: an arc "a u v w" or a vertex "idx lon lat id".  Arcs that
// do not come grouped by tail are sorted by it, stably, so every vertex keeps
// its arcs in file order (the reference's push_back).  Then each arc looks for
// its reverse in its head's list, and a lock-free union-find (roots link under
// smaller roots by compare-and-swap) tells whether the graph is connected.
//
// Only the plain form is taken here: one record per line and as many lines as
// the header says, unsigned decimal numbers in range, no self loops, a
// permutation of positions, every reverse arc there, one component.  Anything
// else returns false and the host reader (io.cpp) decides, with its own rules
// and errors.  Bound: the host reading the files (60 MB for 2.8M arcs) and the
// copies; the kernels take well under a millisecond.  On one GB300 the load of a
// 1M-vertex graph takes 5 ms, 26 ms by the host reader on 16 threads.
#include <dlfcn.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>

#include "graph.h"
#include "quiet.h"
#include "sort.h"

namespace gh {

namespace {

constexpr int kBytes = 64;                       // text per thread
constexpr int kTextThreads = 256;
constexpr int64_t kTextBlock = kBytes * kTextThreads;
constexpr int kScanDegree = 512;  // longest list searched arc by arc
constexpr int kLineBytes = 256;   // longest line read by one thread

// Later kernels run behind the earlier ones without the host having looked:
// each does nothing once `odd` or `unsorted` is set, so none reads arrays that
// were not filled.
struct LoadFlags {
  int odd;       // not the plain form: a line, the number of lines, a vertex without an ID line, a long list
  int unsorted;  // a tail smaller than its predecessor's
  int missing;   // an arc without its reverse
  int split;     // more than one component
};

__device__ __forceinline__ bool stopped(const LoadFlags *f) { return f->odd || f->unsorted; }

// A record starts at a non-newline byte that follows a newline; text[0] is the
// newline that ends the header.
__device__ __forceinline__ int line_starts(const char *text, int64_t size, int64_t base, unsigned long long *mask) {
  unsigned long long m = 0;
  char prev = base > 0 && base <= size ? text[base - 1] : 0;
  if (base + kBytes <= size) {
    const uint4 *p = reinterpret_cast<const uint4 *>(text + base);
#pragma unroll
    for (int q = 0; q < kBytes / 16; q++) {
      const uint4 x = p[q];
      const unsigned w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int k = 0; k < 16; k++) {
        const char c = (char)(w[k >> 2] >> (8 * (k & 3)));
        if (prev == '\n' && c != '\n') m |= 1ull << (16 * q + k);
        prev = c;
      }
    }
  } else {
    for (int k = 0; k < kBytes && base + k < size; k++) {
      const char c = text[base + k];
      if (prev == '\n' && c != '\n') m |= 1ull << k;
      prev = c;
    }
  }
  *mask = m;
  return __popcll(m);
}

// The two files' records: the ID file's text first, the Edge file's at a
// 256-byte boundary behind it, each in blocks of its own.
struct LoadArgs {
  const char *text[2];
  int64_t size[2];
  unsigned blocks[2];
  int *count;            // lines per block, and one word more
  const int64_t *first;  // lines before each block
  int n;
  int64_t m;
  int *part, *pos, *tail, *v, *w, *parent;
  LoadFlags *flags;
};

// Lines per block; what the parser only sets in part starts unset.
__global__ void __launch_bounds__(kTextThreads) count_lines_kernel(LoadArgs A) {
  __shared__ int s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  const int f = blockIdx.x >= A.blocks[0];
  const int64_t base = (blockIdx.x - (f ? A.blocks[0] : 0)) * kTextBlock + (int64_t)threadIdx.x * kBytes;
  unsigned long long m;
  int c = line_starts(A.text[f], A.size[f], base, &m);
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, c);
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t == 0) {
    A.count[A.blocks[0] + A.blocks[1]] = 0;
    *A.flags = LoadFlags{};
  }
  for (int64_t i = t; i < A.n; i += (int64_t)gridDim.x * blockDim.x) A.part[i] = A.pos[i] = -1;
  __syncthreads();
  if (threadIdx.x == 0) A.count[blockIdx.x] = s_sum;
}

struct Reader {
  const char *p, *e;  // e: the text's end, or the longest line's
  __device__ char at() const { return p < e ? *p : '\n'; }
  __device__ bool blanks() {  // at least one space or tab
    const char *s = p;
    while (at() == ' ' || at() == '\t') p++;
    return p > s;
  }
  __device__ bool number(long long &v) {  // 1 to 10 digits
    v = 0;
    int d = 0;
    while (d < 11 && at() >= '0' && at() <= '9') {
      v = v * 10 + (at() - '0');
      p++;
      d++;
    }
    return d >= 1 && d <= 10;
  }
  __device__ bool field() {  // anything without blanks
    const char *s = p;
    while (at() != ' ' && at() != '\t' && at() != '\n' && at() != '\r') p++;
    return p > s;
  }
  __device__ bool end(const char *text_end) {  // nothing but blanks up to the end of the line
    while (at() == ' ' || at() == '\t' || at() == '\r') p++;
    return p < e ? *p == '\n' : e == text_end;
  }
};

// "a u v w" into tail, v and w; "idx lon lat id" into part[idx] = id, pos[id] = idx.
__global__ void __launch_bounds__(kTextThreads) parse_lines_kernel(LoadArgs A) {
  const unsigned nb = A.blocks[0] + A.blocks[1];
  const int n = A.n;
  if (A.first[A.blocks[0]] != n || A.first[nb] - n != A.m) {  // lines in all
    if (blockIdx.x == 0 && threadIdx.x == 0) A.flags->odd = 1;
    return;
  }
  const bool arcs = blockIdx.x >= A.blocks[0];
  const char *text = A.text[arcs];
  const int64_t size = A.size[arcs], records = arcs ? A.m : n;
  __shared__ int s_warp[kTextThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t base = (blockIdx.x - (arcs ? A.blocks[0] : 0)) * kTextBlock + (int64_t)threadIdx.x * kBytes;
  unsigned long long m;
  const int cnt = line_starts(text, size, base, &m);
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  int64_t k = A.first[blockIdx.x] - (arcs ? n : 0) + incl - cnt;
  for (int w = 0; w < wid; w++) k += s_warp[w];
  bool odd = false;
  while (m) {
    const int64_t at = base + (__ffsll(m) - 1);
    Reader r{text + at, text + min(size, at + kLineBytes)};
    m &= m - 1;
    long long x, y, z;
    if (arcs) {
      bool ok = r.at() == 'a';
      r.p++;
      ok = ok && r.blanks() && r.number(x) && r.blanks() && r.number(y) && r.blanks() && r.number(z) && r.end(text + size);
      ok = ok && x >= 1 && x <= n && y >= 1 && y <= n && x != y && z <= INT_MAX && k < records;
      if (ok) {
        A.tail[k] = (int)x - 1;
        A.v[k] = (int)y - 1;
        A.w[k] = (int)z;
      }
      odd |= !ok;
    } else {
      bool ok = r.number(x) && r.blanks() && r.field() && r.blanks() && r.field() && r.blanks() && r.number(y) && r.end(text + size);
      ok = ok && x < n && y < n && k < records;
      if (ok) {
        A.part[x] = (int)y;
        A.pos[y] = (int)x;
      }
      odd |= !ok;
    }
    k++;
  }
  if (odd) A.flags->odd = 1;
}

// Whether the tails come in order and every position and vertex has its line;
// every vertex a component of its own.
__global__ void sorted_kernel(LoadArgs A) {
  if (A.flags->odd) return;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = t + 1; i < A.m; i += step)
    if (A.tail[i] < A.tail[i - 1]) A.flags->unsorted = 1;
  bool odd = false;
  for (int64_t i = t; i < A.n; i += step) {
    odd |= A.part[i] < 0 || A.pos[i] < 0;
    A.parent[i] = (int)i;
  }
  if (odd) A.flags->odd = 1;
}

__global__ void iota_kernel(int *a, int64_t m) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = (int)i;
}

__global__ void gather_arcs_kernel(const int *from, const int *v, const int *w, int *v2, int *w2, int64_t m) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    v2[i] = v[from[i]];
    w2[i] = w[from[i]];
  }
}

// off[u] = the first arc whose tail is >= u.
__global__ void offsets_kernel(const int *tail, int64_t m, int n, int *off, const LoadFlags *flags) {
  if (stopped(flags)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= m; i += (int64_t)gridDim.x * blockDim.x) {
    const int prev = i == 0 ? -1 : tail[i - 1], cur = i == m ? n : tail[i];
    for (int u = prev + 1; u <= cur; u++) off[u] = (int)i;
  }
}

__device__ __forceinline__ int find_root(int *parent, int x) {
  for (;;) {
    const int p = *(volatile int *)(parent + x);
    if (p == x) return x;
    const int q = *(volatile int *)(parent + p);
    if (q != p) *(volatile int *)(parent + x) = q;  // halving: an ancestor closer to the root, never a larger id
    x = p;
  }
}

// Reverse arcs and components.  Roots only ever link under smaller ids, so
// every find and every link loop ends.
__global__ void check_arcs_kernel(const int *tail, const int *head, const int *off, int64_t m, int *parent,
                                  LoadFlags *flags) {
  if (stopped(flags)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const int u = tail[i], v = head[i];
    const int b0 = off[v], b1 = off[v + 1];
    if (b1 - b0 > kScanDegree) {  // too long to search arc by arc
      flags->odd = 1;
      return;
    }
    bool back = false;
    for (int e = b0; e < b1 && !back; e++) back = __ldg(head + e) == u;
    if (!back) flags->missing = 1;
    if (u < v) continue;
    int a = find_root(parent, u), b = find_root(parent, v);
    while (a != b) {
      if (a < b) {
        const int t = a;
        a = b;
        b = t;
      }
      const int old = atomicCAS(parent + a, a, b);
      if (old == a) break;
      a = find_root(parent, old);
      b = find_root(parent, b);
    }
  }
}

__global__ void check_connected_kernel(int *parent, int n, LoadFlags *flags) {
  if (stopped(flags)) return;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    if (find_root(parent, v) != 0) flags->split = 1;
}

unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>(4096, (n + 255) / 256)); }

// Offsets and checks of arcs sorted by tail.
void check_arcs(const DeviceInput &in, const LoadArgs &A, cudaStream_t s) {
  offsets_kernel<<<blocks_for(A.m + 1), 256, 0, s>>>(A.tail, A.m, A.n, in.off, A.flags);
  check_arcs_kernel<<<blocks_for(A.m), 256, 0, s>>>(A.tail, in.v, in.off, A.m, A.parent, A.flags);
  check_connected_kernel<<<blocks_for(A.n), 256, 0, s>>>(A.parent, A.n, A.flags);
  GH_CUDA(cudaGetLastError());
}

// One allocation for the graph, one for the scratch, seven kernels and one
// wait: a batch's loads are short (a 4,096-vertex graph's 0.5 ms with a wait and
// an allocation per step, 0.31 with one of each and thirteen kernels, 0.27 now).
bool parse_input(Graph &g, const char *ids, int64_t ids_size, const char *arcs, int64_t arcs_size, int64_t m) {
  const int n = g.n;
  if (n > ids_size / 7 || m > arcs_size / 7) return false;  // a record takes eight bytes, the last one seven
  RelaxedCapture relaxed;
  Workspace ws;
  QuietStream q;
  auto in = std::make_shared<DeviceInput>();
  GH_CUDA(cudaGetDevice(&in->device));
  in->mem.reserve(4 * (3 * (size_t)n + 2 * (size_t)m) + 5 * 256 + 256);
  in->off = in->mem.get<int>((int64_t)n + 1);
  in->v = in->mem.get<int>(m);
  in->w = in->mem.get<int>(m);
  in->part = in->mem.get<int>(n);
  in->pos = in->mem.get<int>(n);
  const int64_t nb = (ids_size + kTextBlock - 1) / kTextBlock + (arcs_size + kTextBlock - 1) / kTextBlock;
  ws.reserve((size_t)(ids_size + arcs_size + 4 * (m + n) + 12 * (nb + 1) + 32 * (nb / kScanTile + 2)) + (64 << 10));
  LoadArgs A{};
  A.flags = ws.get<LoadFlags>(1);
  A.tail = ws.get<int>(m);
  A.parent = ws.get<int>(n);
  char *text[2] = {ws.get<char>(ids_size), ws.get<char>(arcs_size)};
  A.count = ws.get<int>(nb + 1);
  int64_t *first = ws.get<int64_t>(nb + 1);
  GH_CUDA(cudaMemcpyAsync(text[0], ids, ids_size, cudaMemcpyHostToDevice, q.s));
  GH_CUDA(cudaMemcpyAsync(text[1], arcs, arcs_size, cudaMemcpyHostToDevice, q.s));
  A.text[0] = text[0];
  A.text[1] = text[1];
  A.size[0] = ids_size;
  A.size[1] = arcs_size;
  A.blocks[0] = (unsigned)((ids_size + kTextBlock - 1) / kTextBlock);
  A.blocks[1] = (unsigned)(nb - A.blocks[0]);
  A.first = first;
  A.n = n;
  A.m = m;
  A.part = in->part;
  A.pos = in->pos;
  A.v = in->v;
  A.w = in->w;
  count_lines_kernel<<<(unsigned)nb, kTextThreads, 0, q.s>>>(A);
  GH_CUDA(cudaGetLastError());
  exclusive_scan<int>(A.count, first, nb + 1, ws, q.s);
  parse_lines_kernel<<<(unsigned)nb, kTextThreads, 0, q.s>>>(A);
  sorted_kernel<<<blocks_for(std::max<int64_t>(m, n)), 256, 0, q.s>>>(A);
  GH_CUDA(cudaGetLastError());
  check_arcs(*in, A, q.s);
  LoadFlags f{};
  q.read(&f, A.flags, sizeof(f));
  if (f.odd) return false;
  if (f.unsorted) {  // the arcs of a vertex in file order: a stable sort by tail
    int *from = ws.get<int>(m), *v2 = in->mem.get<int>(m), *w2 = in->mem.get<int>(m);
    iota_kernel<<<blocks_for(m), 256, 0, q.s>>>(from, m);
    int bits = 1;
    while (bits < 32 && (int64_t(1) << bits) <= n) bits++;
    radix_sort_pairs(reinterpret_cast<unsigned *>(A.tail), from, m, bits, ws, q.s);
    gather_arcs_kernel<<<blocks_for(m), 256, 0, q.s>>>(from, in->v, in->w, v2, w2, m);
    GH_CUDA(cudaGetLastError());
    in->v = v2;
    in->w = w2;
    GH_CUDA(cudaMemsetAsync(A.flags, 0, sizeof(LoadFlags), q.s));
    check_arcs(*in, A, q.s);
    q.read(&f, A.flags, sizeof(f));
  }
  if (f.odd || f.missing || f.split) return false;
  g.m = m;
  g.input = in;
  return true;
}

// Whether this process has used the GPU already.  A process that has not is
// left alone: it may still fork, and its children use the GPU.
bool driver_initialised() {
  void *lib = dlopen("libcuda.so.1", RTLD_LAZY | RTLD_NOLOAD);
  if (!lib) return false;
  using Count = int (*)(int *);
  const Count count = reinterpret_cast<Count>(dlsym(lib, "cuDeviceGetCount"));
  int devices = 0;
  const bool up = count && count(&devices) == 0 && devices > 0;
  dlclose(lib);
  return up;
}

}  // namespace

DeviceInput::~DeviceInput() {
  RelaxedCapture relaxed;
  mem.release();
}

// ids / arcs: the text after each file's header, from the newline that ends
// it.  True: g.m and g.input are set and every check of the loader holds.
bool load_input_gpu(Graph &g, const char *ids, int64_t ids_size, const char *arcs, int64_t arcs_size, int64_t m) {
  if (m < 1 || m >= INT32_MAX || ids_size < 1 || arcs_size < 1 || ids[0] != '\n' || arcs[0] != '\n') return false;
  if (!driver_initialised()) return false;
  try {
    return parse_input(g, ids, ids_size, arcs, arcs_size, m);
  } catch (const Error &) {  // no room on the device, or no device: the host reader needs neither
    cudaGetLastError();
    return false;
  }
}

// The graph's input on the device, uploaded from the host reader's arrays if need be.
// Loading names no device, so a graph may be built on another than it was
// parsed on.
const DeviceInput &input_device(Graph &g) {
  int device = 0;
  GH_CUDA(cudaGetDevice(&device));
  if (g.input && g.input->device != device) {
    input_host(g);
    g.input.reset();
  }
  if (!g.input) {
    GH_CHECK((int64_t)g.adj_off.size() == (int64_t)g.n + 1 && (int)g.part_ids.size() == g.n, H2H_ERR_STATE,
             "the input arcs are not loaded");
    auto in = std::make_shared<DeviceInput>();
    in->device = device;
    in->off = in->mem.get<int>((int64_t)g.n + 1);
    in->v = in->mem.get<int>(g.m);
    in->w = in->mem.get<int>(g.m);
    in->part = in->mem.get<int>(g.n);
    in->pos = in->mem.get<int>(g.n);
    GH_CUDA(cudaMemcpy(in->off, g.adj_off.data(), sizeof(int) * ((size_t)g.n + 1), cudaMemcpyHostToDevice));
    if (g.m) {
      GH_CUDA(cudaMemcpy(in->v, g.adj_v.data(), sizeof(int) * g.m, cudaMemcpyHostToDevice));
      GH_CUDA(cudaMemcpy(in->w, g.adj_w.data(), sizeof(int) * g.m, cudaMemcpyHostToDevice));
    }
    GH_CUDA(cudaMemcpy(in->part, g.part_ids.data(), sizeof(int) * (size_t)g.n, cudaMemcpyHostToDevice));
    GH_CUDA(cudaMemcpy(in->pos, g.id_hash.data(), sizeof(int) * (size_t)g.n, cudaMemcpyHostToDevice));
    g.input = in;
  }
  return *g.input;
}

// The input's host arrays, which the accessors read; downloaded once where the
// file was parsed on the device.
const HostInput &input_host(const Graph &g) {
  std::lock_guard<std::mutex> lock(g.host_lock);
  HostInput &h = const_cast<Graph &>(g);
  if (g.input && (int64_t)g.adj_off.size() != (int64_t)g.n + 1) {
    const DeviceInput &in = *g.input;
    RelaxedCapture relaxed;
    OnDevice there(in.device);
    QuietStream q;
    h.adj_v.resize(g.m);
    h.adj_w.resize(g.m);
    h.part_ids.resize(g.n);
    h.id_hash.resize(g.n);
    std::vector<int> off((size_t)g.n + 1);
    q.read(h.adj_v.data(), in.v, sizeof(int) * (size_t)g.m);
    q.read(h.adj_w.data(), in.w, sizeof(int) * (size_t)g.m);
    q.read(h.part_ids.data(), in.part, sizeof(int) * (size_t)g.n);
    q.read(h.id_hash.data(), in.pos, sizeof(int) * (size_t)g.n);
    q.read(off.data(), in.off, sizeof(int) * off.size());
    h.adj_off.swap(off);
  }
  return h;
}

}  // namespace gh
