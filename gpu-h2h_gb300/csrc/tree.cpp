// tree.cpp -- label layout on the host, mallocH2HLabel_noHub
// (H2HConsturction.cu:618-722): the position lists of the level-synchronous
// fill.  The tree, the offsets and the block fill's position lists are built on
// the GPU (tree_gpu.cu, labels.cu).
#include <algorithm>
#include <atomic>

#include "graph.h"
#include "pool.h"

namespace gh {

void Graph::drop_build() {
  plan.reset();
  tree.reset();
  sets.reset();
  dev.release();
  for (std::vector<int> *v : {&elim, &x_id, &x_w, &father, &depth, &first, &pos_id, &pos_pos, &pos_w, &tree_bfs, &tree_hash})
    std::vector<int>().swap(*v);
  for (std::vector<int64_t> *v : {&x_off, &dis_hash, &pos_hash, &drow_host}) std::vector<int64_t>().swap(*v);
  head = -1;
  tree_height = n_levels = gpu_vertices = 0;
  x_total = decomposition_size = euler_n = h2h_size = rmq_total = pos_n = updates = row0 = row1 = 0;
  contracted = labelled = false;
}

void allocate_labels_and_bfs(Graph &g) {
  Clock clk;
  const int n = g.n;
  g.pos_n = g.x_total + n;
  // host position lists only for the level-synchronous fill; the block
  // fill builds them on the GPU from the device lists
  if (uses_level_fill(g)) {
    host_tree(g);
    if ((int64_t)g.x_id.size() != g.x_total) download_lists(g);
    Pool pool(useful_threads(g.threads, g.n));
    g.pos_id.resize(g.pos_n);
    g.pos_pos.resize(g.pos_n);
    g.pos_w.resize(g.pos_n);
    std::atomic<int> bad{-1};
    pool.parallel_for(n, 1024, [&](int64_t b, int64_t e, int) {
      std::vector<std::pair<int64_t, int>> tmp;
      for (int64_t vv = b; vv < e; vv++) {
        const int v = (int)vv;
        const int d = g.depth[v];
        tmp.clear();
        for (int64_t k = g.x_off[v]; k < g.x_off[v + 1]; k++) {
          int a = g.x_id[k], p = g.depth[a] - 1;
          if (p < 0 || p >= d - 1) { bad = v; continue; }
          tmp.push_back({(int64_t)p << 32 | (uint32_t)a, g.x_w[k]});
        }
        tmp.push_back({(int64_t)(d - 1) << 32 | (uint32_t)v, 0});
        std::sort(tmp.begin(), tmp.end());  // positions are distinct
        int64_t o = g.pos_hash[v];
        for (size_t k = 0; k < tmp.size(); k++) {
          g.pos_pos[o + k] = (int)(tmp[k].first >> 32);
          g.pos_id[o + k] = (int)(tmp[k].first & 0xffffffff);
          g.pos_w[o + k] = tmp[k].second;
        }
      }
    });
    GH_CHECK(bad.load() < 0, H2H_ERR_STATE, "an upper neighbour is not an ancestor in the tree");
  } else {
    std::vector<int>().swap(g.pos_id);
    std::vector<int>().swap(g.pos_pos);
    std::vector<int>().swap(g.pos_w);
  }
  g.t.malloc_labels = clk.us();
}

}  // namespace gh
