"""The blocked L4 fill at the sizes where it can go wrong: blocks of one node,
full blocks and one node more, small subtrees that do and do not fit their
father's block, separators around one and two staging steps, ragged column
ends.  Labels must equal the oracle's, entry by entry (int32, zero
tolerance); with weights that differ by direction they must equal the fill's
recursion evaluated row by row."""
import numpy as np
import pytest

from small_graphs import clique, clique_with_tails, grid, path, star, write

pytestmark = pytest.mark.gpu


GRAPHS = {"pair": path(2), "path33": path(33), "path200": path(200), "star15": star(15), "star31": star(31),
          "star32": star(32), "star70": star(70), "clique31": clique(31), "clique32": clique(32),
          "clique33": clique(33), "clique34": clique(34), "clique65": clique(65), "clique98": clique(98),
          "tails16": clique_with_tails(40, 16), "tails17": clique_with_tails(36, 17),
          "tails3": clique_with_tails(97, 3), "grid": grid(37, 41)}


@pytest.mark.parametrize("name", GRAPHS)
def test_labels_match_oracle(tmp_path, name):
    import gpuh2h
    from oracle import oracle
    n, edges = GRAPHS[name]
    H = 3 if n > 100 else 1
    files = write(tmp_path, n, [(u, v, w, w) for u, v, w in edges], H)
    for C in {1, H}:
        g = gpuh2h.Graph("t", H, C, 2, 1, files=files)
        g.contraction_noHub(1)
        g.constructLabel_noHub(2, 1, gpuh2h.LABEL_L4)
        o = oracle.OracleGraph(*files, H, C, 2).contract().build_labels(l4=True)
        assert np.array_equal(g.order(), o.order())
        got, ref = g.labels(), o.labels()
        for k in ("dis_hash", "pos_hash", "pos_pos", "dis"):
            assert np.array_equal(got[k], ref[k]), (name, C, k)
        g.close()
        o.close()


def test_one_way_weights_follow_the_recursion(tmp_path):
    import gpuh2h
    n, edges = grid(19, 23)
    files = write(tmp_path, n, [(u, v, w, 1 + (w * 5 + u) % 17) for u, v, w in edges], 3)
    g = gpuh2h.Graph("t", 3, 1, 2, 1, files=files)
    g.contraction_noHub(1)
    g.constructLabel_noHub(2, 1, gpuh2h.LABEL_L4)
    lab, (off, ids, ws), (father, depth, _) = g.labels(), g.adj(), g.tree()
    rows = {}
    for v in g.bfs()[0]:
        d = depth[v]
        anc = np.zeros(d, np.int64)
        a = v
        for j in range(d - 1, -1, -1):
            anc[j] = a
            a = father[a]
        row = np.zeros(d, np.int64)
        for j in range(d - 1):
            best = 1 << 40
            for u, w in zip(ids[off[v]:off[v + 1]], ws[off[v]:off[v + 1]]):
                p = depth[u] - 1
                best = min(best, w + (rows[u][j] if p > j else 0 if p == j else rows[anc[j]][p]))
            row[j] = best
        rows[v] = row
        assert np.array_equal(lab["dis"][lab["dis_hash"][v]:lab["dis_hash"][v] + d], row), v
    g.close()
