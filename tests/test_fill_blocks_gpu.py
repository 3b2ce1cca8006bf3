"""The blocked L4 fill at the sizes where it can go wrong: blocks of one node,
full blocks and one node more, small subtrees that do and do not fit their
father's block, separators around one and two staging steps, ragged column
ends.  Labels must equal the oracle's, entry by entry (int32, zero
tolerance); with weights that differ by direction they must equal the fill's
recursion evaluated row by row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _write(root, n, edges, H):
    """Edge / ID / Cut files of an undirected graph (u, v, w forth, w back);
    the partition halves the vertex range level by level."""
    e, i, c = (str(root / f) for f in ("Edge.txt", "ID.txt", "Cut.txt"))
    with open(e, "w") as f:
        f.write("%d %d\n" % (n, 2 * len(edges)))
        for u, v, w, x in edges:
            f.write("a %d %d %d\na %d %d %d\n" % (u + 1, v + 1, w, v + 1, u + 1, x))
    with open(i, "w") as f:
        f.write("%d\n" % n + "".join("%d 0.0 0.0 %d\n" % (k, k) for k in range(n)))
    with open(c, "w") as f:
        f.write("%d\n" % H)
        cells = [(0, n)]
        for h in range(1, H + 1):
            f.write("".join("%d %d %d\n" % (h, a, b) for a, b in cells))
            cells = [x for a, b in cells for x in ((a, (a + b) // 2), ((a + b) // 2, b))]
    return e, i, c


def _path(n):
    return n, [(k, k + 1, 1 + k % 7) for k in range(n - 1)]


def _star(leaves):
    return leaves + 1, [(leaves, k, 3 + k % 5) for k in range(leaves)]


def _clique(n):
    return n, [(a, b, 5 + (a * 7 + b * 11) % 23) for a in range(n) for b in range(a)]


def _clique_with_tails(n, tail):
    """Tails are light subtrees of `tail` nodes hanging off a clique's chain."""
    n0, edges = _clique(n)
    edges = list(edges)
    for k in range(n):
        prev = k
        for t in range(tail):
            edges.append((prev, n0, 1 + (k + t) % 9))
            prev = n0
            n0 += 1
    return n0, edges


def _grid(r, c):
    e = []
    for y in range(r):
        for x in range(c):
            if x + 1 < c:
                e.append((y * c + x, y * c + x + 1, 1 + (3 * x + 5 * y) % 13))
            if y + 1 < r:
                e.append((y * c + x, (y + 1) * c + x, 1 + (7 * x + 2 * y) % 11))
    return r * c, e


GRAPHS = {"pair": _path(2), "path33": _path(33), "path200": _path(200), "star15": _star(15), "star31": _star(31),
          "star32": _star(32), "star70": _star(70), "clique31": _clique(31), "clique32": _clique(32),
          "clique33": _clique(33), "clique34": _clique(34), "clique65": _clique(65), "clique98": _clique(98),
          "tails16": _clique_with_tails(40, 16), "tails17": _clique_with_tails(36, 17),
          "tails3": _clique_with_tails(97, 3), "grid": _grid(37, 41)}


@pytest.mark.parametrize("name", GRAPHS)
def test_labels_match_oracle(tmp_path, name):
    import gpuh2h
    from oracle import oracle
    n, edges = GRAPHS[name]
    H = 3 if n > 100 else 1
    files = _write(tmp_path, n, [(u, v, w, w) for u, v, w in edges], H)
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
    n, edges = _grid(19, 23)
    files = _write(tmp_path, n, [(u, v, w, 1 + (w * 5 + u) % 17) for u, v, w in edges], 3)
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
