"""The elimination on bit rows at the sizes where it can go wrong: cells of
one member, one word and one member more, cells spread over a cluster, rows
in global memory, parallel arcs inside and across cells, weights that differ
by direction.  Order, lists and weights must equal the oracle's, and the list
kernels' (zero tolerance)."""
import numpy as np
import pytest

from small_graphs import clique, grid, path, star, write

pytestmark = pytest.mark.gpu


def _repeat(edges, every):
    """Every `every`-th edge twice more, once lighter and once heavier."""
    out = []
    for k, (u, v, w) in enumerate(edges):
        if k % every == 0:
            out.append((u, v, w + 9))
        out.append((u, v, w))
        if k % every == 0:
            out.append((u, v, max(1, w - 2)))
    return out


def _twisted(edges):
    return [(u, v, w, 1 + (w * 7 + u + 3 * v) % 31) for u, v, w in edges]


CASES = {
    # name: (n, edges, H, the C values)
    "one": (1, [], 1, (1,)),
    "path2": (*path(2), 1, (1,)),
    "path65": (*path(65), 2, (1, 2)),
    "star33": (*star(33), 1, (1,)),
    "clique32": (*clique(32), 1, (1,)),
    "clique33": (*clique(33), 2, (1, 2)),
    "grid": (*grid(37, 41), 4, (1, 2, 3, 4)),
    "parallel": (37 * 41, _repeat(grid(37, 41)[1], 5), 4, (1, 2, 3, 4)),
    "every_edge_parallel": (23 * 9, _repeat(grid(23, 9)[1], 1), 3, (1, 2, 3)),
    "cluster": (*grid(41, 43), 1, (1,)),
    "global_rows": (*grid(72, 73), 1, (1,)),
}


@pytest.mark.parametrize("name", CASES)
def test_order_and_lists_match_oracle(tmp_path, monkeypatch, name):
    import gpuh2h
    from oracle import oracle
    n, edges, H, Cs = CASES[name]
    files = write(tmp_path, n, _twisted(edges), H)
    for C in Cs:
        o = oracle.OracleGraph(*files, H, C, 2).contract()
        ref = dict(zip(("hash", "id", "w"), o.adj()))
        for lists in (False, True):
            if lists:
                monkeypatch.setenv("GPUH2H_LIST_ELIM", "1")
            else:
                monkeypatch.delenv("GPUH2H_LIST_ELIM", raising=False)
            g = gpuh2h.Graph("t", H, C, 2, 1, files=files)
            g.contraction_noHub(1)
            assert np.array_equal(g.order(), o.order()), (name, C, lists)
            got = dict(zip(("hash", "id", "w"), g.adj()))
            for k in ref:
                assert np.array_equal(got[k], ref[k]), (name, C, lists, k)
            assert np.array_equal(g.tree()[0], o.father())
            g.close()
        o.close()


def test_batch_rebuild_takes_new_weights(tmp_path):
    """A rebuild on bit rows computes weights alone: equal to a fresh build,
    parallel arcs and one-way weights included."""
    import gpuh2h
    specs = []
    for k, name in enumerate(("parallel", "clique33", "grid")):
        n, edges, H, _ = CASES[name]
        d = tmp_path / str(k)
        d.mkdir()
        specs.append((write(d, n, _twisted(edges), H), H))
    graphs = [gpuh2h.Graph("b", H, 1, 2, 1, files=f) for f, H in specs]
    b = gpuh2h.Batch(graphs, 2)
    for rnd in range(2):
        for i, g in enumerate(graphs):
            off, v, w = g.input_arcs()
            new = ((w.astype(np.int64) * (rnd + 3) + 5 * np.arange(len(w))) % 97 + 1).astype(np.int32)
            b.set_weights(i, new)
            edge = str(tmp_path / ("e%d" % i))
            gpuh2h.write_edge_file(edge, off, v, new)
        b.rebuild()
        for i, (g, (f, H)) in enumerate(zip(graphs, specs)):
            s = gpuh2h.Graph("s", H, 1, 2, 1, files=(str(tmp_path / ("e%d" % i)), f[1], f[2]))
            s.contraction_noHub(1)
            s.constructLabel_noHub(2, 1, gpuh2h.LABEL_L4)
            assert all(np.array_equal(x, y) for x, y in zip(g.adj(), s.adj()))
            assert np.array_equal(g.labels()["dis"], s.labels()["dis"])
            s.close()
    b.close()
    for g in graphs:
        g.close()
