"""Lists that outgrow the pool of the elimination on bit rows: a random graph
of degree 6 fills in to about half of a clique, more than the 192 entries a
vertex the pool starts with.  The run is repeated with a larger pool; order
and lists equal the list kernels' (zero tolerance)."""
import random

import numpy as np
import pytest

from small_graphs import grid, write

pytestmark = pytest.mark.gpu


def _random(n, degree, seed):
    rng = random.Random(seed)
    edges = {(k, k + 1) for k in range(n - 1)}  # connected
    while len(edges) < n * degree // 2:
        u, v = rng.randrange(n), rng.randrange(n)
        if u != v:
            edges.add((min(u, v), max(u, v)))
    return n, [(u, v, 1 + rng.randrange(50), 1 + rng.randrange(50)) for u, v in sorted(edges)]


@pytest.mark.parametrize("H", (1, 2))
@pytest.mark.parametrize("batch", (False, True))
def test_pool_grows(tmp_path, monkeypatch, capfd, H, batch):
    import gpuh2h
    n, edges = _random(3200, 6, 7)
    (tmp_path / "a").mkdir()
    (tmp_path / "b").mkdir()
    files = [write(tmp_path / "a", n, edges, H)]
    if batch:
        m, small = grid(11, 13)
        files.append(write(tmp_path / "b", m, [(u, v, w, w) for u, v, w in small], H))
    monkeypatch.setenv("GPUH2H_TRACE", "1")
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("GPUH2H_LIST_ELIM", "1")
        gs = [gpuh2h.Graph("g", H, 1, 2, 1, files=f) for f in files]
        capfd.readouterr()
        b = gpuh2h.Batch(gs, 2) if batch else gs[0].contraction_noHub(1)
        assert ("list pool grown" in capfd.readouterr().err) == (not lists)
        got.append([x for g in gs for x in (g.order(), *g.adj())])
        if batch:
            b.close()
        for g in gs:
            g.close()
    assert all(np.array_equal(x, y) for x, y in zip(*got))
