"""Cells whose rows outgrow a cluster's shared memory: one grid of up to 128
CTAs per cell, for one graph and for two side by side.  Order and lists equal
the list kernels' (zero tolerance)."""
import numpy as np
import pytest

from small_graphs import grid, write

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", (((83, 84),), ((83, 84), (84, 85)), ((127, 129),)))
def test_large_cells_match_list_kernels(tmp_path, monkeypatch, capfd, sizes):
    import gpuh2h
    files = []
    for k, (r, c) in enumerate(sizes):
        (tmp_path / str(k)).mkdir()
        n, edges = grid(r, c)
        files.append(write(tmp_path / str(k), n, [(u, v, w, 1 + (3 * w + u) % 17) for u, v, w in edges], 1))
    monkeypatch.setenv("GPUH2H_TRACE", "1")
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("GPUH2H_LIST_ELIM", "1")
        gs = [gpuh2h.Graph("g", 1, 1, 2, 1, files=f) for f in files]
        capfd.readouterr()
        b = gpuh2h.Batch(gs, 2) if len(gs) > 1 else gs[0].contraction_noHub(1)
        assert ("one grid" in capfd.readouterr().err) == (not lists)
        got.append([x for g in gs for x in (g.order(), *g.adj())])
        if len(gs) > 1:
            b.close()
        for g in gs:
            g.close()
    assert all(np.array_equal(x, y) for x, y in zip(*got))
