"""Partitions far shallower than the graph asks for: the bottom level has many
cells of thousands of members, whose rows lie in global memory on clusters of
1, 2, 4 and 8 CTAs.  Order, lists and weights equal the list kernels' (zero
tolerance)."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,H,ctas", [(400000, 9, 1), (264346, 8, 2), (264346, 7, 4), (264346, 6, 8)])
def test_many_large_cells(tmp_path, monkeypatch, capfd, n, H, ctas):
    import gpuh2h
    gpuh2h.generate_road(str(tmp_path), "r", n=n, target_arcs=int(n * 2.776), aspect_milli=1300, jitter_milli=300,
                         diag_permille=50, hw_tiers=1, hw_permille10=50, hw_k=3, hw_scale_milli=400,
                         partition_height=H, seed=5, cols=0, drop_permille=0)
    files = gpuh2h.files_for(str(tmp_path), "r")
    monkeypatch.setenv("GPUH2H_TRACE", "1")
    got = []
    for lists in (False, True):
        if lists:
            monkeypatch.setenv("GPUH2H_LIST_ELIM", "1")
        g = gpuh2h.Graph("r", H, 2, 8, 1, files=files)
        capfd.readouterr()
        g.contraction_noHub(1)
        err = capfd.readouterr().err
        if not lists:
            bottom = re.findall(r"elim bits level %d: (\d+) cells x (\d+) CTAs.*rows in global memory" % H, err)
            assert bottom == [(str(2 ** (H - 1)), str(ctas))], err
        got.append([g.order(), *g.adj()])
        g.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
