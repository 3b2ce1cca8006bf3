"""Batches at the sizes where the query kernel changes shape: one pair, the
narrow tiles, the last batch read in place from host memory and the first one
copied, one wave of warps and more; both modes, device and host buffers, pairs
with equal and out-of-range ids among them.  Answers must equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built(cfg0_root):
    import gpuh2h
    from oracle import oracle
    files = gpuh2h.files_for(cfg0_root, "cfg0")
    g = gpuh2h.Graph("t", 6, 2, 4, 1, files=files)
    g.contraction_noHub(1)
    g.constructLabel_noHub(2, 1, gpuh2h.LABEL_L4)
    o = oracle.OracleGraph(*files, 6, 2, 4).contract().build_labels(l4=True)
    yield g, o
    g.close()
    o.close()


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 4095, 4096, 4097, 7297, 29185, 58369, 116737, 233473, 300001])
@pytest.mark.parametrize("lca", [True, False])
def test_batch_sizes(built, n, lca):
    import torch

    import gpuh2h
    g, o = built
    x, y = gpuh2h.uniform_pairs(4096, n, n)
    k = min(n, 50000)
    x[:k:3], y[:k:3] = g.local_pairs(len(x[:k:3]), 6, n)  # a run of near pairs
    y[::17] = x[::17]
    ref = o.query_batch(x, y, lca=lca)
    mode = gpuh2h.QUERY_LCA if lca else gpuh2h.QUERY_NOLCA
    assert np.array_equal(g.query(x, y, mode), ref)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = torch.full_like(xd, -7)
    g.query_device(xd.data_ptr(), yd.data_ptr(), out.data_ptr(), n, mode, torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy(), ref)
    # one bad id: its pair answers -1, the others are answered, the next call is clean
    bad = x.copy()
    bad[n // 2] = 4096
    with pytest.raises(gpuh2h.H2HError) as e:
        g.query(bad, y, mode)
    assert e.value.code == -1
    assert np.array_equal(g.query(x, y, mode), ref)
