"""Host batches and server requests in buffers that a kernel must not use in
place: page-locked but not aligned to an int, and page-locked in part only.
They are copied or staged, as pageable ones are, with the same answers."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 9000  # above the sizes that are staged anyway


@pytest.fixture(scope="module")
def graph(tmp_path_factory):
    import gpuh2h
    root = str(tmp_path_factory.mktemp("spans"))
    gpuh2h.generate_road(root, "r", n=4096, target_arcs=11370, partition_height=4, seed=3)
    g = gpuh2h.Graph("r", 4, 2, 2, 1, files=gpuh2h.files_for(root, "r"))
    g.contraction_noHub(1).constructLabel_noHub()
    x, y = gpuh2h.uniform_pairs(4096, N, 5)
    yield g, x, y, g.query(x, y)
    g.close()


def _fill(address, a):
    ctypes.memmove(address, a.ctypes.data, a.nbytes)


def _read(address):
    a = np.empty(N, np.int32)
    ctypes.memmove(a.ctypes.data, address, a.nbytes)
    return a


def _serve(g, px, py, pout):
    import gpuh2h
    srv = gpuh2h.Server(slots=2, slot_pairs=6000)
    gid, rid = srv.add(g), ctypes.c_uint64()
    assert srv._L.h2h_server_submit(srv.s, gid, px, py, pout, N, 0, ctypes.byref(rid)) == 0
    srv.wait(rid.value)
    srv.release(rid.value)
    srv.close()


@pytest.mark.parametrize("which", range(4))  # x, y, out, or all of them off by two bytes
def test_page_locked_but_unaligned(graph, which):
    import torch
    g, x, y, want = graph
    for serve in (False, True):
        hold = [torch.zeros(4 * N + 16, dtype=torch.uint8).pin_memory() for _ in range(3)]
        px, py, pout = (t.data_ptr() + (2 if which in (k, 3) else 0) for k, t in enumerate(hold))
        _fill(px, x)
        _fill(py, y)
        if serve:
            _serve(g, px, py, pout)
        else:
            g.query_host_ptr(px, py, pout, N)
        assert np.array_equal(_read(pout), want)


def test_page_locked_in_part(graph):
    import torch
    g, x, y, want = graph
    page = 65536
    rt = torch.cuda.cudart()
    hold = [np.zeros(4 * N + 3 * page, np.uint8) for _ in range(3)]
    base = [(a.ctypes.data + page - 1) // page * page for a in hold]
    for p in base:
        assert int(rt.cudaHostRegister(p, page, 0)) == 0
    try:
        # the last 16 KB of the range, then ordinary memory
        px, py, pout = (p + page - 16384 for p in base)
        _fill(px, x)
        _fill(py, y)
        _serve(g, px, py, pout)
        assert np.array_equal(_read(pout), want)
        # a copy out of such a buffer is the runtime's to take or refuse
        import gpuh2h
        _fill(pout, np.zeros(N, np.int32))
        try:
            g.query_host_ptr(px, py, pout, N)
            assert np.array_equal(_read(pout), want)
        except gpuh2h.H2HError as e:
            assert e.code == -5
    finally:
        for p in base:
            rt.cudaHostUnregister(p)
    assert np.array_equal(g.query(x, y), want)  # a refused copy is no error of the next call


@pytest.mark.parametrize("which", range(3))
def test_small_batch_in_device_memory(graph, which):
    """Device memory given for host memory is the copies' to refuse, in small
    batches as in large ones; the library does not touch it from the host."""
    import gpuh2h
    import torch
    g, x, y, want = graph
    host = [np.ascontiguousarray(x[:100]), np.ascontiguousarray(y[:100]), np.zeros(100, np.int32)]
    p = [a.ctypes.data for a in host]
    on_device = torch.from_numpy(host[which]).cuda()
    p[which] = on_device.data_ptr()
    try:
        g.query_host_ptr(*p, 100)
        torch.cuda.synchronize()
        assert np.array_equal(on_device.cpu().numpy() if which == 2 else host[2], want[:100])
    except gpuh2h.H2HError as e:
        assert e.code == -5
    assert np.array_equal(g.query(x[:100], y[:100]), want[:100])
