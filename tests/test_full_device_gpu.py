"""Calls that find no room on the device report it and leave what they worked
on as it was."""
import numpy as np
import pytest

from device_room import device_room

pytestmark = pytest.mark.gpu


def _road(root, n, H):
    import gpuh2h
    gpuh2h.generate_road(str(root), "r", n=n, target_arcs=int(n * 2.776), partition_height=H, seed=3)
    return gpuh2h.files_for(str(root), "r")


def test_policy_without_room_keeps_the_tasks(tmp_path):
    """The task tables of a policy that cuts every block finely take 12 MB here."""
    import gpuh2h
    g = gpuh2h.Graph("r", 9, 2, 2, 1, files=_road(tmp_path, 70000, 9))
    b = gpuh2h.Batch([g])
    want, policy, info = g.labels()["dis"], b.policy(), b.info()
    b.rebuild()
    fine = " ".join(["0/64/32"] * 12)
    with device_room(6 << 20):
        with pytest.raises(gpuh2h.H2HError) as e:
            b.set_policy(fine)
        assert e.value.code == -6
        assert b.policy() == policy and b.info()["fill_tiles"] == info["fill_tiles"]
    b.rebuild()
    assert np.array_equal(g.labels()["dis"], want)
    with device_room(6 << 20):
        assert b.tune(1) == b.policy()  # candidates without room are passed over
    b.rebuild()
    assert np.array_equal(g.labels()["dis"], want)
    b.set_policy(fine)
    b.rebuild()
    assert b.policy() == fine and b.info()["fill_tiles"] > info["fill_tiles"]
    assert np.array_equal(g.labels()["dis"], want)
    b.close()
    g.close()


@pytest.mark.parametrize("room_mb", (100, 220, 400))
def test_failed_batch_leaves_loaded_graphs(tmp_path, room_mb):
    """The batch fails in its elimination, with its lists made but not their
    weights, and at its label rows."""
    import gpuh2h
    files = _road(tmp_path, 70000, 9)
    ref = gpuh2h.Graph("r", 9, 2, 2, 1, files=files).contraction_noHub(1).constructLabel_noHub()
    want, adj = ref.labels()["dis"], ref.adj()
    ref.close()
    gs = [gpuh2h.Graph("r", 9, 2, 2, 1, files=files) for _ in range(2)]
    with device_room(room_mb << 20):
        with pytest.raises(gpuh2h.H2HError) as e:
            gpuh2h.Batch(gs)
        assert e.value.code == -6
    for g in gs:
        for call in (g.order, g.adj, g.constructLabel_noHub):
            with pytest.raises(gpuh2h.H2HError) as e:
                call()
            assert e.value.code == -4
        assert g.info()["pos_size"] == 0 and g.info()["device_bytes"] == 0
    gs[0].contraction_noHub(1)
    assert all(np.array_equal(a, b) for a, b in zip(gs[0].adj(), adj))
    gs[0].constructLabel_noHub()
    assert np.array_equal(gs[0].labels()["dis"], want)
    b = gpuh2h.Batch(gs[1:])
    assert np.array_equal(gs[1].labels()["dis"], want)
    b.close()
    for g in gs:
        g.close()


def test_weights_leave_room_for_labels(tmp_path):
    """A single build's highest use is 1.54 GB here, 1.69 when what only the weights
    need stays until the labels are filled."""
    import gpuh2h
    gpuh2h.generate_road(str(tmp_path), "r", n=264346, target_arcs=int(264346 * 2.776), aspect_milli=1300,
                         jitter_milli=300, diag_permille=50, hw_tiers=1, hw_permille10=50, hw_k=3, hw_scale_milli=400,
                         partition_height=11, seed=5, cols=0, drop_permille=0)
    files = gpuh2h.files_for(str(tmp_path), "r")
    gpuh2h.Graph("r", 11, 2, 8, 1, files=files).contraction_noHub(1).constructLabel_noHub().close()
    with device_room(1600 << 20):
        g = gpuh2h.Graph("r", 11, 2, 8, 1, files=files).contraction_noHub(1).constructLabel_noHub()
    assert g.info()["label_size"] > 0
    g.close()


@pytest.mark.parametrize("batch", (False, True))
def test_triangles_without_room_use_the_list_kernels(tmp_path, monkeypatch, capfd, batch):
    """The update triangles of a clique take 64 MB, its lists 9."""
    import gpuh2h
    from small_graphs import clique, write
    n, edges = clique(1500)
    files = write(tmp_path, n, [(u, v, w, w) for u, v, w in edges], 1)

    def build():
        b = gpuh2h.Batch([g]) if batch else g.contraction_noHub(1).constructLabel_noHub()
        out = [g.order(), *g.adj(), g.labels()["dis"]]
        if batch:
            b.rebuild()
            assert np.array_equal(g.labels()["dis"], out[-1])
            b.close()
        return out

    g = gpuh2h.Graph("g", 1, 1, 2, 1, files=files)
    want = build()
    g.close()
    g = gpuh2h.Graph("g", 1, 1, 2, 1, files=files)
    monkeypatch.setenv("GPUH2H_TRACE", "1")
    capfd.readouterr()
    with device_room((180 if batch else 150) << 20):
        got = build()
    err = capfd.readouterr().err
    assert "elim bits heap" in err and "elim heap" in err
    assert all(np.array_equal(a, b) for a, b in zip(want, got))
    g.close()


def test_labels_after_a_fill_without_room(tmp_path):
    """A label fill of either kind that finds no room can be followed by either."""
    import gpuh2h
    files = _road(tmp_path, 70000, 9)
    want = {}
    for mode in (gpuh2h.LABEL_L3, gpuh2h.LABEL_L4):
        ref = gpuh2h.Graph("r", 9, 2, 2, 1, files=files).contraction_noHub(1).constructLabel_noHub(2, 1, mode)
        want[mode] = ref.labels()["dis"]
        ref.close()
    for modes in ((3, 4), (4, 4), (4, 3), (3, 3), (3, 4, 3)):
        g = gpuh2h.Graph("r", 9, 2, 2, 1, files=files).contraction_noHub(1)
        adj = g.adj()
        with device_room(20 << 20):
            for mode in modes[:-1]:
                with pytest.raises(gpuh2h.H2HError) as e:
                    g.constructLabel_noHub(2, 1, mode)
                assert e.value.code == -6
        g.constructLabel_noHub(2, 1, modes[-1])
        assert np.array_equal(g.labels()["dis"], want[modes[-1]])
        assert all(np.array_equal(a, b) for a, b in zip(g.adj(), adj))
        g.close()
