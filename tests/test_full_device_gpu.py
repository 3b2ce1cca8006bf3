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
