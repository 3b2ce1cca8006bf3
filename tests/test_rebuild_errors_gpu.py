"""A rebuild whose block weights did not finish says so: the fill that follows
them in the captured graph must not clear their error word.  The limits lie
far below the time the weights of this graph take (0.1 ms), so a block's wait
for the blocks below it runs out; every wait is bounded and the kernels
return."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit_ms", ("0.01", "0.03"))
def test_unfinished_weights_are_reported(tmp_path, monkeypatch, limit_ms):
    import gpuh2h
    gpuh2h.generate_road(str(tmp_path), "r", n=4096, target_arcs=11370, partition_height=4, seed=3)
    g = gpuh2h.Graph("r", 4, 2, 2, 1, files=gpuh2h.files_for(str(tmp_path), "r"))
    b = gpuh2h.Batch([g])
    want = g.labels()["dis"]
    monkeypatch.setenv("GPUH2H_SPIN_LIMIT_MS", limit_ms)  # read when the rebuild is captured
    with pytest.raises(gpuh2h.H2HError, match="block weights"):
        b.rebuild()
    monkeypatch.delenv("GPUH2H_SPIN_LIMIT_MS")
    b.set_policy(b.policy())  # the next rebuild is captured anew
    b.rebuild()
    assert np.array_equal(g.labels()["dis"], want)
    b.close()
    g.close()
