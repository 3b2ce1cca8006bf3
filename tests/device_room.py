"""Takes the device's free memory but for a few bytes, so that the allocations
of a call fail as they do on a full device."""
import contextlib
import ctypes


@contextlib.contextmanager
def device_room(leave):
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cu = ctypes.CDLL("libcuda.so.1")
    free, total, p = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_uint64()
    assert cu.cuMemGetInfo_v2(ctypes.byref(free), ctypes.byref(total)) == 0
    want = (free.value - leave) & ~((2 << 20) - 1)
    while want > 0 and cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(want)) != 0:
        want -= 2 << 20
    assert want > 0
    try:
        yield
    finally:
        assert cu.cuMemFree_v2(p) == 0
