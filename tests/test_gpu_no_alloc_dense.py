"""The allocation-free entry point has no neighbourhood lists: on a dense scene its default launch
shape has to be the one that suits the tree."""
import ctypes
import time

import pytest

from hussar_gb300 import PathTracer, _lib, gb300, scenes

pytestmark = pytest.mark.gpu


def test_default_shape_suits_the_tree(product_lib):
    """The default against the 384-entry stack asked for: with the 512-entry one it took 1.2
    times as long here."""
    torch = pytest.importorskip("torch")
    P, N = 24, 256
    be = gb300.Backend(scenes.boxes_mesh(11, 83334, 100.0), None)
    t = PathTracer()
    t.doGuiding, t.maxDepth = False, 4
    poses = scenes.plane_poses(P, 3, 12.0)
    raw = bytes((_lib.AntennaC * P)(*[a.to_c() for a in poses]))
    d_ant = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()
    d_budget = torch.full((P,), 1 << 15, dtype=torch.int64, device="cuda")
    d_offset = torch.zeros(P, dtype=torch.int64, device="cuda")
    d_rows = torch.zeros(2 * P * N, device="cuda")
    rf, fl = scenes.rf_77ghz(N, 5e6)[0].to_c(), t.flags_c()
    ptr = lambda x: ctypes.c_void_p(x.data_ptr())

    def once():
        torch.cuda.synchronize()
        start = time.perf_counter()
        _lib.check(product_lib.hsr_simulate_batch_device_noalloc(
            be.handle, ctypes.byref(rf), N, ctypes.byref(fl), P, ptr(d_ant), ptr(d_ant), ptr(d_budget), ptr(d_offset),
            _lib.HSR_PHASE_SPLIT_FP64, ptr(d_rows), None))
        torch.cuda.synchronize()
        return time.perf_counter() - start

    best = {0: 1e9, 128: 1e9}
    for _ in range(12):
        for threshold in best:
            be.set_launch_config(queue_threshold=threshold)
            best[threshold] = min(best[threshold], once(), once())
    assert best[0] < 1.08 * best[128], best
