"""Guided calls on one scene, one after the other, over device buffers and over host arrays, also
right after a call that was interrupted: each plans its schedule in the scene's host memory,
and each gets its own rows."""
import ctypes

import numpy as np
import pytest

from hussar_gb300 import FrameConfig, HsrError, PathTracer, Scene, _lib, gb300, scenes

pytestmark = pytest.mark.gpu

N = 256


def test_calls_in_a_row(product_lib):
    torch = pytest.importorskip("torch")
    w = scenes.dihedral_workload(poses=40)
    t = PathTracer()
    t.maxDepth = 2
    t.configureFrame(FrameConfig(1, N, 1))
    be = gb300.Backend(w.mesh, t)
    rf, fl = w.rf.to_c(), t.flags_c()
    vp = lambda x: ctypes.c_void_p(x.data_ptr())

    def device_rows(lo, hi, budget, splat):
        P = hi - lo
        ants = (_lib.AntennaC * P)(*[a.to_c() for a in w.tx[lo:hi]])
        d_ant = torch.frombuffer(bytearray(bytes(ants)), dtype=torch.uint8).cuda()
        d_b, d_o = torch.from_numpy(budget).cuda(), torch.zeros(P, dtype=torch.int64, device="cuda")
        out = torch.full((P, N, 2), float("nan"), device="cuda")
        torch.cuda.synchronize()
        _lib.check(product_lib.hsr_simulate_batch_device(
            be.handle, ctypes.byref(rf), N, ctypes.byref(fl), P, vp(d_ant), vp(d_ant), vp(d_b), vp(d_o),
            _lib.HSR_PHASE_REFERENCE_FP32, splat, vp(out), None))
        torch.cuda.synchronize()
        return out.cpu().numpy().view(np.complex64)[..., 0]

    rng = np.random.default_rng(1)
    for lo, hi in ((0, 40), (3, 5), (1, 30), (7, 8), (0, 40)):
        # the first iteration is 2^14 samples: one iteration, without training, for every pose
        budget = rng.integers(1, 1 << 14, hi - lo).astype(np.int64)
        for splat in (_lib.HSR_SPLAT_DIRICHLET16, _lib.HSR_SPLAT_FINE_SYNTH):
            with pytest.raises(HsrError):
                t.run(be, Scene(w.rf, w.tx[0], w.rx[0]), 1 << 16, interruptFlag=lambda: True)
            got = device_rows(lo, hi, budget, splat)
            want = be.simulate_batch(w.rf, N, t, w.tx[lo:hi], w.rx[lo:hi], budget, splat_mode=splat)
            again = device_rows(lo, hi, budget, splat)
            for a, b, c in zip(got, again, want):
                assert np.linalg.norm(a - c) <= 1e-5 * np.linalg.norm(c)
                assert np.linalg.norm(b - c) <= 1e-5 * np.linalg.norm(c)
