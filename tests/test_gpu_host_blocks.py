"""A scene's host blocks (poses, guided schedule, rows): calls of growing and shrinking size,
rows below and above the size that the device writes to host memory itself (256 KB), plain,
fine-histogram, guided, far-field and interrupted ones in turn on one scene give what each
gives on a scene of its own. Sums are FP64 in any order and rounded to FP32 once: 1e-6
relative L2; the synthesis and the guiding trees add in FP32: 2e-5."""
import numpy as np
import pytest

from hussar_gb300 import FFAntenna, FrameConfig, PathTracer, Scene, _lib, gb300, scenes

pytestmark = pytest.mark.gpu

# (poses, bins, mode): 64 rows of 512 bins are 256 KB without the status word before them
CALLS = [(1, 64, "plain"), (63, 512, "plain"), (64, 512, "plain"), (2, 100, "plain"), (1, 128, "interrupted"),
         (5, 128, "guided"), (64, 512, "fine"), (1, 33, "guided"), (64, 512, "guided"), (1, 64, "interrupted"),
         (7, 96, "ff"), (2, 64, "fine"), (1, 64, "plain")]


def run(be, poses, n, mode):
    t = PathTracer()
    t.doGuiding = mode in ("guided", "interrupted")
    rf, _ = scenes.rf_77ghz(n, 5e6)
    ants = scenes.plane_poses(poses, poses + 1, 30.0)
    budget = [1 << (14 if t.doGuiding else 10)] * poses
    if mode == "interrupted":  # returns with the poses staged and nothing traced
        t.configureFrame(FrameConfig(1, n, 1))
        be._integrator = t
        with pytest.raises(RuntimeError):
            t.run(be, Scene(rf, ants[0], ants[0]), budget[0], interruptFlag=True)
        return None
    if mode == "ff":
        ff = [FFAntenna([0.6, 0.0, 0.8], [0.1 * k, 1, -0.075 * k], [0, 0, 3], 0.5 + k) for k in range(poses)]
        return be.simulate_batch_ff(rf, n, t, ff, ff, budget)
    splat = _lib.HSR_SPLAT_FINE_SYNTH if mode == "fine" else _lib.HSR_SPLAT_DIRICHLET16
    return be.simulate_batch(rf, n, t, ants, ants, budget, splat_mode=splat)


def test_calls_in_turn_equal_calls_alone(product_lib):
    mesh = scenes.boxes_mesh(11, 60, 30.0)
    one = gb300.Backend(mesh, None)
    for poses, n, mode in CALLS:
        got = run(one, poses, n, mode)
        if mode == "interrupted":
            continue
        ref = run(gb300.Backend(mesh, None), poses, n, mode)
        assert np.isfinite(ref).all() and np.linalg.norm(ref) > 0
        bound = 1e-6 if mode in ("plain", "ff") else 2e-5
        assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref), (poses, n, mode)
