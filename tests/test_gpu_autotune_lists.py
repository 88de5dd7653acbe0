"""On a scene with neighbourhood lists the autotuner chooses among what its launches obey: work
items, CTAs per SM and thresholds within their one path stack."""
import numpy as np
import pytest

from hussar_gb300 import PathTracer, gb300, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [64, 2048])
def test_only_what_has_an_effect(product_lib, bins):
    """A batch of a few items, whose times differ by more than a candidate has to win by: over
    many attempts a field without effect would be chosen by chance."""
    be = gb300.Backend(scenes.boxes_mesh(5, 4000, 20.0), None)
    t = PathTracer()
    t.doGuiding, t.maxDepth = False, 4
    poses = scenes.plane_poses(4, 3, 18.0)
    rf = scenes.rf_77ghz(bins, 5e6 * bins / 256)[0]
    seen = [be.autotune(rf, bins, t, poses, poses, np.full(4, 300)) for _ in range(60)]
    assert {s["queue_threshold"] for s in seen} <= {32, 64, 128}
    assert {s["field_on_hit"] for s in seen} == {0} and {s["coherent_order"] for s in seen} == {0}
