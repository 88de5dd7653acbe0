"""Ray queries walk the tree with a warp's lanes in step: every answer equals, bit for bit, the
one the same ray gets alone in a call, and the oracle's. Rays from everywhere, parallel to
the axes, with limits, with no number in them; counts around a warp and a block."""
import numpy as np
import pytest

from hussar_gb300 import gb300, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(product_lib, oracle_lib):
    mesh = scenes.boxes_mesh(21, 1500, 30.0)
    return gb300.Backend(mesh, None), oracle_lib.Scene(mesh)


def rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-40, 40, (n, 3)) * [1, 0.2, 1]
    d = rng.normal(size=(n, 3))
    d[::7, 0] = 0
    d[::11] = np.eye(3)[rng.integers(0, 3, len(d[::11]))] * rng.choice([-1, 1], (len(d[::11]), 1))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    far = np.where(rng.random(n) < 0.3, rng.uniform(0, 5, n), np.inf)
    return o.astype(np.float32), d.astype(np.float32), far.astype(np.float32)


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 20000])
def test_answers_equal_the_oracle(setup, n):
    be, ora = setup
    o, d, far = rays(n, n)
    got, want = be.intersect(o, d, far), ora.intersect(o, d, far)
    np.testing.assert_array_equal(got[3], want[3])
    hit = got[3] >= 0
    np.testing.assert_array_equal(got[0][hit], np.asarray(want[0])[hit])
    np.testing.assert_array_equal(be.visible(o, d, far), ora.visible(o, d, far))


def test_lanes_do_not_touch_each_other(setup):
    """Rays with no number in them among others: each ray as if it were alone."""
    be, _ = setup
    o, d, far = rays(300, 5)
    o[5::29] = np.nan
    o[6::29, 1] = np.inf
    d[7::29] = np.nan
    far[8::29] = 0
    together = [*be.intersect(o, d, far), be.visible(o, d, far)]
    for k in range(300):
        s = slice(k, k + 1)
        for x, y in zip(together, [*be.intersect(o[s], d[s], far[s]), be.visible(o[s], d[s], far[s])]):
            assert x[s].tobytes() == y.tobytes(), k
