"""Ray queries on whatever arrays the caller has: at odd byte addresses, and with results
written over the inputs, the answers are those of separate, aligned arrays."""
import ctypes

import numpy as np
import pytest

from hussar_gb300 import _lib, gb300, scenes

pytestmark = pytest.mark.gpu

N = 1 << 20


@pytest.fixture(scope="module")
def setup(product_lib):
    be = gb300.Backend(scenes.boxes_mesh(21, 1500, 30.0), None)
    rng = np.random.default_rng(4)
    d = rng.normal(size=(N, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return be, rng.uniform(-15, 15, (N, 3)).astype(np.float32), d.astype(np.float32), \
        rng.uniform(0.5, 9.0, N).astype(np.float32)


def at_byte(a, off):
    """A copy of the array that starts `off` bytes past a 64-byte boundary."""
    raw = np.zeros(a.nbytes + 128, np.uint8)
    start = (-raw.ctypes.data) % 64 + off
    out = raw[start: start + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


@pytest.mark.parametrize("off", [1, 2, 3, 4])
def test_any_byte_address(setup, off):
    be, o, d, far = (x[:5000] if isinstance(x, np.ndarray) else x for x in setup)
    want, seen = be.intersect(o, d, far), be.visible(o, d, far)
    for k in range(3):
        args = [at_byte(x, off if j == k else 0) for j, x in enumerate((o, d, far))]
        for a, b in zip([*be.intersect(*args), be.visible(*args)], [*want, seen]):
            assert a.tobytes() == b.tobytes(), k
    # results at odd addresses too (the Python wrapper's own are aligned)
    out = [at_byte(np.zeros_like(x), off) for x in want]
    _lib.check(_lib.lib().hsr_intersect(be.handle, len(o), *[ctypes.c_void_p(x.ctypes.data) for x in (o, d, far, *out)]))
    for a, b in zip(out, want):
        assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("shift", [0, 1, N // 2])
def test_results_over_the_inputs(setup, shift):
    """Distances written over the limits, `shift` rays further on: every ray still has the
    limit that the call was given."""
    be, o, d, far = setup
    t, p, n, prim = be.intersect(o, d, far)
    buf = np.zeros(N + shift, np.float32)
    buf[:N] = far
    got = [np.zeros_like(x) for x in (p, n, prim)]
    _lib.check(_lib.lib().hsr_intersect(be.handle, N, *[ctypes.c_void_p(x) for x in
               (o.ctypes.data, d.ctypes.data, buf.ctypes.data, buf.ctypes.data + 4 * shift,
                *[x.ctypes.data for x in got])]))
    assert buf[shift: shift + N].tobytes() == t.tobytes()
    for a, b in zip(got, (p, n, prim)):
        assert a.tobytes() == b.tobytes()
