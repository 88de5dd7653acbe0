"""Ray queries refuse fewer directions or limits than origins before the device sees them."""
import numpy as np
import pytest

from hussar_gb300 import HsrError, gb300


@pytest.mark.parametrize("n, directions, limits", [(3, 2, 3), (3, 3, 2), (1, 1, 0), (2, 2, 1), (5, 1, 5)])
def test_short_arrays(product_lib, n, directions, limits):
    be = gb300.Backend.__new__(gb300.Backend)  # no scene: what passes the check fails in the library
    be._scene = None
    o, d, far = np.zeros((n, 3)), np.ones((directions, 3)), np.ones(limits)
    for query in (be.intersect, be.visible):
        with pytest.raises(ValueError, match="%d origins" % n):
            query(o, d, far)
        with pytest.raises(HsrError):
            query(o[:1], np.ones((1, 3)), np.ones(1))
        with pytest.raises(HsrError):  # longer arrays are read as far as the origins go
            query(o, np.ones((n + 1, 3)), np.ones(n + 2))
