"""Antenna packing takes and refuses what a C structure filled for each antenna does."""
import numpy as np
import pytest

from hussar_gb300 import FFAntenna, core, scenes


def ff(n):
    return [FFAntenna([0.6, 0.0, 0.8], [0, 1 + 0.5j * k, 0], [k, 2, 3], 0.5 + k) for k in range(n)]


@pytest.mark.parametrize("wrap", [iter, lambda a: (x for x in a), lambda a: dict.fromkeys(a).keys(),
                                  lambda a: np.array(a, object)], ids=["iterator", "generator", "keys", "array"])
def test_any_iterable(wrap):
    nf, far = scenes.plane_poses(5, 1), ff(5)
    assert core._antenna_array(wrap(nf), 5).tobytes() == core._antenna_array(nf, 5).tobytes()
    assert core._ff_antenna_array(wrap(far), 5).tobytes() == core._ff_antenna_array(far, 5).tobytes()
    with pytest.raises(IndexError):
        core._antenna_array(wrap(nf), 4)


@pytest.mark.parametrize("field", ["direction", "polarization", "scene_center"])
def test_vectors_of_another_length_are_refused(field):
    """Two antennas whose lengths are off by opposite amounts fill as many floats as two good ones."""
    far = ff(4)
    setattr(far[1], field, getattr(far[1], field)[:2])
    setattr(far[2], field, np.concatenate([getattr(far[2], field), getattr(far[2], field)[:1]]))
    with pytest.raises(ValueError):
        core._ff_antenna_array(far, 4)


def test_vectors_as_lists():
    far = ff(4)
    want = core._ff_antenna_array(far, 4).tobytes()
    for a in far[1:3]:
        a.direction, a.scene_center = a.direction.tolist(), a.scene_center.tolist()
    assert core._ff_antenna_array(far, 4).tobytes() == want
