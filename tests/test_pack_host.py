"""Antenna packing (hussar_gb300/core.py): the columns written for all poses at once are the
bytes of the C structures filled one by one, whatever the sequence holds."""
import ctypes

import numpy as np
import pytest

from hussar_gb300 import FFAntenna, NFAntenna, _lib, core, scenes


class Tilted(NFAntenna):
    """A user's own antenna: its to_c() decides what the device gets."""

    def to_c(self):
        a = super().to_c()
        a.position[1] += 2.0
        return a


def nf(n):
    return scenes.plane_poses(n, n + 1)


def ff(n):
    d = np.array([0.6, 0.0, 0.8])
    return [FFAntenna(d, [0.1j * k, 1 + 2j, -0.075j * k], [k, 2, 3], 0.5 + k) for k in range(n)]


def structs(antennas, struct, count):
    return bytes((struct * count)(*[a.to_c() for a in antennas]))


@pytest.mark.parametrize("n", [0, 1, 2, 91])
def test_bytes_equal_the_structures(n):
    assert core._antenna_array(nf(n), n).tobytes() == structs(nf(n), _lib.AntennaC, n)
    assert core._ff_antenna_array(ff(n), n).tobytes() == structs(ff(n), _lib.FfAntennaC, n)
    mixed = nf(n) + [Tilted((1, 2, 3), np.eye(3)[[1, 2, 0]])]
    assert core._antenna_array(tuple(mixed), n + 1).tobytes() == structs(mixed, _lib.AntennaC, n + 1)


def test_other_lengths():
    """A shorter sequence leaves zeros, a longer one is refused, as a ctypes array does."""
    assert core._antenna_array(nf(2), 3).tobytes() == structs(nf(2), _lib.AntennaC, 3)
    with pytest.raises(IndexError):
        structs(nf(3), _lib.AntennaC, 2)
    with pytest.raises(IndexError):
        core._antenna_array(nf(3), 2)
    assert core._antenna_array(nf(2), 2).shape[1] * 4 == ctypes.sizeof(_lib.AntennaC)
