"""Batches over device buffers: rows written over the poses and budgets they come from, and
buffers at odd addresses, give what separate buffers give."""
import ctypes

import numpy as np
import pytest

from hussar_gb300 import PathTracer, _lib, gb300, scenes

pytestmark = pytest.mark.gpu

N = 256


def setup(poses, guided=False):
    torch = pytest.importorskip("torch")
    t = PathTracer()
    t.doGuiding, t.maxDepth = guided, 2
    w = scenes.dihedral_workload(poses=poses)
    ants = bytes((_lib.AntennaC * poses)(*[a.to_c() for a in w.tx]))
    budget = (100 + 7 * np.arange(poses) % 91).astype(np.int64)
    parts = [ants, ants, budget.tobytes(), np.zeros(poses, np.int64).tobytes()]
    return torch, w, t, gb300.Backend(w.mesh, None), parts


def place(torch, parts, at, size):
    """One buffer of `size` bytes with the parts at the byte offsets `at`; their addresses."""
    raw = np.zeros(size, np.uint8)
    for p, k in zip(parts, at):
        raw[k: k + len(p)] = np.frombuffer(p, np.uint8)
    buf = torch.from_numpy(raw).cuda()
    return buf, [buf.data_ptr() + k for k in at]


def rows(product_lib, torch, w, t, be, poses, addresses, out, graph):
    modes = (_lib.HSR_PHASE_REFERENCE_FP32, _lib.HSR_SPLAT_DIRICHLET16)
    torch.cuda.synchronize()
    if graph:
        g = be.batch_graph(w.rf, N, t, poses, *addresses, out, *modes)
        g.launch(None)
        g.status()
    else:
        _lib.check(product_lib.hsr_simulate_batch_device(
            be.handle, ctypes.byref(w.rf.to_c()), N, ctypes.byref(t.flags_c()), poses,
            *[ctypes.c_void_p(a) for a in addresses], *modes, ctypes.c_void_p(out), None))
    torch.cuda.synchronize()


def close(a, b):
    for x, y in zip(a, b):
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)


@pytest.mark.parametrize("graph", [False, True], ids=["call", "graph"])
def test_rows_over_the_budgets(product_lib, graph):
    """The budgets lie where the first rows are written, and there are more rows than the chip
    normalises at once."""
    P = 6000
    torch, w, t, be, parts = setup(P)
    want = be.simulate_batch(w.rf, N, t, w.tx, w.rx, np.frombuffer(parts[2], np.int64))
    size = 8 * P * N
    buf, at = place(torch, parts, [size, size + 48 * P, 0, size + 96 * P], size + 104 * P)
    rows(product_lib, torch, w, t, be, P, at, buf.data_ptr(), graph)
    close(buf[:size].cpu().numpy().view(np.complex64).reshape(P, N), want)


@pytest.mark.parametrize("guided", [False, True], ids=["plain", "guided"])
@pytest.mark.parametrize("off", [1, 2, 4])
def test_any_byte_address(product_lib, off, guided):
    """Antennas, budgets and offsets packed one after the other from an odd address."""
    P = 5
    torch, w, t, be, parts = setup(P, guided)
    want = be.simulate_batch(w.rf, N, t, w.tx, w.rx, np.frombuffer(parts[2], np.int64))
    buf, at = place(torch, parts, [off, off + 48 * P, off + 96 * P, off + 104 * P], 112 * P + 64)
    out = torch.zeros((P, N, 2), device="cuda")
    for graph in (False,) if guided else (False, True):
        out.zero_()
        rows(product_lib, torch, w, t, be, P, at, out.data_ptr(), graph)
        close(out.cpu().numpy().view(np.complex64)[..., 0], want)
