"""The guiding step (k_guide_step) on trees at the edges of its level-by-level passes,
against the oracle's walk: new topology, links and probabilities equal bit for bit."""
import numpy as np
import pytest

from hussar_gb300 import gb300, scenes

pytestmark = pytest.mark.gpu
MAX = 2048


def grow(rng, leaves_to_split, pick):
    """A tree grown by splitting leaves: child links (children follow their parent)."""
    child, depth = [-1], [0]
    for _ in range(leaves_to_split):
        open_ = [i for i, c in enumerate(child) if c < 0 and depth[i] < 24]
        if not open_ or len(child) + 2 > MAX:
            break
        i = pick(rng, open_, depth)
        child[i] = len(child)
        child += [-1, -1]
        depth += [depth[i] + 1] * 2
    return child


def any_leaf(rng, open_, depth):
    return open_[rng.integers(len(open_))]


def deepest(rng, open_, depth):
    return max(open_, key=lambda i: depth[i])


def chains(rng, open_, depth):
    """64 chains below a complete tree of depth 6: more nodes split than a tree holds."""
    shallow = [i for i in open_ if depth[i] < 6]
    return shallow[0] if shallow else min((i for i in open_ if i % 2 or depth[i] == 6), key=lambda i: depth[i])


CASES = {
    "root": (0, any_leaf, "even"), "two leaves, one empty": (1, any_leaf, "sparse"),
    "random": (300, any_leaf, "even"), "random, mostly empty": (300, any_leaf, "sparse"),
    "random, heavy-tailed": (500, any_leaf, "heavy"), "to the depth limit": (24, deepest, "heavy"),
    "full": (1023, any_leaf, "heavy"), "more than fits": (959, chains, "chains"), "no information": (100, any_leaf, "none"),
}


@pytest.mark.parametrize("name", CASES)
def test_step_equals_the_oracle(product_lib, oracle_lib, name):
    count, pick, kind = CASES[name]
    rng = np.random.default_rng(sum(map(ord, name)))
    be = gb300.Backend(scenes.dihedral_mesh(), None)
    for trial in range(3):
        child = grow(rng, count, pick)
        n = len(child)
        tc, acc = np.full(MAX, -1, np.int32), np.zeros(MAX, np.float32)
        tc[:n] = child
        leaf = tc[:n] < 0
        if kind == "even":
            acc[:n] = rng.uniform(0.5, 1, n)
        elif kind == "sparse":
            acc[:n] = rng.uniform(0.5, 1, n) * (rng.random(n) < 0.1)
            acc[n - 1] = 1
        elif kind == "heavy":
            acc[:n] = np.exp(rng.normal(0, 6, n))
        elif kind == "chains":
            depth = np.zeros(n, int)
            for i in range(n):
                if child[i] >= 0:
                    depth[child[i]] = depth[child[i] + 1] = depth[i] + 1
            # energy sqrt(acc 2^-depth): the chains' ends carry all of it, equally
            acc[:n] = (depth == depth.max()) * 2.0 ** depth * rng.uniform(0.9, 1.1, n)
        acc[:n] *= leaf
        g = gb300.Guide(be)
        g.write(n, np.full(MAX, -1, np.int32), np.full(MAX, 0.5, np.float32), tc, acc)
        og = oracle_lib.Guide()
        og.set(oracle_lib.GuideState(*g.read()))
        g.step()
        og.step()
        got, want = oracle_lib.GuideState(*g.read()), og.get()
        assert got.count == want.count
        if name == "more than fits":
            assert got.count >= MAX - 1
        m = got.count
        np.testing.assert_array_equal(got.train_child[:m], want.train_child[:m])
        np.testing.assert_array_equal(got.samp_child[:n], want.samp_child[:n])
        assert got.samp_p[:n].tobytes() == want.samp_p[:n].tobytes()
        assert not got.acc2[:m].any()
