"""Kernels at the sizes and orders where they can go wrong (tile edges, remainders, index orders),
bit for bit against the oracle."""
import numpy as np
import pytest

import meshoptimizer_gb300 as mg
from meshoptimizer_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from meshoptimizer_gb300 import build

    build.build()
    mg.load()


def _same(a, b):
    return np.array_equal(np.asarray(a, np.float32).view(np.uint32), np.asarray(b, np.float32).view(np.uint32))


def _strips(sizes, seed):
    """One strip of two vertex rows per size (vertices rounded up to even), far apart, in one buffer."""
    rng = np.random.default_rng(seed)
    idx, pos, base = [], [], 0
    for k, n in enumerate(sizes):
        cols = max(2, (n + 1) // 2)
        a = np.arange(cols - 1)
        idx.append(np.stack([a, a + 1, a + cols, a + cols, a + 1, a + cols + 1], 1).reshape(-1) + base)
        p = np.stack([np.tile(np.arange(cols), 2) * 0.01, np.repeat([0.0, 0.02], cols), 0.01 * rng.standard_normal(2 * cols)], 1)
        pos.append(p + [0, k, 0])
        base += 2 * cols
    return np.concatenate(idx).astype(np.uint32), np.concatenate(pos).astype(np.float32)


@pytest.mark.parametrize("sizes", [(4, 6), (254, 256, 258), (510, 512, 514, 8), (1030, 34, 30)], ids=str)
def test_prune_component_tiles(port, sizes):
    """Component radii around the measuring kernel's tile of 256 vertices."""
    idx, pos = _strips(sizes, len(sizes))
    opt = mg.SimplifyPrune | mg.SimplifyLockBorder
    for target in (0, W.target_count(len(idx), 0.5)):
        for error in (1e-2, 1e-1, 1.0):
            ref, ref_err = port.simplify("port", idx, pos, target, error, opt)
            out, err = mg.simplify(idx, pos, target, error, opt)
            assert np.array_equal(out, ref)
            assert err == ref_err


@pytest.mark.parametrize("order", ["rows", "reversed", "shuffled"])
@pytest.mark.parametrize("amp,ratio", [(0.02, 1.0), (0.02, 0.4), (0.2, 0.6)])
def test_update_vertex_orders(port, order, amp, ratio):
    """The position solve depends on vertex order: long index-ordered chains, forwards and backwards, and none."""
    idx, pos = W.heightfield(67, seed=21, amp=amp)
    n = len(pos)
    new = {"rows": np.arange(n), "reversed": np.arange(n)[::-1], "shuffled": np.random.default_rng(4).permutation(n)}[order]
    p = np.empty_like(pos)
    p[new] = pos
    i = new[idx].astype(np.uint32)
    target = W.target_count(len(i), ratio)
    ref = port.simplify_with_update("port", i, p, target, 1.0, 0)
    got = mg.simplify_with_update(i, p, target, 1.0, 0)
    assert np.array_equal(got[0], ref[0])
    assert _same(got[1], ref[1])
    assert not _same(got[1], p)
