"""The batch kernel's forms and where meshes run: batches that need several, bit for bit against the oracle."""
import os
import subprocess
import sys

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


def _grid(nx, ny, amp, seed):
    a = (np.arange(ny - 1)[:, None] * nx + np.arange(nx - 1)[None, :]).reshape(-1)
    idx = np.stack([a, a + 1, a + nx, a + nx, a + 1, a + nx + 1], 1).reshape(-1).astype(np.uint32)
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    z = amp * np.random.default_rng(seed).standard_normal((ny, nx))
    return idx, np.stack([x, y, z], -1).reshape(-1, 3).astype(np.float32)


def _same(port, ms, res):
    seen = {}
    for i, (m, (out, err)) in enumerate(zip(ms, res)):
        key = (id(m["indices"]), id(m["positions"]), id(m.get("attributes")), m["target"], m["error"], m.get("options", 0))
        if key not in seen:
            seen[key] = port.simplify("port", m["indices"], m["positions"], m["target"], m["error"], m.get("options", 0),
                                      attributes=m.get("attributes"), weights=m.get("weights"), lock=m.get("lock"))
        ref, ref_err = seen[key]
        assert np.array_equal(out, ref), f"mesh {i}"
        assert err == ref_err, f"mesh {i}"


def _small(count, attributes=0, nx=13, ny=11):
    rng = np.random.default_rng(count + attributes)
    distinct = []
    for k in range(8):
        idx, pos = _grid(nx, ny, 0.1, k)
        m = dict(indices=idx, positions=pos, target=len(idx) // 6 * 3, error=1.0)
        if attributes:
            m.update(attributes=rng.standard_normal((len(pos), attributes)).astype(np.float32),
                     weights=rng.uniform(0.1, 1.0, attributes).astype(np.float32))
        distinct.append(m)
    return [distinct[i % 8] for i in range(count)]


@pytest.mark.parametrize("count,attributes", [(1, 0), (8, 3), (2000, 0), (700, 2)])
def test_batch_with_wide_meshes(port, count, attributes):
    """Small meshes stay in shared memory next to one of many indices and one over a large vertex buffer."""
    ms = _small(count, attributes)
    idx, pos = _grid(104, 101, 0.2, 3)
    assert len(idx) > 60000
    wide = [dict(indices=idx, positions=pos, target=len(idx) // 6 * 3, error=1.0)]
    few, fp = _grid(13, 11, 0.1, 0)
    far = np.concatenate([fp, np.random.default_rng(2).uniform(0, 100, (24100 - len(fp), 3)).astype(np.float32)])
    wide.append(dict(indices=few, positions=far, target=len(few) // 6 * 3, error=1.0))
    for at in (0, count // 2, count):  # wherever they stand in the batch
        batch = ms[:at] + wide + ms[at:]
        for _ in range(2):  # with the size class's trials and without
            res = mg.simplify_batch(batch)
            assert mg.last_batch_placement() == (count, 2)
        _same(port, batch, res)
    res = mg.simplify_batch(wide)
    assert mg.last_batch_placement() == (0, 2)
    _same(port, wide, res)


def test_tuned_per_form():
    """A batch with attributes is timed itself, also after a positions-only one of its size class (in a
    process of its own: what is timed is kept for the process)."""
    code = """
import sys
sys.path[:0] = [%r, %r]
import test_gpu_batch_forms as T
import meshoptimizer_gb300 as mg

def launches(ms):
    n = mg.launch_count()
    mg.simplify_batch(ms)
    return mg.launch_count() - n

lean, full = T._small(400), T._small(400, 3)
first, again, other, once = launches(lean), launches(lean), launches(full), launches(full)
assert first > 3 and again == 1 and other > 3 and once == 1, (first, again, other, once)
assert mg.tuning(len(lean[0]["indices"]))["batch_smem_kib"] in (54, 110, 216)
"""
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", code % (here, os.path.dirname(here))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("budget", [8 << 10, 16 << 10, 200 << 10, 4 << 20])
def test_server_budget_bounds_what_it_holds(port, budget):
    """Requests that shared memory holds whatever they need hold no slab where the budget has no room for
    one, and go on together; one that may need a slab larger than the budget is refused."""
    torch = pytest.importorskip("torch")
    idx, pos = _grid(17, 17, 0.1, 3)
    di, dp = torch.from_numpy(idx.view(np.int32)).cuda(), torch.from_numpy(pos).cuda()
    # a sparse group may use a vertex per index
    gi, gp = _grid(33, 33, 0.1, 5)
    ga = torch.zeros(len(gp) * 8, dtype=torch.float32, device="cuda")
    gd, gv = torch.from_numpy(gi.view(np.int32)).cuda(), torch.from_numpy(np.concatenate([gp] * 6)).cuda()
    outs = [torch.empty(max(len(idx), len(gi)), dtype=torch.int32, device="cuda") for _ in range(60)]
    torch.cuda.synchronize()
    ref, ref_err = port.simplify("port", idx, pos, 300, 1.0, 0)
    with mg.Server(memory_budget=budget) as srv:
        tickets = [srv.submit(di.data_ptr(), len(idx), dp.data_ptr(), len(pos), 300, 1.0, 0, o.data_ptr()) for o in outs]
        if budget < 1 << 20:
            with pytest.raises(mg.SimplifyError) as e:
                srv.submit(gd.data_ptr(), len(gi), gv.data_ptr(), len(gp) * 6, 300, 1.0, mg.SimplifySparse, outs[0].data_ptr(),
                           d_attributes=ga.data_ptr(), attr_stride=32, weights=np.ones(8, np.float32))
            assert e.value.status == mg.STATUS_OUT_OF_MEMORY
        for t, o in zip(tickets, outs):
            status, n, err, _ = srv.wait(t)
            assert status == 0
            assert np.array_equal(o[:n].cpu().numpy().view(np.uint32), ref)
            assert err == ref_err
        assert srv.stats()["peak_reserved"] <= budget


def _ribbon(tris, seed):
    return _grid(tris // 2 + 1, 2, 0.1, seed)


def _quads(count, seed):
    """Separate quads: every vertex is on a border."""
    p = np.random.default_rng(seed).random((count, 1, 3)) * 10 + np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0.1]])[None]
    idx = (np.arange(count)[:, None] * 4 + np.array([0, 1, 2, 2, 1, 3])[None]).reshape(-1)
    return idx.astype(np.uint32), p.reshape(-1, 3).astype(np.float32)


@pytest.mark.parametrize("tris", [2, 40, 128, 200])
def test_open_meshes_in_shared_memory(port, tris):
    """Meshes whose vertices are mostly on borders have a larger capacity than expected; after a batch of
    them, the next one's shared memory is sized for it."""
    for make in (_ribbon, lambda t, s: _quads(t // 2, s)):
        distinct = []
        for k in range(4):
            idx, pos = make(tris, k)
            distinct.append(dict(indices=idx, positions=pos, target=len(idx) // 6 * 3, error=1.0))
        ms = [distinct[i % 4] for i in range(600)]
        for _ in range(2):
            res = mg.simplify_batch(ms)
        assert mg.last_batch_placement() == (len(ms), 0)
        _same(port, ms, res)
    # and back: ordinary meshes of the same number of indices
    idx, pos = _grid(11, tris // 20 + 1, 0.1, 1)
    ms = [dict(indices=idx, positions=pos, target=len(idx) // 6 * 3, error=1.0)] * 600
    for _ in range(2):
        _same(port, ms, mg.simplify_batch(ms))


@pytest.mark.parametrize("attributes", [0, 2])
@pytest.mark.parametrize("tris", [20, 120, 240])
def test_unshared_sparse_groups_in_shared_memory(port, tris, attributes):
    """Sparse groups with three vertices per triangle (flat shaded): more than a surface's share of them. A
    process of its own, so that this kind is the first of its size class."""
    code = """
import sys
sys.path[:0] = [%r, %r, %r]
import numpy as np
import oracle
import test_gpu_batch_forms as T
import meshoptimizer_gb300 as mg

idx, pos = T._grid(11, %d // 20 + 1, 0.1, 1)
n, count, attributes = len(idx), 300, %d
flat = np.concatenate([pos[idx] + [20 * (i %% 8), 0, 0] for i in range(count)]).astype(np.float32)
at = np.random.default_rng(1).standard_normal((len(flat), max(attributes, 1))).astype(np.float32)
ms = []
for i in range(count):
    m = dict(indices=(np.arange(n) + n * i).astype(np.uint32), positions=flat, target=n // 6 * 3, error=1.0, options=mg.SimplifySparse)
    if attributes:
        m.update(attributes=at, weights=np.full(attributes, 0.3, np.float32))
    ms.append(m)
for _ in range(2):
    res = mg.simplify_batch(ms)
assert mg.last_batch_placement() == (count, 0), mg.last_batch_placement()
T._same(oracle, ms[:20], res[:20])
"""
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    r = subprocess.run([sys.executable, "-c", code % (here, root, os.path.join(root, "oracle"), tris, attributes)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def _stars(count):
    """A lattice of 1,682 triangles, and flat stars whose centres cannot move anywhere: ten candidates each of
    no error, all of whose flips are rejected before the lattice's candidates are looked at."""
    idx, pos = _grid(30, 30, 0.3, 1)
    a = np.arange(10) * np.pi / 5
    rad = np.where(np.arange(10) % 2, 0.15, 1.0)
    ring = np.concatenate([[[0, 0, 0]], np.stack([rad * np.cos(a), rad * np.sin(a), 0 * a], 1)])
    fan = np.stack([np.zeros(10, int), 1 + np.arange(10), 1 + (np.arange(10) + 1) % 10], 1).reshape(-1)
    centre = np.stack([np.arange(count) % 64 * 3.0, np.arange(count) // 64 * 3.0, np.full(count, 5.0)], 1)
    si = (np.arange(count)[:, None] * 11 + fan[None]).reshape(-1) + len(pos)
    sp = (centre[:, None] + ring[None]).reshape(-1, 3)
    return np.concatenate([idx, si]).astype(np.uint32), np.concatenate([pos, sp]).astype(np.float32)


@pytest.mark.parametrize("threads,smem_kb", [(128, 54), (256, 110), (512, 216)])
@pytest.mark.parametrize("count", [10, 22, 41, 42, 45, 60, 300])
def test_walks_that_hand_over(port, count, threads, smem_kb):
    """Passes that are walked in sorted order and end before, at and after the position where the rounds take
    over (448), with the stop rules' terms carried over."""
    idx, pos = _stars(count)
    opt = mg.SimplifyErrorAbsolute | mg.SimplifyLockBorder
    ms = [dict(indices=idx, positions=pos, target=len(idx) - 3 * goal, error=err, options=opt)
          for goal in (1, 10, 40, 100, 150, 160) for err in (1e9, 0.05)]
    mg.set_batch_config(threads, smem_kb * 1024)
    try:
        res = mg.simplify_batch(ms)
    finally:
        mg.set_batch_config(0)
    _same(port, ms, res)


def test_walk_costs_no_more_than_rounds():
    """15,000 rejected candidates before the first that counts, with a goal that is walked (100 triangles) and
    one that goes in rounds (200): the kernel's times are alike (a walk to the end took several times more)."""
    torch = pytest.importorskip("torch")
    idx, pos = _stars(1500)
    di, dp = torch.from_numpy(idx.view(np.int32)).cuda(), torch.from_numpy(pos).cuda()
    out = torch.empty_like(di)
    times = {}
    mg.set_batch_config(256, 110 * 1024)
    try:
        for goal in (100, 200):
            d = mg.BatchDescriptors([dict(d_indices=di.data_ptr(), index_count=len(idx), d_positions=dp.data_ptr(), vertex_count=len(pos),
                                          target=len(idx) - 3 * goal, error=1e9, options=mg.SimplifyErrorAbsolute | mg.SimplifyLockBorder,
                                          d_destination=out.data_ptr())])
            for _ in range(2):
                mg.simplify_batch_device(d)
            mg.set_kernel_profile("kBatch")
            for _ in range(5):
                mg.simplify_batch_device(d)
            n, ms = mg.kernel_profile()
            mg.set_kernel_profile(None)
            times[goal] = ms / n
    finally:
        mg.set_batch_config(0)
    assert times[100] < 1.25 * times[200], times


def _odd_values(kind, nx, ny, seed):
    """A lattice some of whose errors are not finite: attributes that are infinite, whose squares overflow or
    that are NaN, or positions that are NaN."""
    rng = np.random.default_rng(seed)
    idx, pos = _grid(nx, ny, 0.1, seed)
    attr = rng.standard_normal((len(pos), 3)).astype(np.float32)
    at = rng.permutation(len(pos))[: max(1, len(pos) // 9)]
    value = {"inf": np.inf, "huge": 1e25, "nan": np.nan, "mixed": np.nan, "nan_position": 0.0, "all_inf": np.inf}[kind]
    if kind == "nan_position":
        pos[at[: max(1, len(at) // 4)], 1] = np.nan
    elif kind == "all_inf":
        attr[:] = rng.choice([-np.inf, np.inf], attr.shape)
    else:
        attr[at, rng.integers(0, 3, len(at))] = value
        if kind == "mixed":
            attr[at[::2], 0], attr[at[1::3], 1] = np.inf, -1e25
    return dict(indices=idx, positions=pos, attributes=attr, weights=np.array([0.5, 1.0, 0.25], np.float32))


ODD = ["inf", "huge", "nan", "mixed", "nan_position", "all_inf"]


@pytest.mark.parametrize("threads,smem_kb", [(128, 54), (256, 110), (512, 216), (256, 2)])
@pytest.mark.parametrize("kind", ODD)
def test_odd_values_in_batches(port, kind, threads, smem_kb):
    """Infinite and NaN errors in the walk, the rounds, the stop rules and the sort."""
    ms = []
    for nx, ny in ((3, 3), (9, 8), (17, 17), (26, 23)):
        m = _odd_values(kind, nx, ny, nx)
        tris = len(m["indices"]) // 3
        for removed in sorted({1, tris // 4, min(150, tris // 2), tris // 2, tris}):
            for error in (1e-2, 3e38, np.inf):
                for opt in (0, mg.SimplifyErrorAbsolute):
                    ms.append(dict(m, target=3 * (tris - removed), error=error, options=opt))
    mg.set_batch_config(threads, smem_kb * 1024)
    try:
        res = mg.simplify_batch(ms)
    finally:
        mg.set_batch_config(0)
    for i, (m, (out, err)) in enumerate(zip(ms, res)):
        ref, ref_err = port.simplify("port", m["indices"], m["positions"], m["target"], m["error"], m["options"], attributes=m["attributes"],
                                     weights=m["weights"])
        assert np.array_equal(out, ref), f"mesh {i}"
        assert err == ref_err or (np.isnan(err) and np.isnan(ref_err)), f"mesh {i}"


@pytest.mark.parametrize("kind", ODD)
def test_odd_values_in_the_pass_loop(port, kind):
    """The same on the single-mesh path, whose first window is predicted from the errors."""
    mg.set_dropin_batch_limit(0)
    try:
        for nx, ny in ((9, 8), (40, 37), (120, 97)):
            m = _odd_values(kind, nx, ny, nx)
            tris = len(m["indices"]) // 3
            for removed in (tris // 50 + 1, tris // 2, tris):
                for error in (1e-2, np.inf):
                    for prune in (0, mg.SimplifyPrune):
                        if prune and kind == "nan_position":
                            continue
                        target = 3 * (tris - removed)
                        ref, ref_err = port.simplify("port", m["indices"], m["positions"], target, error, prune, attributes=m["attributes"],
                                                     weights=m["weights"])
                        out, err = mg.simplify(m["indices"], m["positions"], target, error, prune, attributes=m["attributes"], weights=m["weights"])
                        assert np.array_equal(out, ref)
                        assert err == ref_err or (np.isnan(err) and np.isnan(ref_err))
    finally:
        mg.set_dropin_batch_limit()


@pytest.mark.parametrize("call", ["device", "batch", "groups"])
def test_in_place_as_the_first_call(call):
    """Destinations may alias indices, also in the first call of a size class, whose shapes would be timed on
    its meshes (a process of its own)."""
    code = """
import sys
sys.path[:0] = [%r, %r, %r]
import numpy as np, torch
import oracle
import test_gpu_batch_forms as T
import meshoptimizer_gb300 as mg

call = %r
idx, pos = T._grid(17, 13, 0.1, 1)
target = len(idx) // 6 * 3
dp = torch.from_numpy(pos).cuda()
count = {"device": 1, "batch": 40, "groups": 40}[call]
d = torch.from_numpy(np.tile(idx.view(np.int32), count)).cuda()
opt = mg.SimplifySparse if call == "groups" else 0
if call == "device":
    n, err = mg.simplify_device(d.data_ptr(), d.data_ptr(), len(idx), dp.data_ptr(), len(pos), 12, target, 1.0)
    counts, errs = [n], [err]
elif call == "batch":
    at = [d.data_ptr() + 4 * len(idx) * i for i in range(count)]
    counts, errs = mg.simplify_batch_device([dict(d_indices=p, index_count=len(idx), d_positions=dp.data_ptr(), vertex_count=len(pos), target=target,
                                                  error=1.0, d_destination=p) for p in at])
else:
    # every group uses every position, so all are locked but for one group's: one group, many separate vertex copies
    posn = np.concatenate([pos + [0, 0, 50 * i] for i in range(count)]).astype(np.float32)
    ii = np.concatenate([idx + len(pos) * i for i in range(count)]).astype(np.uint32)
    d = torch.from_numpy(ii.view(np.int32)).cuda()
    dp = torch.from_numpy(posn).cuda()
    remap = torch.arange(len(posn), dtype=torch.int32, device="cuda")
    locks = torch.zeros(len(posn), dtype=torch.uint8, device="cuda")
    off = np.arange(count + 1) * len(idx)
    counts, errs = mg.simplify_groups_device(d.data_ptr(), d.data_ptr(), off, dp.data_ptr(), len(posn), 12, remap.data_ptr(), locks.data_ptr(),
                                             [target] * count, 1.0, 0)
got = d.cpu().numpy().view(np.uint32)
for i in range(count):
    p, base = (pos, 0) if call != "groups" else (posn[len(pos) * i:len(pos) * (i + 1)], len(pos) * i)
    ref, ref_err = oracle.simplify("port", idx, np.ascontiguousarray(p), target, 1.0, opt)
    out = got[len(idx) * i:len(idx) * i + int(counts[i])]
    assert np.array_equal(out, ref + np.uint32(base)), i
    assert errs[i] == np.float32(ref_err), i
"""
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    r = subprocess.run([sys.executable, "-c", code % (here, root, os.path.join(root, "oracle"), call)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("threads,smem_kb", [(128, 54), (512, 216), (256, 2)])
def test_windows_that_the_error_limit_ends(port, threads, smem_kb):
    """Passes with many triangles to remove that the error limit ends after none, a few (walked: up to 31) and
    more candidates, up to all of them, and limits of zero and infinity."""
    ms = []
    for nx, ny, amp in ((17, 17, 0.1), (26, 23, 0.02), (40, 21, 0.0)):
        idx, pos = _grid(nx, ny, amp, nx)
        attr = np.random.default_rng(nx).standard_normal((len(pos), 2)).astype(np.float32)
        for error in [0.0, np.inf] + [float(10.0 ** (-e / 6)) for e in range(6, 30)]:
            for extra in (dict(), dict(options=mg.SimplifyRegularize), dict(attributes=attr, weights=np.full(2, 0.1, np.float32))):
                ms.append(dict(dict(indices=idx, positions=pos, target=0, error=error), **extra))
    mg.set_batch_config(threads, smem_kb * 1024)
    try:
        res = mg.simplify_batch(ms)
    finally:
        mg.set_batch_config(0)
    _same(port, ms, res)
