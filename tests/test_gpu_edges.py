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


@pytest.fixture
def single_path():
    mg.set_dropin_batch_limit(0)
    yield
    mg.set_dropin_batch_limit()


# the pass loop's runs of triangles, vertices and candidates per block and its sort's tiles of 512:
# fewer than one of each, exactly one, one more, several per block; the last is above the size where
# two blocks per SM run it (pruning calls are not tuned, so the size decides)
@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (5, 5), (17, 17), (18, 17), (14, 26), (33, 65), (91, 90), (301, 299), (421, 410)])
@pytest.mark.parametrize("options", [0, mg.SimplifyPrune | mg.SimplifyLockBorder])
def test_pass_loop_sizes(port, single_path, nx, ny, options):
    if nx > 300 and not options & mg.SimplifyPrune:
        pytest.skip("the two sizes are there for the untuned calls")
    a = (np.arange(ny - 1)[:, None] * nx + np.arange(nx - 1)[None, :]).reshape(-1)
    idx = np.stack([a, a + 1, a + nx, a + nx, a + 1, a + nx + 1], 1).reshape(-1).astype(np.uint32)
    rng = np.random.default_rng(nx * 1000 + ny)
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    pos = np.stack([x, y, 0.4 * rng.standard_normal((ny, nx))], -1).reshape(-1, 3).astype(np.float32)
    for ratio, error in ((0.0, 1.0), (0.3, 2e-2)):
        target = W.target_count(len(idx), ratio)
        ref, ref_err = port.simplify("port", idx, pos, target, error, options)
        for device_loop in (True, False):
            mg.set_device_loop(device_loop)
            try:
                out, err = mg.simplify(idx, pos, target, error, options)
            finally:
                mg.set_device_loop(True)
            assert np.array_equal(out, ref)
            assert err == ref_err


@pytest.mark.parametrize("amp", [0.0, 1e-4])
def test_pass_loop_equal_keys(port, single_path, amp):
    """All candidates in a few sort bins: long runs of equal keys across the sorting blocks."""
    idx, pos = W.heightfield(49, seed=2, amp=amp)
    target = W.target_count(len(idx), 0.2)
    ref, ref_err = port.simplify("port", idx, pos, target, 1e-1, mg.SimplifyPrune)
    out, err = mg.simplify(idx, pos, target, 1e-1, mg.SimplifyPrune)
    assert np.array_equal(out, ref)
    assert err == ref_err


def _meshlet_groups(case):
    """Groups of the sphere's triangles in file order and the parameters they are cut with."""
    idx, pos, _, _ = W.octa_sphere(6, seed=9)
    tri = idx.reshape(-1, 3)
    if case == "frontier":  # whole strips: frontiers beyond the 128 slots kept in shared memory
        h, p = W.heightfield(120, seed=3, amp=0.02)
        return [h[: 3 * 6000], h], p, (256, 100, 512, 0.0, 2.0)
    if case == "ties":  # a flat lattice: scores and distances tie
        h, p = W.heightfield(33, seed=3, amp=0.0)
        return [h, h[::-1].copy()], p, (64, 16, 64, 0.0, 1.0)
    if case == "islands":  # separate triangles: every step asks for the nearest one
        pick = tri[np.random.default_rng(3).permutation(len(tri))[:1100]].reshape(-1)
        return [pick, pick[: 3 * 33], pick[: 3 * 31]], pos, (64, 8, 64, 0.5, 0.0)
    if case == "doubled":  # each triangle twice, and some that name a vertex twice
        t = tri[:300].copy()
        t[::7, 1] = t[::7, 0]
        return [np.repeat(t, 2, axis=0).reshape(-1)], pos, (96, 20, 96, 0.25, 2.0)
    if case == "hubs":  # one vertex with hundreds of triangles; more vertices than 3 per 4 triangles
        n = 700
        p = np.stack([np.cos(np.arange(n + 1)), np.sin(np.arange(n + 1)), 0.1 * np.cos(3.0 * np.arange(n + 1))], 1).astype(np.float32)
        fan = np.stack([np.full(n - 1, n), np.arange(n - 1), np.arange(1, n)], 1).astype(np.uint32).reshape(-1)
        loose = np.arange(699, dtype=np.uint32)
        return [fan, loose], p, (64, 16, 126, 0.0, 2.0)
    # "sizes": around the warp, the 128-triangle meshlet, the table and the largest group kept in shared memory
    cuts = [1, 31, 32, 33, 127, 128, 129, 340, 342, 511, 513, 1023, 1700, 4095, 4097]
    return [tri[: n].reshape(-1) for n in cuts], pos, (128, 42, 128, 0.0, 2.0)


@pytest.mark.parametrize("level", [-1, 0, 1, 9])
@pytest.mark.parametrize("case", ["frontier", "ties", "islands", "doubled", "hubs", "sizes"])
def test_meshlet_edges(case, level):
    import meshlets as ML

    groups, pos, params = _meshlet_groups(case)
    got = mg.build_meshlets_flex_groups(groups, pos, *params, optimize_level=level)
    for g, idx in enumerate(groups):
        m, v, t = ML.build_meshlets_flex(idx, pos, *params, kind="port")
        if level >= 0:
            v, t = ML.optimize_meshlets(m, v, t, level, kind="port")
        for a, b in zip(got[g], (m, v, t)):
            assert np.array_equal(a, b), f"group {g}"


def test_meshlets_wide_group():
    """One group of more corners than 16-bit ids hold."""
    import meshlets as ML

    idx, pos = W.heightfield(107, seed=5, amp=0.05)
    assert len(idx) > 65535
    (m, v, t), = mg.build_meshlets_flex_groups([idx], pos, 128, 42, 128, 0.0, 2.0, optimize_level=1)
    rm, rv, rt = ML.build_meshlets_flex(idx, pos, 128, 42, 128, 0.0, 2.0, kind="port")
    rv, rt = ML.optimize_meshlets(rm, rv, rt, 1, kind="port")
    assert np.array_equal(m, rm) and np.array_equal(v, rv) and np.array_equal(t, rt)


@pytest.mark.parametrize("size,shift", [(1, 0), (3, 1), (4, 0), (6, 2), (8, 8), (8, 4), (12, 0), (16, 0), (16, 8), (20, 4), (48, 0), (132, 0), (256, 0), (256, 1)])
@pytest.mark.parametrize("corners", [3, 1023, 1026, 8190])
def test_compaction_units(port, size, shift, corners):
    """Vertex sizes and alignments of every copy width, index counts around a tile of 1024."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(size * 100 + corners + shift)
    vc = corners // 2 + 5
    idx = rng.integers(0, vc, corners).astype(np.uint32)
    verts = rng.integers(0, 256, (vc, size)).astype(np.uint8)
    ref_idx, ref_verts, n = port.optimize_vertex_fetch("port", idx, verts)
    ref_remap, _ = port.optimize_vertex_fetch_remap("port", idx, vc)
    src = torch.zeros(vc * size + 64, dtype=torch.uint8, device="cuda")
    src[shift:shift + vc * size] = torch.from_numpy(verts.reshape(-1)).cuda()
    for in_place in (False, True):
        di = torch.from_numpy(idx.view(np.int32).copy()).cuda()
        s = src.clone()
        d = s if in_place else torch.full_like(s, 7)
        remap = torch.zeros(vc, dtype=torch.int32, device="cuda")
        assert mg.optimize_vertex_fetch_remap_device(remap.data_ptr(), di.data_ptr(), corners, vc) == n
        assert np.array_equal(remap.cpu().numpy().view(np.uint32), ref_remap)
        assert mg.optimize_vertex_fetch_device(d.data_ptr() + shift, di.data_ptr(), corners, s.data_ptr() + shift, vc, size) == n
        assert np.array_equal(di.cpu().numpy().view(np.uint32), ref_idx)
        got = d.cpu().numpy()
        assert np.array_equal(got[shift:shift + n * size].reshape(n, size), np.asarray(ref_verts).view(np.uint8).reshape(-1, size)[:n])
        # nothing outside the used rows
        keep = (s if in_place else torch.full_like(s, 7)).cpu().numpy() if not in_place else src.cpu().numpy()
        assert np.array_equal(got[:shift], keep[:shift]) and np.array_equal(got[shift + n * size:], keep[shift + n * size:])


def test_compaction_bad_index_changes_nothing():
    torch = pytest.importorskip("torch")
    idx = np.arange(3000, dtype=np.int32) % 700
    idx[2999] = 700
    di = torch.from_numpy(idx.copy()).cuda()
    src = torch.arange(700 * 16, dtype=torch.int32, device="cuda").to(torch.uint8)
    d = torch.full_like(src, 9)
    with pytest.raises(mg.SimplifyError) as e:
        mg.optimize_vertex_fetch_device(d.data_ptr(), di.data_ptr(), 3000, src.data_ptr(), 700, 16)
    assert e.value.status == mg.STATUS_INVALID_ARGUMENT
    assert np.array_equal(di.cpu().numpy(), idx) and bool((d == 9).all())


def _grid(nx, ny, amp, seed):
    a = (np.arange(ny - 1)[:, None] * nx + np.arange(nx - 1)[None, :]).reshape(-1)
    idx = np.stack([a, a + 1, a + nx, a + nx, a + 1, a + nx + 1], 1).reshape(-1).astype(np.uint32)
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    z = amp * np.random.default_rng(seed).standard_normal((ny, nx))
    return idx, np.stack([x, y, z], -1).reshape(-1, 3).astype(np.float32)


def _batch_same(port, ms, threads, smem_kb):
    mg.set_batch_config(threads, smem_kb * 1024)
    try:
        res = mg.simplify_batch(ms)
    finally:
        mg.set_batch_config(0)
    for i, (m, (out, err)) in enumerate(zip(ms, res)):
        ref, ref_err = port.simplify("port", m["indices"], m["positions"], m["target"], m["error"], m.get("options", 0),
                                     attributes=m.get("attributes"), weights=m.get("weights"), lock=m.get("lock"))
        assert np.array_equal(out, ref), f"mesh {i}"
        assert err == ref_err, f"mesh {i}"


SHAPES = [(128, 54), (256, 110), (512, 216), (256, 2)]


@pytest.mark.parametrize("threads,smem_kb", SHAPES)
@pytest.mark.parametrize("amp", [0.0, 1e-3, 0.3])
def test_batch_decision_windows(port, threads, smem_kb, amp):
    """Passes whose expected window is just below, at and above the one that a warp walks (224: a goal of
    160 or 161 triangles), flat meshes (more candidates of one sort key than are ranked in place), and
    passes that run out of candidates or reach the error limit in the middle of a window."""
    ms = []
    for nx, ny in ((2, 2), (4, 3), (9, 9), (17, 17), (14, 26)):
        idx, pos = _grid(nx, ny, amp, nx)
        tris = len(idx) // 3
        for removed in (31, 32, 33, 158, 159, 160, 161, 162, 163, 164, tris):
            if removed <= tris:
                for error in (1.0, 1e-2):
                    ms.append(dict(indices=idx, positions=pos, target=3 * (tris - removed), error=error, options=mg.SimplifyErrorAbsolute))
    _batch_same(port, ms, threads, smem_kb)


@pytest.mark.parametrize("threads,smem_kb", SHAPES)
@pytest.mark.parametrize("count", [1, 8, 9])
def test_batch_attribute_rows(port, threads, smem_kb, count):
    """Attribute gradients summed in registers (up to eight, where there is room) and in place."""
    rng = np.random.default_rng(count)
    ms = []
    for nx, ny in ((5, 4), (17, 17), (24, 20)):
        idx, pos = _grid(nx, ny, 0.1, nx)
        ms.append(dict(indices=idx, positions=pos, attributes=rng.standard_normal((len(pos), count)).astype(np.float32),
                       weights=rng.uniform(0.1, 1.0, count).astype(np.float32), target=len(idx) // 12 * 3, error=1.0))
    _batch_same(port, ms, threads, smem_kb)


@pytest.mark.parametrize("threads,smem_kb", SHAPES)
def test_batch_beyond_estimate(port, threads, smem_kb):
    """Meshes that need more vertices or candidates than the launch's shared memory was sized for, so that
    they start there and go on in the slab: a sparse subset of separate triangles (three vertices for each)
    and of fans, next to ordinary ones."""
    rng = np.random.default_rng(9)
    shared = rng.uniform(0, 1, (6000, 3)).astype(np.float32)
    idx, pos = _grid(17, 17, 0.1, 3)
    ms = [dict(indices=idx, positions=pos, target=300, error=1.0)]
    for tris in (64, 300, 700, 1024):
        soup = rng.permutation(6000)[: 3 * tris].astype(np.uint32)
        fan = np.stack([np.zeros(tris, np.int64), np.arange(1, tris + 1), np.arange(2, tris + 2)], 1).reshape(-1).astype(np.uint32)
        for i in (soup, fan):
            ms.append(dict(indices=i, positions=shared, target=0, error=1.0, options=mg.SimplifySparse))
            ms.append(dict(indices=i, positions=shared, target=len(i) // 6 * 3, error=1.0, options=mg.SimplifySparse | mg.SimplifyPermissive))
    _batch_same(port, ms, threads, smem_kb)


@pytest.mark.parametrize("indices,vertices", [(60000, 10201), (60003, 10201), (59994, 24000), (59994, 24001)])
def test_batch_id_width(port, indices, vertices):
    """The largest meshes with 16-bit ids and the smallest with 32-bit ones, by indices and by vertices."""
    idx, pos = _grid(101, 101, 0.2, 1)
    idx = np.concatenate([idx, idx[: max(0, indices - len(idx))]])[:indices]
    pos = np.concatenate([pos, np.random.default_rng(2).uniform(0, 100, (vertices - len(pos), 3)).astype(np.float32)])
    ms = [dict(indices=idx, positions=pos, target=W.target_count(len(idx), 0.5), error=1e-1)]
    small, sp = _grid(9, 9, 0.2, 1)
    ms.append(dict(indices=small, positions=sp, target=30, error=1.0))
    _batch_same(port, ms, 512, 110)


@pytest.mark.parametrize("factor", ["0.01", "0.3", "60"])
def test_pass_loop_windows(port, single_path, monkeypatch, factor):
    """Passes decided in many windows, in a few, and in one that takes every candidate, next to the predicted
    one of the other tests. The factor is read where a thread's state is made, so each case has a thread."""
    from concurrent.futures import ThreadPoolExecutor

    monkeypatch.setenv("MESHOPTGPU_WINDOW_FACTOR", factor)
    for nx, ny, amp, ratio, error in ((17, 17, 0.2, 0.2, 1.0), (120, 90, 0.0, 0.3, 1.0), (301, 299, 0.4, 0.1, 1.0), (301, 299, 0.4, 0.0, 1e-3)):
        idx, pos = _grid(nx, ny, amp, nx)
        target = W.target_count(len(idx), ratio)
        ref, ref_err = port.simplify("port", idx, pos, target, error, mg.SimplifyPrune)
        with ThreadPoolExecutor(1) as pool:
            out, err = pool.submit(mg.simplify, idx, pos, target, error, mg.SimplifyPrune).result()
        assert np.array_equal(out, ref)
        assert err == ref_err


@pytest.mark.parametrize("sizes", [(1022, 1024, 1026), (2046, 2048, 2050, 4), (6000, 510), (4,) * 300, (2050,) + (4,) * 40], ids=lambda s: f"{len(s)}x{s[0]}")
def test_prune_component_blocks(port, sizes):
    """Component radii around the block's tile of 1,024 vertices (512 and more per component on average), and
    many small components with one warp each, also with a large one among them."""
    idx, pos = _strips(sizes, len(sizes))
    opt = mg.SimplifyPrune | mg.SimplifyLockBorder
    for target in (0, W.target_count(len(idx), 0.5)):
        for error in (1e-2, 1e-1, 1.0):
            ref, ref_err = port.simplify("port", idx, pos, target, error, opt)
            out, err = mg.simplify(idx, pos, target, error, opt)
            assert np.array_equal(out, ref)
            assert err == ref_err


@pytest.mark.parametrize("budget", [16 << 10, 64 << 10, 1 << 20])
def test_server_small_budget(port, budget):
    """Meshes that run in shared memory are taken however small the memory budget, one after another."""
    torch = pytest.importorskip("torch")
    idx, pos = _grid(17, 17, 0.1, 3)
    di, dp = torch.from_numpy(idx.view(np.int32)).cuda(), torch.from_numpy(pos).cuda()
    outs = [torch.empty(len(idx), dtype=torch.int32, device="cuda") for _ in range(20)]
    torch.cuda.synchronize()
    ref, ref_err = port.simplify("port", idx, pos, 300, 1.0, 0)
    with mg.Server(memory_budget=budget) as srv:
        tickets = [srv.submit(di.data_ptr(), len(idx), dp.data_ptr(), len(pos), 300, 1.0, 0, o.data_ptr()) for o in outs]
        for t, o in zip(tickets, outs):
            status, n, err, _ = srv.wait(t)
            assert status == 0
            assert np.array_equal(o[:n].cpu().numpy().view(np.uint32), ref)
            assert err == ref_err


@pytest.mark.parametrize("ratio", [0.99, 0.9, 0.5])
def test_first_window_of_a_plane(port, single_path, ratio):
    """All errors are zero: the first pass decides about as many candidates as it has triangles to remove,
    not all of them."""
    idx, pos = _grid(257, 257, 0.0, 1)
    target = W.target_count(len(idx), ratio)
    ref, ref_err = port.simplify("port", idx, pos, target, 1e-2, 0)
    for _ in range(2):  # the first call of a size class may time launch shapes
        out, err = mg.simplify(idx, pos, target, 1e-2, 0)
    assert np.array_equal(out, ref)
    assert err == ref_err
    goal = (len(idx) - target) // 3
    assert mg.last_round_trace()[0][0] <= min(2 * goal + 4096, mg.last_pass_stats()[0]["candidates"])


@pytest.mark.parametrize("sizes", [(510,) + (4,) * 400, (512,) + (4,) * 400, (4,) * 400 + (514, 4, 4000), (600,) * 40 + (4,) * 700, (4,) * 127], ids=lambda s: f"{len(s)}x{max(s)}")
def test_prune_wide_among_small(port, sizes):
    """Large components among many small ones: each is measured by the block its own size asks for."""
    idx, pos = _strips(sizes, len(sizes))
    opt = mg.SimplifyPrune | mg.SimplifyLockBorder
    for target in (0, W.target_count(len(idx), 0.5)):
        for error in (1e-2, 1e-1):
            ref, ref_err = port.simplify("port", idx, pos, target, error, opt)
            out, err = mg.simplify(idx, pos, target, error, opt)
            assert np.array_equal(out, ref)
            assert err == ref_err


def test_prune_large_component_among_specks():
    """A body's radius takes about as long with thousands of specks around it as alone."""
    torch = pytest.importorskip("torch")
    idx, pos = _grid(300, 300, 0.05, 3)
    speck = np.array([0, 1, 2, 2, 1, 3])
    corner = np.array([[0, 0, 0], [0.1, 0, 0], [0, 0.1, 0], [0.1, 0.1, 0]])
    times = {}
    for count in (0, 3000):
        si = (np.arange(count)[:, None] * 4 + speck[None]).reshape(-1) + len(pos)
        sp = (np.random.default_rng(3).random((count, 1, 3)) * 300 + corner[None]).reshape(-1, 3)
        di = torch.from_numpy(np.concatenate([idx, si]).astype(np.uint32).view(np.int32)).cuda()
        dp = torch.from_numpy(np.concatenate([pos, sp]).astype(np.float32)).cuda()
        out = torch.empty_like(di)

        def call():
            mg.simplify_device(out.data_ptr(), di.data_ptr(), len(di), dp.data_ptr(), len(dp), 12, len(idx) // 12 * 3, 1e-2,
                               mg.SimplifyPrune | mg.SimplifyLockBorder)

        call()
        mg.set_kernel_profile("kMeasure")
        for _ in range(5):
            call()
        times[count] = mg.kernel_profile()[1]
        mg.set_kernel_profile(None)
    assert times[3000] < 1.3 * times[0], times


@pytest.mark.parametrize("corners", [608 * 1024 * 2 + 3, 608 * 1024 * 16 + 1023, 608 * 1024 * 17 + 1026])
def test_compaction_many_tiles(corners):
    """Several tiles per block of the vertex order, around the 16 whose first uses a block keeps."""
    torch = pytest.importorskip("torch")
    corners = corners // 3 * 3
    vc = 500_003
    g = torch.Generator(device="cuda").manual_seed(corners)
    di = torch.randint(0, vc, (corners,), generator=g, dtype=torch.int32, device="cuda")
    src = torch.arange(vc, dtype=torch.int32, device="cuda")
    # the first position of every vertex, and its rank among them
    first = torch.full((vc,), corners, dtype=torch.int64, device="cuda").scatter_reduce_(0, di.long(), torch.arange(corners, device="cuda"), "amin")
    used = first < corners
    want = torch.full((vc,), -1, dtype=torch.int32, device="cuda")
    want[torch.argsort(first)[: int(used.sum())]] = torch.arange(int(used.sum()), dtype=torch.int32, device="cuda")
    remap = torch.zeros(vc, dtype=torch.int32, device="cuda")
    assert mg.optimize_vertex_fetch_remap_device(remap.data_ptr(), di.data_ptr(), corners, vc) == int(used.sum())
    assert torch.equal(remap, want)
    dst, new = torch.full_like(src, -7), di.clone()
    assert mg.optimize_vertex_fetch_device(dst.data_ptr(), new.data_ptr(), corners, src.data_ptr(), vc, 4) == int(used.sum())
    assert torch.equal(new, want[di.long()])
    assert torch.equal(dst[: int(used.sum())], torch.argsort(first)[: int(used.sum())].int()) and bool((dst[int(used.sum()):] == -7).all())


def test_small_mesh_takes_no_longer(single_path):
    """A mesh of 128 triangles on the single-mesh path against one of 2,048: a pass has work that does not
    shrink with the mesh, which more than one block shares."""
    torch = pytest.importorskip("torch")
    times = {}
    for nx in (9, 33):
        idx, pos = _grid(nx, nx, 0.05, 3)
        di, dp = torch.from_numpy(idx.view(np.int32)).cuda(), torch.from_numpy(pos).cuda()
        out = torch.empty_like(di)

        def call():
            mg.simplify_device(out.data_ptr(), di.data_ptr(), len(di), dp.data_ptr(), len(dp), 12, len(idx) // 12 * 3, 1e-2, 0)

        call()
        call()
        mg.set_kernel_profile("kPassLoop")
        for _ in range(5):
            call()
        times[nx] = mg.kernel_profile()[1] / 5
        mg.set_kernel_profile(None)
    assert times[9] < 1.15 * times[33], times
