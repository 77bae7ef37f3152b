"""Performance cases: the work that programs have this library do, through its public calls.

Meshes are seeded: lattice heightfields (white noise, or 6-octave value noise for terrain),
subdivided octahedron spheres and latitude/longitude globes with normals and UVs (the UV seam
split into duplicate vertices), small lattice patches of a displaced sphere, and scans made of
disconnected pieces. Sizes follow the benchmark's workloads, with ragged ones between them.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs, output buffers and handles, as a program holds them before the call
    run(state)            one pass; returns every output
    work(case)            bytes a pass cannot do without (inputs read once, outputs written once)
    exact(case, seed)     the outputs in plain torch where they have a value of their own, else None
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import meshoptimizer_gb300 as mg

FLT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # a prop's next level of detail, made through the drop-in call on host arrays: the smallest call
        dict(name="prop_host_510", kind="mesh", surface="globe", nx=17, ny=15, ratio=0.5, error=1e-2, options=0, host=True),
        # one streamed terrain tile, device resident, its border kept so that it meets its neighbours
        dict(name="tile_101x67", kind="mesh", surface="noise", nx=101, ny=67, ratio=0.3, error=1e-2, options=mg.SimplifyLockBorder, host=False),
        # the benchmark's heightfield: an ordinary asset without attributes
        dict(name="heightfield_256", kind="mesh", surface="noise", nx=256, ny=256, ratio=0.25, error=1e-2, options=0, host=False),
        # the benchmark's headline: a large asset with normals and UVs
        dict(name="sphere_attr_2m", kind="mesh", surface="octa", nx=9, ny=0, ratio=0.1, error=5e-3, options=0, host=False),
        # the benchmark's stress terrain: the largest single mesh
        dict(name="terrain_3163", kind="mesh", surface="fractal", nx=3163, ny=3163, ratio=0.01, error=5e-2, options=0, host=False),
        # a scan of disconnected pieces on host arrays, small pieces pruned: the drop-in call of an asset converter
        dict(name="scan_host_prune", kind="scan", parts=23, side=131, ratio=0.1, error=2e-2, options=mg.SimplifyPrune | mg.SimplifyLockBorder),
        # the benchmark's batch: 4,096 independent cluster groups of 200 to 512 triangles
        dict(name="groups_4096", kind="groups", count=4096, tmin=200, tmax=512, ratio=0.5, error=2e-2),
        # one level of a cluster-LOD build: locks between groups, then every group simplified to half
        dict(name="lod_level_2048", kind="level", levels=9, group_tris=1024),
        # the same build's second step: the simplified groups cut into meshlets
        dict(name="meshlets_2048", kind="meshlets", levels=9, group_tris=1024, max_vertices=128, min_triangles=42, max_triangles=128),
        # an asset whose vertices move to their best positions (simplifyWithUpdate), updated in place
        dict(name="update_globe_131k", kind="update", nx=367, ny=180, ratio=0.2, error=1e-2, options=mg.SimplifyRegularizeLight),
        # a burst of requests of mixed sizes at the request server
        dict(name="serve_burst_96", kind="serve", count=96, median=20000, tmax=1000000),
        # vertex buffer compaction after a simplification that kept a tenth of the triangles
        dict(name="compact_2m", kind="compact", nx=1449, ny=1449, keep=0.1, floats=8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "mesh", "mesh", "scan", "groups", "level", "meshlets", "update", "serve", "compact"])
    if kind == "mesh":
        tris, aspect = _log(rng, 500, 4e6), rng.uniform(0.5, 2.0)
        nx = max(8, int(math.sqrt(tris / 2 * aspect)) + rng.randrange(3))
        host = rng.random() < 0.3
        options = rng.choice([0, 0, mg.SimplifyLockBorder, mg.SimplifyErrorAbsolute, mg.SimplifyRegularize])
        return dict(kind="mesh", surface=rng.choice(["noise", "fractal", "globe"]), nx=nx, ny=max(8, int(tris / 2 / nx) + rng.randrange(3)),
                    ratio=round(rng.uniform(0.05, 0.6), 3), error=rng.choice([5e-3, 1e-2, 5e-2]), options=options, host=host)
    if kind == "scan":
        return dict(kind="scan", parts=rng.randrange(5, 40), side=int(_log(rng, 20, 180)), ratio=round(rng.uniform(0.05, 0.4), 3), error=2e-2,
                    options=mg.SimplifyPrune | rng.choice([0, mg.SimplifyLockBorder]))
    if kind == "groups":
        tmin = int(_log(rng, 60, 400))
        return dict(kind="groups", count=int(_log(rng, 50, 8000)), tmin=tmin, tmax=tmin + rng.randrange(20, 400), ratio=round(rng.uniform(0.3, 0.7), 3), error=2e-2)
    if kind in ("level", "meshlets"):
        case = dict(kind=kind, levels=rng.choice([6, 7, 8, 9]), group_tris=int(_log(rng, 250, 1500)))
        if kind == "meshlets":
            case.update(max_vertices=rng.choice([64, 96, 128, 192]), min_triangles=rng.randrange(16, 64), max_triangles=rng.choice([64, 126, 128]))
            case["min_triangles"] = min(case["min_triangles"], case["max_triangles"])
        return case
    if kind == "update":
        nx = int(_log(rng, 20, 900))
        return dict(kind="update", nx=nx, ny=max(8, int(nx * rng.uniform(0.4, 1.2))), ratio=round(rng.uniform(0.1, 0.5), 3), error=1e-2,
                    options=rng.choice([0, mg.SimplifyRegularizeLight]))
    if kind == "serve":
        return dict(kind="serve", count=int(_log(rng, 8, 128)), median=int(_log(rng, 3000, 30000)), tmax=rng.choice([60000, 400000, 1000000]))
    nx = int(_log(rng, 60, 1500))
    return dict(kind="compact", nx=nx, ny=max(8, int(nx * rng.uniform(0.5, 1.0))), keep=round(rng.uniform(0.02, 0.9), 3), floats=rng.choice([3, 5, 8, 12]))


# ------------------------------------------------------------------ meshes (torch, on the given device)

def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(seed * 7919 + 13)


def _target(index_count, ratio):
    return int(ratio * index_count / 3) * 3


@functools.lru_cache(maxsize=8)
def _lattice(nx, ny, dev):
    """Two triangles per quad of an ny x nx vertex lattice, row-major: int64 [tris, 3]."""
    a = (torch.arange(ny - 1, device=dev)[:, None] * nx + torch.arange(nx - 1, device=dev)[None, :]).reshape(-1)
    return torch.stack([a, a + 1, a + nx, a + nx, a + 1, a + nx + 1], 1).reshape(-1, 3)


def _height_positions(nx, ny, z, dev):
    step = 1.0 / (max(nx, ny) - 1)
    y, x = torch.meshgrid(torch.arange(ny, device=dev, dtype=torch.float64) * step, torch.arange(nx, device=dev, dtype=torch.float64) * step, indexing="ij")
    return torch.stack([x, y, z.to(torch.float64)], -1).reshape(-1, 3).to(torch.float32)


def _value_noise(nx, ny, gen, dev, octaves=6, cells=16):
    total, amp, norm = torch.zeros(ny, nx, dtype=torch.float64, device=dev), 1.0, 0.0
    step = 1.0 / (max(nx, ny) - 1)
    for _ in range(octaves):
        lat = torch.rand(cells + 1, cells + 1, generator=gen, device=dev, dtype=torch.float64) * 2 - 1

        def axis(n):
            f = torch.arange(n, device=dev, dtype=torch.float64) * (step * cells)
            i = f.to(torch.int64).clamp(max=cells - 1)
            s = f - i
            return i, s * s * (3 - 2 * s)

        (iy, sy), (ix, sx) = axis(ny), axis(nx)
        rows = lat[:, ix] + (lat[:, ix + 1] - lat[:, ix]) * sx
        total += amp * (rows[iy] + (rows[iy + 1] - rows[iy]) * sy[:, None])
        norm += amp
        amp *= 0.5
        cells *= 2
    return total / norm


@functools.lru_cache(maxsize=4)
def _octa(levels, dev):
    """Unit octahedron sphere of 8 * 4^levels triangles, its UV seam split: triangles, unit normals, UVs,
    and for each vertex the one whose position it shares."""
    v = torch.tensor([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], dtype=torch.float64, device=dev)
    t = torch.tensor([[0, 2, 4], [2, 1, 4], [1, 3, 4], [3, 0, 4], [2, 0, 5], [1, 2, 5], [3, 1, 5], [0, 3, 5]], dtype=torch.int64, device=dev)
    for _ in range(levels):
        e = torch.cat([t[:, [0, 1]], t[:, [1, 2]], t[:, [2, 0]]])
        key, inv = torch.unique(e.min(1).values * len(v) + e.max(1).values, return_inverse=True)
        mid = v[key // len(v)] + v[key % len(v)]
        m = inv.reshape(3, -1) + len(v)
        v = torch.cat([v, mid / mid.norm(dim=1, keepdim=True)])
        t = torch.stack([torch.stack([t[:, 0], m[0], m[2]], 1), torch.stack([m[0], t[:, 1], m[1]], 1), torch.stack([m[2], m[1], t[:, 2]], 1), m.T], 1).reshape(-1, 3)
    u = torch.atan2(v[:, 1], v[:, 0]) / (2 * math.pi) + 0.5
    w = torch.acos(v[:, 2].clamp(-1, 1)) / math.pi
    tu = u[t]
    fix = (tu.max(1).values - tu.min(1).values > 0.5)[:, None] & (tu > 0.5)
    src = torch.unique(t[fix])
    dup = torch.full((len(v),), -1, dtype=torch.int64, device=dev)
    dup[src] = len(v) + torch.arange(len(src), device=dev)
    t = torch.where(fix, dup[t], t)
    base = torch.cat([torch.arange(len(v), device=dev), src])
    return t, v[base], torch.cat([u, u[src] - 1]), w[base], base


def _octa_mesh(levels, gen, dev):
    t, n, u, w, base = _octa(levels, dev)
    r = 1 + 0.02 * torch.randn(len(n), generator=gen, device=dev, dtype=torch.float64)
    pos = (n * r[base][:, None]).to(torch.float32)
    return t, pos, torch.cat([n, u[:, None], w[:, None]], 1).to(torch.float32)


def _globe_mesh(nx, ny, gen, dev):
    """A globe without its polar caps, nx columns by ny rows of vertices; the last column repeats the
    first one's positions with u = 1 (the seam)."""
    phi = torch.arange(nx, device=dev, dtype=torch.float64) / (nx - 1)
    theta = (torch.arange(ny, device=dev, dtype=torch.float64) + 0.5) / ny
    r = 1 + 0.2 / max(nx, ny) * torch.randn(ny, nx, generator=gen, device=dev, dtype=torch.float64)
    r[:, -1] = r[:, 0]
    ang = 2 * math.pi * phi
    c, s = torch.cos(ang), torch.sin(ang)
    c[-1], s[-1] = c[0], s[0]
    st, ct = torch.sin(math.pi * theta)[:, None], torch.cos(math.pi * theta)[:, None]
    n = torch.stack([st * c, st * s, ct.expand(ny, nx)], -1)
    uv = torch.stack([phi[None, :].expand(ny, nx), theta[:, None].expand(ny, nx)], -1)
    attr = torch.cat([n, uv], -1).reshape(-1, 5).to(torch.float32)
    return _lattice(nx, ny, dev), (n * r[..., None]).reshape(-1, 3).to(torch.float32), attr


_WEIGHTS = np.array([0.5, 0.5, 0.5, 1.0, 1.0], dtype=np.float32)


def _mesh(case, gen, dev):
    """(triangles, positions, attributes or None)"""
    s, nx, ny = case["surface"], case["nx"], case["ny"]
    if s == "octa":
        return _octa_mesh(nx, gen, dev)
    if s == "globe":
        return _globe_mesh(nx, ny, gen, dev)
    if s == "fractal":
        return _lattice(nx, ny, dev), _height_positions(nx, ny, 0.05 * _value_noise(nx, ny, gen, dev), dev), None
    z = 0.05 * torch.randn(ny, nx, generator=gen, device=dev, dtype=torch.float64)
    return _lattice(nx, ny, dev), _height_positions(nx, ny, z, dev), None


def _indices(t):
    return t.reshape(-1).to(torch.int32).contiguous()


# ------------------------------------------------------------------ kinds

def _prepare_mesh(case, seed):
    dev = "cpu" if case["host"] else "cuda"
    t, pos, attr = _mesh(case, _gen(seed, dev), dev)
    idx = _indices(t)
    s = dict(case=case, target=_target(len(idx), case["ratio"]), weights=None if attr is None else _WEIGHTS)
    if case["host"]:
        s.update(idx=idx.numpy().view(np.uint32), pos=pos.numpy(), attr=None if attr is None else attr.numpy(), dst=np.zeros(len(idx), np.uint32))
    else:
        s.update(idx=idx, pos=pos, attr=attr, dst=torch.zeros_like(idx))
    return s


def _run_mesh(s):
    c = s["case"]
    if c["host"]:
        out, err = mg.simplify(s["idx"], s["pos"], s["target"], c["error"], c["options"], attributes=s["attr"], weights=s["weights"], destination=s["dst"])
        return [len(out), s["dst"].view(np.int32), err]
    a = s["attr"]
    n, err = mg.simplify_device(s["dst"].data_ptr(), s["idx"].data_ptr(), len(s["idx"]), s["pos"].data_ptr(), len(s["pos"]), 12, s["target"], c["error"],
                                c["options"], d_attributes=0 if a is None else a.data_ptr(), attributes_stride=0 if a is None else a.shape[1] * 4,
                                weights=s["weights"], stream=torch.cuda.current_stream().cuda_stream)
    return [n, s["dst"], err]


def _part_sizes(case):
    # a generator of its own: sizes belong to the case, the seed sets positions
    u = np.random.default_rng(case["parts"] * 1009 + case["side"]).uniform(0.05, 1.0, (case["parts"], 2))
    return np.maximum(3, (case["side"] * u).astype(np.int64))


def _prepare_scan(case, seed):
    rng = np.random.default_rng(seed + 101)
    idx, pos, base = [], [], 0
    for nx, ny in _part_sizes(case).tolist():
        t = _lattice(nx, ny, "cpu").numpy()
        y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
        v = np.stack([x, y, 1.0 * rng.standard_normal((ny, nx))], -1).reshape(-1, 3) * (0.6 / case["side"])
        idx.append(t.reshape(-1) + base)
        pos.append(v + rng.uniform(-2, 2, 3))
        base += len(v)
    idx = np.concatenate(idx).astype(np.uint32)
    return dict(case=case, idx=idx, pos=np.concatenate(pos).astype(np.float32), target=_target(len(idx), case["ratio"]), dst=np.zeros_like(idx))


def _run_scan(s):
    c = s["case"]
    out, err = mg.simplify(s["idx"], s["pos"], s["target"], c["error"], c["options"], destination=s["dst"])
    return [len(out), s["dst"].view(np.int32), err]


def _patch_sizes(case):
    # a generator of its own, as for the parts of a scan
    return np.random.default_rng(case["count"] * 31 + case["tmin"]).integers(case["tmin"], case["tmax"] + 1, case["count"])


def _prepare_groups(case, seed):
    rng = np.random.default_rng(seed + 7)
    sizes = _patch_sizes(case)
    quads = 14  # a patch: the first triangles of a strip 14 quads wide, bent onto a displaced sphere
    strip = _lattice(quads + 1, int(sizes.max()) // (2 * quads) + 2, "cpu").numpy()
    idx = [strip[:t].reshape(-1) for t in sizes]
    counts = [int(i.max()) + 1 for i in idx]
    where = rng.permutation(len(sizes))  # each patch has a place of its own on the sphere
    pos = []
    for g, n in enumerate(counts):
        k = np.arange(n)
        lon = 0.0245 * (k % (quads + 1)) + 0.35 * (where[g] % 18)
        lat = 0.0245 * (k // (quads + 1)) - 1.2 + 0.01 * (where[g] // 18 % 160)
        r = 1 + 0.02 * rng.standard_normal(n)
        pos.append(np.stack([r * np.cos(lat) * np.cos(lon), r * np.cos(lat) * np.sin(lon), r * np.sin(lat)], -1))
    di = torch.from_numpy(np.concatenate(idx).astype(np.int32)).cuda()
    dp = torch.from_numpy(np.concatenate(pos).astype(np.float32)).cuda()
    dst = torch.zeros_like(di)
    ib, pb, descs = 0, 0, []
    for i, n in zip(idx, counts):
        descs.append(dict(d_indices=di.data_ptr() + 4 * ib, index_count=len(i), d_positions=dp.data_ptr() + 12 * pb, vertex_count=n, stride=12,
                          target=_target(len(i), case["ratio"]), error=case["error"], options=mg.SimplifyLockBorder, d_destination=dst.data_ptr() + 4 * ib))
        ib, pb = ib + len(i), pb + n
    return dict(case=case, idx=di, pos=dp, dst=dst, batch=mg.BatchDescriptors(descs))


def _run_groups(s):
    counts, errs = mg.simplify_batch_device(s["batch"], stream=torch.cuda.current_stream().cuda_stream)
    return [counts.astype(np.int64), errs, s["dst"]]


def _prepare_level(case, seed):
    t, pos, attr = _octa_mesh(case["levels"], _gen(seed, "cuda"), "cuda")
    c = pos[t].to(torch.float64).mean(1)
    theta, phi = torch.acos((c[:, 2] / c.norm(dim=1)).clamp(-1, 1)), torch.atan2(c[:, 1], c[:, 0])
    bands = max(1, round(math.sqrt(len(t) / case["group_tris"])))
    band = (theta / math.pi * bands).to(torch.int64).clamp(max=bands - 1)
    idx = _indices(t[torch.argsort(band * 8.0 + phi, stable=True)])
    off = np.minimum(np.arange(0, len(idx) + 3 * case["group_tris"], 3 * case["group_tris"]), len(idx)).astype(np.uint64)
    off = off[: int(np.searchsorted(off, len(idx))) + 1]
    remap = torch.empty(len(pos), dtype=torch.int32, device="cuda")
    mg.generate_position_remap_device(remap.data_ptr(), pos.data_ptr(), len(pos), 12)
    # seams stay where attributes differ between vertices of one position
    locks = ((attr != attr[remap.long()]).any(1) * 2).to(torch.uint8)
    targets = (np.diff(off.astype(np.int64)) // 6 * 3).astype(np.uint64)
    return dict(case=case, idx=idx, pos=pos, attr=attr, off=off, remap=remap, locks=locks, targets=targets, dst=torch.zeros_like(idx))


def _run_level(s):
    counts, errs = mg.simplify_groups_device(s["dst"].data_ptr(), s["idx"].data_ptr(), s["off"], s["pos"].data_ptr(), len(s["pos"]), 12,
                                             s["remap"].data_ptr(), s["locks"].data_ptr(), s["targets"], FLT_MAX,
                                             mg.SimplifySparse | mg.SimplifyErrorAbsolute | mg.SimplifyPermissive, d_attributes=s["attr"].data_ptr(),
                                             attributes_stride=20, weights=_WEIGHTS, stream=torch.cuda.current_stream().cuda_stream)
    return [counts.astype(np.int64), errs, s["dst"], s["locks"]]


def _prepare_meshlets(case, seed):
    s = _prepare_level(case, seed)
    counts = _run_level(s)[0]
    off = s["off"].astype(np.int64)
    # the simplified groups, packed
    keep = np.zeros(len(s["idx"]), bool)
    start = np.zeros(len(keep) + 1, np.int64)
    np.add.at(start, off[:-1], 1)
    np.add.at(start, off[:-1] + counts, -1)
    keep[:] = np.cumsum(start)[:-1] > 0
    idx = s["dst"][torch.from_numpy(keep).cuda()].contiguous()
    soff = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    rows = mg.meshlet_rows(soff, case["max_vertices"], case["min_triangles"])
    return dict(case=case, idx=idx, pos=s["pos"], off=soff, rows=rows, meshlets=torch.zeros(int(rows[-1]), 4, dtype=torch.int32, device="cuda"),
                vertices=torch.zeros(len(idx), dtype=torch.int32, device="cuda"), triangles=torch.zeros(len(idx), dtype=torch.uint8, device="cuda"))


def _run_meshlets(s):
    c = s["case"]
    counts = mg.build_meshlets_flex_groups_device(s["meshlets"].data_ptr(), s["vertices"].data_ptr(), s["triangles"].data_ptr(), s["rows"], s["idx"].data_ptr(),
                                                  s["off"], s["pos"].data_ptr(), len(s["pos"]), 12, c["max_vertices"], c["min_triangles"], c["max_triangles"],
                                                  0.0, 2.0, optimize_level=1, stream=torch.cuda.current_stream().cuda_stream)
    return [counts.astype(np.int64), s["meshlets"], s["vertices"], s["triangles"]]


def _prepare_update(case, seed):
    t, pos, attr = _globe_mesh(case["nx"], case["ny"], _gen(seed, "cuda"), "cuda")
    idx = _indices(t)
    # some vertices are locked (rigged) or protected, most are free
    lock = torch.rand(len(pos), generator=_gen(seed + 1, "cuda"), device="cuda")
    lock = (lock < 0.004).to(torch.uint8)
    return dict(case=case, idx=idx, pos=pos, attr=attr, lock=lock, target=_target(len(idx), case["ratio"]), w_idx=torch.empty_like(idx),
                w_pos=torch.empty_like(pos), w_attr=torch.empty_like(attr))


def _run_update(s):
    c = s["case"]
    # the call works in place: the original stays, a working copy is updated
    s["w_idx"].copy_(s["idx"])
    s["w_pos"].copy_(s["pos"])
    s["w_attr"].copy_(s["attr"])
    n, err = mg.simplify_with_update_device(s["w_idx"].data_ptr(), len(s["idx"]), s["w_pos"].data_ptr(), len(s["pos"]), 12, s["target"], c["error"], c["options"],
                                            d_attributes=s["w_attr"].data_ptr(), attributes_stride=20, weights=_WEIGHTS, d_lock=s["lock"].data_ptr(),
                                            stream=torch.cuda.current_stream().cuda_stream)
    return [n, s["w_idx"], s["w_pos"], s["w_attr"], err]


def _serve_sizes(case):
    z = np.random.default_rng(case["count"] + case["median"]).standard_normal(case["count"])
    return np.clip(case["median"] * np.exp(z), 1000, case["tmax"]).astype(np.int64)


@functools.lru_cache(maxsize=1)
def _server():
    return mg.Server()


def _prepare_serve(case, seed):
    gen = _gen(seed, "cuda")
    ratios = np.random.default_rng(seed + 3).uniform(0.1, 0.5, case["count"])
    meshes, total = [], 0
    for k, tris in enumerate(_serve_sizes(case)):
        n = max(3, int(math.sqrt(tris / 2)) + 1)
        idx = _indices(_lattice(n, n, "cuda"))
        z = 0.05 * torch.randn(n, n, generator=gen, device="cuda", dtype=torch.float64)
        meshes.append(dict(idx=idx, pos=_height_positions(n, n, z, "cuda"), target=_target(len(idx), ratios[k]), at=total))
        total += len(idx)
    return dict(case=case, meshes=meshes, dst=torch.zeros(total, dtype=torch.int32, device="cuda"), server=_server())


def _run_serve(s):
    server, dst = s["server"], s["dst"].data_ptr()
    tickets = [server.submit(m["idx"].data_ptr(), len(m["idx"]), m["pos"].data_ptr(), len(m["pos"]), m["target"], 1e-2, 0, dst + 4 * m["at"]) for m in s["meshes"]]
    done = [server.wait(t) for t in tickets]
    if any(d[0] for d in done):
        raise RuntimeError("request failed: status %s" % [d[0] for d in done if d[0]][0])
    return [np.array([d[1] for d in done], np.int64), np.array([d[2] for d in done], np.float32), s["dst"]]


def _prepare_compact(case, seed):
    gen = _gen(seed, "cuda")
    t = _lattice(case["nx"], case["ny"], "cuda")
    kept = torch.randperm(len(t), generator=gen, device="cuda")[: max(1, int(len(t) * case["keep"]))].sort().values
    idx = _indices(t[kept])
    verts = torch.randn(case["nx"] * case["ny"], case["floats"], generator=gen, device="cuda")
    return dict(case=case, idx=idx, verts=verts, w_idx=torch.empty_like(idx), dst=torch.zeros_like(verts))


def _run_compact(s):
    # indices are rewritten in place: the working copy is what the program draws
    s["w_idx"].copy_(s["idx"])
    v = s["verts"]
    n = mg.optimize_vertex_fetch_device(s["dst"].data_ptr(), s["w_idx"].data_ptr(), len(s["idx"]), v.data_ptr(), len(v), v.shape[1] * 4,
                                        stream=torch.cuda.current_stream().cuda_stream)
    return [n, s["dst"], s["w_idx"]]


_KINDS = {
    "mesh": (_prepare_mesh, _run_mesh), "scan": (_prepare_scan, _run_scan), "groups": (_prepare_groups, _run_groups),
    "level": (_prepare_level, _run_level), "meshlets": (_prepare_meshlets, _run_meshlets), "update": (_prepare_update, _run_update),
    "serve": (_prepare_serve, _run_serve), "compact": (_prepare_compact, _run_compact),
}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state["case"]["kind"]][1](state)


def work(case):
    """Bytes: indices 4 each, positions 12, attributes 20 and locks 1 per vertex in; the result's indices and
    updated vertices out. Nothing here is a contraction, so no operations are counted."""
    k = case["kind"]
    if k == "mesh" or k == "update":
        octa = case.get("surface") == "octa"
        tris = 8 * 4 ** case["nx"] if octa else 2 * (case["nx"] - 1) * (case["ny"] - 1)
        verts = tris // 2 + 2 if octa else case["nx"] * case["ny"]
        attrs = 20 if k == "update" or octa or case["surface"] == "globe" else 0
        b = 12 * tris * (1 + case["ratio"]) + verts * (12 + attrs) * (2 if k == "update" else 1)
    elif k == "scan":
        tris = int((2 * (_part_sizes(case) - 1).prod(1)).sum())
        b = 12 * tris * (1 + case["ratio"]) + 6 * tris
    elif k == "groups":
        tris = int(_patch_sizes(case).sum())
        b = 12 * tris * (1 + case["ratio"]) + 12 * (tris * 0.6)
    elif k == "level":
        tris = 8 * 4 ** case["levels"]
        b = 12 * tris * 1.5 + (tris // 2) * (12 + 20 + 4 + 2)
    elif k == "meshlets":
        tris = 4 * 4 ** case["levels"]
        b = 12 * tris + 12 * (tris // 2) + 3 * tris + 4 * (tris * 0.7)
    elif k == "serve":
        tris = int(_serve_sizes(case).sum())
        b = 12 * tris * 1.3 + 6 * tris
    else:
        tris = 2 * (case["nx"] - 1) * (case["ny"] - 1) * case["keep"]
        used = case["nx"] * case["ny"] * (1 - (1 - case["keep"]) ** 6)
        b = 24 * tris + used * case["floats"] * 8
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Simplified index buffers are whole numbers without a 64-bit value; compaction moves vertices as they are."""
    if case["kind"] != "compact":
        return None
    s = _prepare_compact(case, seed)
    used, inv = torch.unique(s["idx"].long(), return_inverse=True)
    first = torch.full((len(used),), len(inv), dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(len(inv), device="cuda"), reduce="amin")
    order = torch.argsort(first)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(len(order), device="cuda")
    moved = torch.zeros_like(s["verts"], dtype=torch.float64)
    moved[: len(used)] = s["verts"][used[order]].to(torch.float64)
    return [len(used), moved, rank[inv].to(torch.int32)]
