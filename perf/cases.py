"""The calls a program makes on this library, with the sizes, options and values it meets.

A scene goes from OBJ text to triangles (`parse_obj`), from triangles to a tree (`build`,
`build_soup`, `build_indexed`, `build_mesh`, `build_batched`) and from the tree to pixels
(`trace`, `trace_mesh`, `pt_sample`).  Every listed case is one such call on the scenes of
`lvbh/scenes.py` (uniform soup, displaced sphere, clustered soup, batches of meshes, exporter
OBJ text); `draw` gives further sizes and options of the same ranges.  One builder serves the
whole process, as a program keeps one per GPU.  Inputs are made on the GPU from the seed.

    listed()  draw(rng)  prepare(case, seed)  run(state)  work(case)  exact(case, seed)
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "webgpu-lvbh-demo_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

PAD = 3.1415  # the pad word parse-obj.js writes after each vertex
_builders = {}


def _builder():
    import lvbh
    if "b" not in _builders:
        _builders["b"] = lvbh.initBVHBuild(0)
    return _builders["b"]


def listed():
    return [
        # a small OBJ model dropped on the page: 3,362 faces with normals, the file's bytes in
        # host memory; all latency
        {"name": "obj_small_host", "kind": "obj", "quads": 41, "scale": 10.0, "normals": True, "host": True},
        # a large model as an exporter writes it: 2,097,152 faces, 80 MB of text on the device
        {"name": "obj_sphere_2m", "kind": "obj", "quads": 1024, "scale": 1.0, "normals": False, "host": False},
        # the reference's own call: a host TRI_ARRAY, MODEL_BOUNDS from the parser, new buffers
        # out; a small model, all latency
        {"name": "build_small_host", "kind": "build", "scene": "floor", "n": 4098, "bounds": True, "host": True,
         "keep": False},
        # one object rebuilt each frame into buffers the program keeps
        {"name": "build_uniform_64k", "kind": "build", "scene": "uniform", "n": 65536, "bounds": False,
         "host": False, "keep": True},
        # an ordinary scene of ragged size, results in new buffers
        {"name": "build_clustered_1m", "kind": "build", "scene": "clustered", "n": 1000003, "bounds": False,
         "host": False, "keep": False},
        # the largest single scene: 2^24 clustered triangles into kept buffers
        {"name": "build_clustered_16m", "kind": "build", "scene": "clustered", "n": 1 << 24, "bounds": False,
         "host": False, "keep": True},
        # a mesh held as vertex and index buffers, built to the reference's layout
        {"name": "indexed_180k", "kind": "indexed", "quads": 300, "bounds": True},
        # a large mesh built to the indexed leaf format (no triangle copies)
        {"name": "mesh_2m", "kind": "mesh", "quads": 1024, "bounds": False},
        # many small and middling meshes in one call, 64 to 262,144 triangles each
        {"name": "batch_1024", "kind": "batch", "meshes": 1024, "lo": 64, "hi": 262144},
        # picking or visibility rays against a mesh in the indexed leaf format, an odd count
        {"name": "trace_mesh_100k", "kind": "trace", "quads": 256, "rays": 100003, "mesh": True},
        # a frame's worth of closest-hit rays against a large mesh
        {"name": "trace_4m", "kind": "trace", "quads": 1024, "rays": 1 << 22, "mesh": False},
        # one bounce of the path tracer at 1920 x 1080, four samples into the picture
        {"name": "pt_1080p", "kind": "pt", "quads": 1024, "width": 1920, "height": 1080, "samples": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["obj", "build", "build", "build", "indexed", "mesh", "batch", "trace", "pt"])
    if kind == "obj":
        quads = _log(rng, 8, 1024)
        return {"kind": "obj", "quads": quads, "scale": rng.choice([1.0, 10.0, 100.0]),
                "normals": quads <= 700 and rng.random() < 0.5, "host": quads <= 300 and rng.random() < 0.5}
    if kind == "build":
        n = _log(rng, 64, 1 << 24)
        scene = rng.choice(["uniform", "clustered", "floor"])
        return {"kind": "build", "scene": scene, "n": n, "bounds": scene == "floor" or rng.random() < 0.3,
                "host": n <= 1 << 20 and rng.random() < 0.25, "keep": rng.random() < 0.5}
    if kind in ("indexed", "mesh"):
        return {"kind": kind, "quads": _log(rng, 6, 1448), "bounds": rng.random() < 0.5}
    if kind == "batch":
        hi = rng.choice([4096, 65536, 262144])
        return {"kind": "batch", "meshes": _log(rng, 8, 1024), "lo": 64, "hi": hi}
    if kind == "trace":
        return {"kind": "trace", "quads": _log(rng, 16, 1024), "rays": _log(rng, 1024, 1 << 22),
                "mesh": rng.random() < 0.4}
    width = _log(rng, 64, 1920)
    return {"kind": "pt", "quads": _log(rng, 16, 1024), "width": width, "height": max(1, width * 9 // 16),
            "samples": rng.randint(1, 6)}


# ---- scenes, on the GPU -----------------------------------------------------------------------

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _soup(vs):
    """Three (N, 3) vertex tensors -> the (N, 12) float32 triangle layout."""
    tri = torch.full((vs[0].shape[0], 12), PAD, dtype=torch.float32, device="cuda")
    for k in range(3):
        tri[:, 4 * k:4 * k + 3] = vs[k]
    return tri


def _uniform(n, g, lo=0.0, ext=1.0):
    c = lo + _rand(g, n, 3) * ext
    return _soup([c + (_rand(g, n, 3) * 2.0 - 1.0) * 0.005 * ext for _ in range(3)])


def _clustered(n, g):
    """90 % of the centroids from 64 Gaussians, 10 % uniform, in random order."""
    means = _rand(g, 64, 3).float()
    sig = torch.exp(math.log(0.002) + _rand(g, 64) * (math.log(0.05) - math.log(0.002))).float()
    which = torch.randint(0, 64, (n,), generator=g, device="cuda")
    c = means[which] + torch.randn((n, 3), generator=g, device="cuda") * sig[which, None]
    back = torch.rand(n, generator=g, device="cuda") < 0.10
    c = torch.where(back[:, None], torch.rand((n, 3), generator=g, device="cuda"), c)
    return _soup([c + (torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0) * 0.001 for _ in range(3)])


def _floor(n, g):
    """A uniform model plus the parser's two floor triangles, and the bounds of the model alone."""
    m = max(1, n - 2)
    tri = _uniform(m, g)
    v = tri.view(m, 3, 4)[:, :, :3].reshape(-1, 3)
    mn, mx = v.min(0).values, v.max(0).values
    h, s = float(mn[2]) + 0.01, 10000.0
    fl = torch.tensor([[-s, -s, h, PAD, s, -s, h, PAD, -s, s, h, PAD], [s, -s, h, PAD, s, s, h, PAD, -s, s, h, PAD]],
                      dtype=torch.float32, device="cuda")
    return torch.cat([tri, fl])[:n].contiguous(), torch.cat([mn, mx]).cpu().numpy()


def _sphere(quads, g):
    """Displaced unit sphere: (V, 3) float64 vertices and (2 quads^2, 3) int64 indices, in grid order."""
    phi, chi = _rand(g, 8) * 2.0 * math.pi, _rand(g, 8) * 2.0 * math.pi
    th = torch.linspace(0.0, math.pi, quads + 1, dtype=torch.float64, device="cuda")[:, None]
    ps = torch.linspace(0.0, 2.0 * math.pi, quads + 1, dtype=torch.float64, device="cuda")[None, :]
    r = torch.ones((quads + 1, quads + 1), dtype=torch.float64, device="cuda")
    for k in range(1, 9):
        r = r + 0.05 * torch.sin(k * th + phi[k - 1]) * torch.cos(k * ps + chi[k - 1])
    xyz = torch.stack([r * torch.sin(th) * torch.cos(ps), r * torch.sin(th) * torch.sin(ps),
                       r * torch.cos(th) * torch.ones_like(ps)], dim=-1).reshape(-1, 3)
    i = torch.arange(quads, device="cuda")
    a = (i[:, None] * (quads + 1) + i[None, :]).reshape(-1)
    b, c, d = a + 1, a + quads + 1, a + quads + 2
    return xyz, torch.stack([a, c, b, b, c, d], dim=1).reshape(-1, 3)


def _box(tri):
    v = tri.view(-1, 3, 4)[:, :, :3].reshape(-1, 3)
    return torch.cat([v.min(0).values, v.max(0).values]).cpu().numpy()


def _mesh_soup(xyz, idx):
    return _soup([xyz[idx[:, k]] for k in range(3)])


def _rays(count, g):
    """Origins on a radius-3 sphere, unit directions toward points of [-1, 1]^3."""
    o = torch.randn((count, 3), generator=g, device="cuda", dtype=torch.float64)
    o = o / o.norm(dim=1, keepdim=True) * 3.0
    d = _rand(g, count, 3) * 2.0 - 1.0 - o
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.zeros((count, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3] = o
    rays[:, 4:7] = d
    return rays


# ---- OBJ text, written on the GPU -------------------------------------------------------------

def _digits(v, width, least):
    """(N,) integers -> (N, width) digit bytes and the mask of those written (at least `least`)."""
    p = 10 ** torch.arange(width - 1, -1, -1, device="cuda")
    return (v[:, None] // p % 10 + 48).to(torch.uint8), (v[:, None] >= p) | (p < 10 ** least)


def _const(n, text):
    b = torch.tensor(list(text.encode()), dtype=torch.uint8, device="cuda").expand(n, -1)
    return b, torch.ones_like(b, dtype=torch.bool)


def _decimal(micro):
    """Integers of 1e-6 units -> the fields of '%.6f'."""
    n = micro.shape[0]
    mag = micro.abs()
    return [(_const(n, "-")[0], (micro < 0)[:, None]), _digits(mag // 1000000, 4, 1), _const(n, "."),
            _digits(mag % 1000000, 6, 6)]


def _lines(fields):
    return torch.cat([f[0] for f in fields], 1)[torch.cat([f[1] for f in fields], 1)]


def _obj_parts(case, seed):
    g = _gen(seed, 1)
    xyz, idx = _sphere(case["quads"], g)
    return torch.round(xyz * (case["scale"] * 1e6)).to(torch.int64), idx


def _obj_text(case, seed):
    """A comment, `o`, `v` lines with six decimals, optionally `vn` lines, `s off`, `f` lines."""
    micro, idx = _obj_parts(case, seed)
    nv, nf = micro.shape[0], idx.shape[0]

    def rows(key, m):
        n = m.shape[0]
        f = [_const(n, key)]
        for a in range(3):
            f += [_const(n, " ")] + _decimal(m[:, a])
        return _lines(f + [_const(n, "\n")])

    head = "# synthetic mesh: %d vertices, %d faces\no mesh\n" % (nv, nf)
    parts = [_const(1, head)[0][0], rows("v", micro)]
    if case["normals"]:
        unit = micro.double() / micro.double().norm(dim=1, keepdim=True).clamp_min(1.0)
        parts.append(rows("vn", torch.round(unit * 1e6).to(torch.int64)))
    parts.append(_const(1, "s off\n")[0][0])
    f = [_const(nf, "f")]
    for a in range(3):
        num = _digits(idx[:, a] + 1, 8, 1)
        f += [_const(nf, " "), num] + ([_const(nf, "//"), num] if case["normals"] else [])
    parts.append(_lines(f + [_const(nf, "\n")]))
    return torch.cat(parts)


# ---- the contract -----------------------------------------------------------------------------

def _scene(case, seed):
    """A build case's soup (device tensor) and MODEL_BOUNDS (6 floats or None)."""
    g = _gen(seed, 2)
    if case["scene"] == "floor":
        return _floor(case["n"], g)
    tri = _uniform(case["n"], g) if case["scene"] == "uniform" else _clustered(case["n"], g)
    return tri, _box(tri) if case["bounds"] else None


def _batch_sizes(case):
    """Log-uniform mesh sizes, the same for every seed (the order is shuffled by it)."""
    m, lo, hi = case["meshes"], case["lo"], case["hi"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / m)) for i in range(m)]


def _batch(case, seed):
    g = _gen(seed, 3)
    sizes = torch.tensor(_batch_sizes(case), device="cuda")
    sizes = sizes[torch.randperm(sizes.numel(), generator=g, device="cuda")]
    corners = (_rand(g, sizes.numel(), 2, 3) * 200.0 - 100.0)
    lo, hi = corners.min(1).values, corners.max(1).values
    mesh = torch.repeat_interleave(torch.arange(sizes.numel(), device="cuda"), sizes)
    n = int(sizes.sum())
    ext = (hi - lo).float()[mesh]
    c = lo.float()[mesh] + torch.rand((n, 3), generator=g, device="cuda") * ext
    tri = _soup([c + (torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0) * (0.005 * ext) for _ in range(3)])
    offs = np.zeros(sizes.numel() + 1, dtype=np.int64)
    offs[1:] = np.cumsum(sizes.cpu().numpy())
    return tri, offs


def _verts4(xyz):
    v = torch.zeros((xyz.shape[0], 4), dtype=torch.float32, device="cuda")
    v[:, :3] = xyz
    return v


def prepare(case, seed):
    import lvbh
    b = _builder()
    kind = case["kind"]
    s = {"kind": kind, "b": b, "case": case}
    if kind == "obj":
        text = _obj_text(case, seed)
        s["text"] = text.cpu().numpy().tobytes() if case["host"] else text
    elif kind == "build":
        tri, bounds = _scene(case, seed)
        s["n"] = case["n"]
        s["bounds"] = None if bounds is None else {"min": bounds[:3].tolist(), "max": bounds[3:].tolist()}
        s["tri"] = tri.cpu().numpy().reshape(-1) if case["host"] else tri
        s["outputs"] = lvbh.empty_outputs(case["n"], tri.device) if case["keep"] else None
    elif kind in ("indexed", "mesh"):
        xyz, idx = _sphere(case["quads"], _gen(seed, 4))
        s["verts"] = xyz.float().contiguous() if kind == "indexed" else _verts4(xyz)
        s["idx"] = idx.to(torch.int32)
        v = xyz.float()
        s["bounds"] = torch.cat([v.min(0).values, v.max(0).values]).cpu().numpy() if case["bounds"] else None
    elif kind == "batch":
        s["tri"], s["offsets"] = _batch(case, seed)
        s["outputs"] = lvbh.empty_outputs(s["tri"].shape[0], s["tri"].device)
    else:
        xyz, idx = _sphere(case["quads"], _gen(seed, 5))
        if kind == "trace" and case["mesh"]:
            s["verts"] = _verts4(xyz)
            s["tree"] = b.build_mesh(s["verts"], idx.to(torch.int32))
        else:
            s["tree"] = b.build_soup(_mesh_soup(xyz, idx))
        if kind == "trace":
            s["rays"] = _rays(case["rays"], _gen(seed, 6))
        else:  # the picture after some samples; the next one is read from it into a second buffer
            w, h = case["width"], case["height"]
            s["pos"], s["lat"] = lvbh.camera([float(x) for x in s["tree"].bounds], 0.1 * (seed % 60))
            st = [torch.zeros((4, h, w, 4), dtype=torch.float32, device="cuda") for _ in range(2)]
            for k in range(case["samples"]):
                b.pt_sample(s["tree"], None if k == 0 else st[k % 2], st[(k + 1) % 2], w, h, s["pos"], s["lat"],
                            reset=k == 0)
            s["state_in"], s["state_out"] = st[case["samples"] % 2], st[(case["samples"] + 1) % 2]
    torch.cuda.synchronize()
    return s


def _built(r):
    return {"nodes": r.nodes, "tris": r.tris, "parents": r.parents, "leaf_index": r.leaf_index, "morton": r.morton,
            "bounds": r.bounds}


def run(state):
    b, kind, case = state["b"], state["kind"], state["case"]
    if kind == "obj":
        r = b.parse_obj(state["text"])
        return {"num_tris": r["NUM_TRIS"], "tri": r["TRI_ARR"],
                "bounds": np.array(r["BOUNDS"]["min"] + r["BOUNDS"]["max"])}
    if kind == "build":
        if state["outputs"] is None:
            r = b.build(state["tri"], state["n"], state["bounds"])
            return {"nodes": r["BVH_BUFFER"], "tris": r["O_TRIANGLE_BUFFER"], "parents": r["PARENT_BUFFER"],
                    "leaf_index": r["IDX_BUFFER"], "morton": r["Z_IDX_BUFFER"], "bounds": r["BOUNDS"]}
        bounds = state["bounds"]
        tri = state["tri"].reshape(-1, 12)
        return _built(b.build_soup(tri, None if bounds is None else bounds["min"] + bounds["max"],
                                   outputs=state["outputs"]))
    if kind == "indexed":
        return _built(b.build_indexed(state["verts"], state["idx"], state["bounds"]))
    if kind == "mesh":
        return _built(b.build_mesh(state["verts"], state["idx"], state["bounds"]))
    if kind == "batch":
        r = b.build_batched(state["tri"], state["offsets"], outputs=state["outputs"])
        return dict(_built(r), bounds=r.seg_bounds)
    if kind == "trace":
        hit = b.trace_mesh(state["tree"], state["verts"], state["rays"]) if case["mesh"] \
            else b.trace(state["tree"], state["rays"])
        return {"prim": hit[0], "t": hit[1], "stack": hit[2]}
    return b.pt_sample(state["tree"], state["state_in"], state["state_out"], case["width"], case["height"],
                       state["pos"], state["lat"])


def work(case):
    """Bytes: every input once and every output once.  Operations: a comparison or two per key and
    box word for builds, one walk from the root to a leaf per ray."""
    kind = case["kind"]
    out = 64 + 8 + 4 + 4  # node, parent links, permutation and key per triangle
    if kind == "obj":
        q = case["quads"]
        nv, nf = (q + 1) ** 2, 2 * q * q
        text = 30 * nv + (31 * nv if case["normals"] else 0) + nf * (3 * (len(str(nv)) + 1) + 2)
        if case["normals"]:
            text += nf * 3 * (len(str(nv)) + 2)
        return {"bytes": text + 48 * (nf + 2), "flops": 10 * text}
    if kind == "build":
        return {"bytes": case["n"] * (48 + 48 + out), "flops": 60 * case["n"]}
    if kind in ("indexed", "mesh"):
        n, nv = 2 * case["quads"] ** 2, (case["quads"] + 1) ** 2
        rows = 12 * nv + 48 * n if kind == "indexed" else 16 * nv + 12 * n
        return {"bytes": n * (12 + out) + rows, "flops": 60 * n}
    if kind == "batch":
        n = sum(_batch_sizes(case))
        return {"bytes": n * (48 + 48 + out), "flops": 60 * n}
    n = 2 * case["quads"] ** 2
    walk = 2 * 24 * math.ceil(math.log2(n)) + 45
    if kind == "trace":
        leaf = 12 * n + 16 * (case["quads"] + 1) ** 2 if case["mesh"] else 48 * n
        return {"bytes": 64 * n + leaf + case["rays"] * (32 + 12), "flops": walk * case["rays"]}
    px = case["width"] * case["height"]
    return {"bytes": 112 * n + 128 * px, "flops": walk * px}


def _closest(xyz, idx, rays):
    """Distance of each ray's closest hit over all triangles, in double; -1 where it hits none."""
    v = xyz.float().double()
    v0, e1, e2 = v[idx[:, 0]], v[idx[:, 1]] - v[idx[:, 0]], v[idx[:, 2]] - v[idx[:, 0]]
    nrm = torch.linalg.cross(e1, e2)
    out = []
    step = max(1, (1 << 27) // max(1, idx.shape[0]))
    for r in rays.double().split(step):
        o, d = r[:, 0:3], r[:, 4:7]
        d = torch.where(d.abs() < float(np.float32(1e-5)), d + float(np.float32(1e-5)), d)
        # the triple products of Moeller-Trumbore, as matrix products over (ray, triangle)
        det = -(d @ nrm.T)
        od = torch.linalg.cross(o, d)
        u = (od @ e2.T) - (d @ torch.linalg.cross(e2, v0).T)
        w = -(od @ e1.T) + (d @ torch.linalg.cross(e1, v0).T)
        t = (o @ nrm.T) - (nrm * v0).sum(1)
        u, w, t = u / det, w / det, t / det
        ok = (det.abs() >= 1e-10) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > 0)
        best = torch.where(ok, t, torch.full_like(t, math.inf)).min(1).values
        out.append(torch.where(best.isinf(), torch.full_like(best, -1.0), best))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "obj":
        micro, idx = _obj_parts(case, seed)
        xyz = micro.double() / 1e6
        v = xyz[:, [0, 2, 1]]  # the parser swaps y and z
        used = v[idx.reshape(-1)]
        mn, mx = used.min(0).values, used.max(0).values
        tri = torch.full((idx.shape[0] + 2, 12), PAD, dtype=torch.float64, device="cuda")
        for k in range(3):
            tri[:-2, 4 * k:4 * k + 3] = v[idx[:, k]]
        h, s = float(mn[2]) + 0.01, 10000.0
        tri[-2:] = torch.tensor([[-s, -s, h, PAD, s, -s, h, PAD, -s, s, h, PAD],
                                 [s, -s, h, PAD, s, s, h, PAD, -s, s, h, PAD]], dtype=torch.float64, device="cuda")
        return {"num_tris": None, "tri": tri, "bounds": torch.cat([mn, mx])}
    if kind == "build":
        tri, bounds = _scene(case, seed)
        box = torch.from_numpy(np.asarray(bounds if bounds is not None else _box(tri), dtype=np.float64))
        return {"nodes": None, "tris": None, "parents": None, "leaf_index": None, "morton": None, "bounds": box}
    if kind in ("indexed", "mesh"):
        v = _sphere(case["quads"], _gen(seed, 4))[0].float().double()
        return {"nodes": None, "tris": None, "parents": None, "leaf_index": None, "morton": None,
                "bounds": torch.cat([v.min(0).values, v.max(0).values])}
    if kind == "batch":
        tri, offs = _batch(case, seed)
        v = tri.view(-1, 3, 4)[:, :, :3]
        lo, hi = v.min(1).values.double(), v.max(1).values.double()
        mesh = torch.repeat_interleave(torch.arange(len(offs) - 1, device="cuda"),
                                       torch.from_numpy(np.diff(offs)).to("cuda"))[:, None].expand(-1, 3)
        box = torch.zeros((len(offs) - 1, 6), dtype=torch.float64, device="cuda")
        box[:, :3] = box[:, :3].scatter_reduce(0, mesh, lo, "amin", include_self=False)
        box[:, 3:] = box[:, 3:].scatter_reduce(0, mesh, hi, "amax", include_self=False)
        return {"nodes": None, "tris": None, "parents": None, "leaf_index": None, "morton": None, "bounds": box}
    if kind == "trace":
        if case["rays"] * 2 * case["quads"] ** 2 > 1.5e10:
            return None
        xyz, idx = _sphere(case["quads"], _gen(seed, 5))
        return {"prim": None, "t": _closest(xyz, idx, _rays(case["rays"], _gen(seed, 6))), "stack": None}
    return None
