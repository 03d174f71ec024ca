"""Traversal over every form its loads branch on: node records on a 32-byte boundary and off it,
triangle rows that start on either half of a 32-byte window, the first and last leaf, and rays with
NaN, infinite, zero and denormal components - each word equal to the oracle's."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shifted(t, by16):
    """A copy of t whose data starts by16 * 16 bytes past a 256-byte boundary."""
    import torch
    flat = torch.zeros(t.numel() + 4 * by16, dtype=t.dtype, device=t.device)
    flat[4 * by16:] = t.reshape(-1)
    return flat[4 * by16:].reshape(t.shape)


def rays_for(seed, count=512):
    rng = np.random.default_rng(seed)
    rays = np.zeros((count, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-1.0, 2.0, (count, 3))
    rays[:, 4:7] = rng.uniform(0.0, 1.0, (count, 3)) - rays[:, 0:3]
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-40, -1e-5, 3e38], np.float32)
    for i in range(count // 2):  # one or two components replaced in every other ray
        for _ in range(1 + i % 2):
            rays[2 * i, rng.choice([0, 1, 2, 4, 5, 6])] = odd[rng.integers(odd.size)]
    return rays


@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 257, 4097])
@pytest.mark.parametrize("node_shift,tri_shift", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_forms_vs_oracle(builder, n, node_shift, tri_shift):
    import oracle
    import torch
    from lvbh import scenes
    res = builder.build_soup(torch.from_numpy(scenes.uniform_soup(n, seed=n, half_offset=0.2)).cuda())
    ref = res.to_numpy()
    rays = rays_for(n)
    moved = dataclasses.replace(res, nodes=shifted(res.nodes, node_shift), tris=shifted(res.tris, tri_shift))
    got = builder.trace(moved, torch.from_numpy(rays).cuda())
    want = oracle.trace(ref["nodes"], ref["tris"], rays, threads=0)
    for g, w, name in zip(got, want, ("prim", "t", "stack")):
        g = g.cpu().numpy().view(np.uint32)
        assert np.array_equal(g, np.ascontiguousarray(w).view(np.uint32)), (name, np.nonzero(g != w.view(np.uint32))[0][:8])


@pytest.mark.parametrize("node_shift", [0, 1])
def test_mesh_forms(builder, node_shift):
    import torch
    from lvbh import scenes
    xyz, idx = scenes.sphere_mesh(24, indexed=True)
    v4 = np.zeros((xyz.shape[0], 4), np.float32)
    v4[:, :3] = xyz
    dv = torch.from_numpy(v4).cuda()
    mesh = builder.build_mesh(dv, torch.from_numpy(idx.astype(np.int32)).cuda())
    soup = builder.build_soup(torch.from_numpy(scenes.sphere_mesh(24)).cuda())
    rays = torch.from_numpy(rays_for(9, 2048)).cuda()
    moved = dataclasses.replace(mesh, nodes=shifted(mesh.nodes, node_shift))
    for a, b in zip(builder.trace_mesh(moved, dv, rays), builder.trace(soup, rays)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("node_shift,tri_shift", [(1, 0), (0, 1)])
def test_bounce_forms(builder, node_shift, tri_shift):
    import lvbh
    import torch
    from lvbh import scenes
    res = builder.build_soup(torch.from_numpy(scenes.sphere_mesh(12)).cuda())
    moved = dataclasses.replace(res, nodes=shifted(res.nodes, node_shift), tris=shifted(res.tris, tri_shift))
    pos, lat = lvbh.camera([float(x) for x in res.bounds])
    st = [torch.zeros((4, 23, 31, 4), dtype=torch.float32, device="cuda") for _ in range(4)]
    for k in range(6):
        for r, a, b in ((res, st[k % 2], st[(k + 1) % 2]), (moved, st[2 + k % 2], st[2 + (k + 1) % 2])):
            builder.pt_sample(r, None if k == 0 else a, b, 31, 23, pos, lat, reset=k == 0)
        assert torch.equal(st[(k + 1) % 2].view(torch.int32), st[2 + (k + 1) % 2].view(torch.int32))
