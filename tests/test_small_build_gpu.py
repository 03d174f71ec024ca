"""The one-kernel front of small builds (65,536 triangles and fewer) at the edges of its blocks and keys
per thread, and builds in buffers that repeat, alternate and change (launched directly or as a graph)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 31, 33, 1023, 1024, 1025, 3 * 1024 + 1, 16384, 16385, 32768, 32769, 65536, 65537, 131071, 131072, 131073]


def scene(n, kind):
    from lvbh import scenes
    if kind == "clustered":
        return scenes.clustered_soup(n, seed=n), None
    tri = scenes.uniform_soup(n, seed=n)
    if kind == "equal":
        tri[:] = tri[0]  # one key: the sort must keep input order
    if kind == "narrow":  # bounds well inside the scene: saturating and aliasing coordinates
        return tri, np.array([0.4, 0.4, 0.4, 0.45, 0.6, 0.5], np.float32)
    return tri, None


@pytest.mark.parametrize("kind", ["clustered", "equal", "narrow"])
@pytest.mark.parametrize("n", EDGES)
def test_edges_vs_oracle(builder, n, kind):
    import oracle
    from test_parity_gpu import assert_same, build_np
    tri, bounds = scene(n, kind)
    _, got = build_np(builder, tri, bounds)
    assert_same(got, oracle.build(tri, bounds, threads=0), f"{kind} {n}")


@pytest.mark.parametrize("quads", [1, 22, 23, 90, 128, 181, 256])
@pytest.mark.parametrize("given", [False, True])
def test_mesh_equals_soup(builder, quads, given):
    import torch
    from lvbh import scenes
    xyz, idx = scenes.sphere_mesh(quads, indexed=True)
    v4 = np.full((xyz.shape[0] + 3, 4), 7.0, np.float32)  # rows past the used ones take no part
    v4[:xyz.shape[0], :3] = xyz
    bounds = np.array([-1, -1, -1, 1, 1, 1.5], np.float32) if given else None
    mesh = builder.build_mesh(torch.from_numpy(v4).cuda(), torch.from_numpy(idx.astype(np.int32)).cuda(), bounds)
    soup = builder.build_soup(torch.from_numpy(scenes.sphere_mesh(quads)).cuda(), bounds)
    for k in ("nodes", "parents", "leaf_index", "morton"):
        assert torch.equal(getattr(mesh, k), getattr(soup, k)), k
    assert np.array_equal(mesh.bounds.view(np.uint32), soup.bounds.view(np.uint32))


def test_errors_do_not_stay(builder):
    """Non-finite vertices and bad indices fail their own build, and only that one."""
    import lvbh
    import torch
    from lvbh import _native, scenes
    tri = torch.from_numpy(scenes.uniform_soup(5000, seed=1)).cuda()
    bad = tri.clone()
    bad[4321, 5] = float("nan")
    xyz, idx = scenes.sphere_mesh(20, indexed=True)
    idx = idx.astype(np.int32)
    wrong = idx.copy()
    wrong[500, 1] = xyz.shape[0]
    v4 = np.zeros((xyz.shape[0], 4), np.float32)
    v4[:, :3] = xyz
    dxyz, dv4 = torch.from_numpy(xyz).cuda(), torch.from_numpy(v4).cuda()
    want = builder.build_soup(tri).nodes.clone()
    for call in (lambda: builder.build_soup(bad), lambda: builder.build_soup(bad, [0, 0, 0, 1, 1, 1]),
                 lambda: builder.build_mesh(dv4, torch.from_numpy(wrong).cuda()),
                 lambda: builder.build_indexed(dxyz, torch.from_numpy(wrong).cuda())):
        with pytest.raises(lvbh.LvbhError) as e:
            call()
        assert e.value.code == _native.EINVAL
        assert torch.equal(builder.build_soup(tri).nodes, want)
        builder.build_mesh(dv4, torch.from_numpy(idx).cuda())


@pytest.mark.parametrize("n", [5000, 150000])
def test_buffers_repeat_and_change(n):
    """The same buffers again and again (a graph from the second build on), others in between, other
    contents in the same buffers: every result is that of its own input."""
    import lvbh
    import torch
    from lvbh import scenes
    b = lvbh.BVHBuilder(0)
    soups = [torch.from_numpy(scenes.uniform_soup(n, seed=s)).cuda() for s in (1, 2, 3)]
    want = [b.build_soup(s, graph=False).nodes.clone() for s in soups]
    bufs = [s.clone() for s in soups]
    outs = [lvbh.empty_outputs(n, soups[0].device) for _ in range(2)]
    for step, (buf, content, out) in enumerate([(0, 0, 0), (0, 0, 0), (0, 1, 0), (1, 2, 0), (0, 0, 1), (0, 2, 1), (0, 1, 1),
                                                (0, 0, 0), (0, 1, 0), (2, 1, 1), (2, 2, 1), (2, 0, 1)]):
        bufs[buf].copy_(soups[content])
        outs[out]["nodes"].fill_(-1)
        assert torch.equal(b.build_soup(bufs[buf], outputs=outs[out]).nodes, want[content]), step
    offs = [0, n // 3, n]
    batch = [b.build_batched(s, offs, graph=False).nodes.clone() for s in soups]
    for step, (buf, content, out) in enumerate([(0, 0, 0), (0, 1, 0), (0, 2, 0), (1, 1, 0), (0, 0, 0), (0, 1, 1), (0, 2, 1)]):
        bufs[buf].copy_(soups[content])
        outs[out]["nodes"].fill_(-1)
        assert torch.equal(b.build_batched(bufs[buf], offs, outputs=outs[out]).nodes, batch[content]), step
    b.close()
