"""Plain builds whose sort chunks hold one, two, four and eight tiles, at the lines between them and past
the chunk counts that the chunk scan keeps in registers (512), from each key pass: a soup's box reduced,
given bounds, an indexed mesh.  The same words as a batch of that one mesh, whose sort looks back over its
tiles and has no chunks.  And builds above 2^22 triangles (a graph from the first one on) in buffers that
change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 4096
BOX = np.array([0.1, 0, 0, 0.9, 1, 1.5], np.float32)


def soup(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    c = torch.rand((n, 1, 3), generator=g, device="cuda")
    tri = torch.full((n, 3, 4), 3.1415, device="cuda")
    tri[:, :, :3] = c + 0.01 * torch.rand((n, 3, 3), generator=g, device="cuda")
    tri[n // 2:n // 2 + n // 8, :, :3] = tri[n // 2, :, :3].clone()  # equal keys across tiles and chunks
    return tri.reshape(n, 12)


def same(a, b, fields=("morton", "leaf_index", "nodes", "parents", "tris")):
    import torch
    for k in fields:
        assert torch.equal(getattr(a, k).view(torch.int32), getattr(b, k).view(torch.int32)), k


@pytest.mark.parametrize("tiles", [513, 591, 592, 1183, 1184, 2367, 2368])
def test_chunks_of_one_to_eight_tiles(builder, tiles):
    import torch
    n = tiles * TILE - (TILE - 1 if tiles % 2 else 1029)  # a ragged last tile, of one key at times
    tri = soup(n, tiles)
    v4 = tri.reshape(3 * n, 4)
    order = torch.randperm(3 * n, generator=torch.Generator(device="cuda").manual_seed(tiles), device="cuda")
    rows = torch.empty_like(v4)
    rows[order] = v4  # vertex i of the soup is row order[i]
    idx = order.to(torch.int32).reshape(n, 3)
    for bounds in (None, BOX):
        want = builder.build_batched(tri, [0, n], seg_bounds=None if bounds is None else BOX[None])
        same(builder.build_soup(tri, bounds), want)
        same(builder.build_mesh(rows, idx, bounds), want, ("morton", "leaf_index", "nodes", "parents"))


def test_twice_the_triangles_of_the_largest_scene(builder):
    n = (1 << 25) + 12345  # 1,028 chunks of eight tiles
    tri = soup(n, 5)
    want = builder.build_batched(tri, [0, n])
    same(builder.build_soup(tri), want)
    want = builder.build_batched(tri, [0, n], seg_bounds=BOX[None])
    same(builder.build_soup(tri, BOX), want)


def test_large_builds_in_changing_buffers():
    import lvbh
    import torch
    n = (1 << 22) + 4099
    b = lvbh.BVHBuilder(0)
    soups = [soup(n, s) for s in (1, 2, 3)]
    want = [b.build_soup(s, graph=False).nodes.clone() for s in soups]
    given = [b.build_soup(s, BOX, graph=False).nodes.clone() for s in soups]
    bufs = [s.clone() for s in soups[:2]]
    outs = [lvbh.empty_outputs(n, soups[0].device) for _ in range(2)]
    for step, (buf, content, out, box) in enumerate([(0, 0, 0, 0), (0, 1, 0, 0), (1, 2, 0, 0), (1, 0, 1, 0), (0, 2, 1, 0),
                                                     (0, 2, 1, 1), (0, 1, 1, 1), (1, 1, 0, 1), (0, 0, 0, 0)]):
        bufs[buf].copy_(soups[content])
        outs[out]["nodes"].fill_(-1)
        got = b.build_soup(bufs[buf], BOX if box else None, outputs=outs[out]).nodes
        assert torch.equal(got, (given if box else want)[content]), step
    b.close()
