"""The straddling pass at the edges of its levels: 24 tree blocks of 256 leaves per group, 16 groups
per unit of the next level, 16 of those per unit of the level after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUP = 24 * 256


@pytest.mark.parametrize("n", [GROUP - 1, GROUP, GROUP + 1, 2 * GROUP + 1, 16 * GROUP, 16 * GROUP + 1,
                               17 * GROUP + 257, 256 * GROUP + 1])
def test_level_edges_vs_oracle(builder, n):
    import oracle
    from lvbh import scenes
    from test_parity_gpu import assert_same, build_np
    tri = scenes.clustered_soup(n, seed=n)
    _, got = build_np(builder, tri, None)
    assert_same(got, oracle.build(tri, None, threads=0), f"n {n}")


def test_levels_in_a_batch(builder):
    """Meshes of one block, one group, two groups and two levels in one batch equal their own builds."""
    import torch
    from lvbh import scenes
    sizes = [1, 200, 257, GROUP, GROUP + 1, 0, 16 * GROUP + 300, 3 * GROUP, 2]
    offs = np.concatenate([[0], np.cumsum(sizes)])
    soup = np.concatenate([scenes.uniform_soup(m, seed=i) for i, m in enumerate(sizes)])
    batch = builder.build_batched(torch.from_numpy(soup).cuda(), offs).to_numpy()
    for i, m in enumerate(sizes):
        if not m:
            continue
        a, b = offs[i], offs[i + 1]
        alone = builder.build_soup(torch.from_numpy(soup[a:b]).cuda()).to_numpy()
        for key, w in (("nodes", 1), ("tris", 1), ("parents", 2), ("leaf_index", 1), ("morton", 1)):
            x = np.ascontiguousarray(batch[key][w * a:w * b]).view(np.uint32)
            assert np.array_equal(x, np.ascontiguousarray(alone[key]).view(np.uint32)), (i, m, key)
