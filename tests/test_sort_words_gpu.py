"""The plain sort's two rankings (by shared words up to 512 tiles of 4,096 keys, by ballots above), at
the line and at ragged ends: leaf_index is the stable argsort of the keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "runs"])
@pytest.mark.parametrize("n", [65_537, 4096 * 17, 4096 * 200 + 31, 4096 * 512 - 1, 4096 * 512, 4096 * 512 + 1])
def test_stable_order_at_the_line(builder, n, kind):
    import torch
    from lvbh import scenes
    tri = scenes.uniform_soup(n, seed=n)
    if kind == "runs":  # rows with fewer and with more equal digits than the words are kept for
        tri = tri[np.repeat(np.arange(n), np.random.default_rng(n).integers(1, 40, n))[:n]]
    res = builder.build_soup(torch.from_numpy(np.ascontiguousarray(tri)).cuda()).to_numpy()
    perm = res["leaf_index"].view(np.uint32).astype(np.int64)
    key = np.empty(n, np.uint32)
    key[perm] = res["morton"].view(np.uint32)
    np.testing.assert_array_equal(perm, np.argsort(key, kind="stable"))
