"""Stage times of profiled small builds, whose box, keys and sort are one kernel: every stage of the list
is reported, and what a build skips is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# One kernel of 20 to 30 us: reading the triangles and agreeing on the box takes a load from DRAM, two
# block barriers and two cluster barriers, over a microsecond (2 %); the four sort passes take four times
# the same and more.  The keys, three divisions a triangle, are only known to take some time.
@pytest.mark.parametrize("n", [1, 1000, 5000, 20000, 65536])
@pytest.mark.parametrize("mesh", [False, True])
def test_each_stage_has_its_share(builder, n, mesh):
    import torch
    from lvbh import scenes
    tri = scenes.uniform_soup(n, seed=n)
    if mesh:
        xyz, idx = scenes.indexed_from_soup(tri)
        v4 = np.zeros((3 * n, 4), np.float32)
        v4[:, :3] = xyz
        args = (torch.from_numpy(v4).cuda(), torch.from_numpy(idx.astype(np.int32)).cuda())
        build = builder.build_mesh
    else:
        args, build = (torch.from_numpy(tri).cuda(),), builder.build_soup
    box = [0, 0, 0, 1, 1, 1]
    want = build(*args), build(*args, box)
    for given in (False, True, False):
        res = build(*args, box if given else None, profile=True)
        ms = res.stage_ms
        front = ms["bounds"] + ms["morton"] + ms["sort"]
        assert 0.002 < front < 5.0, ms
        assert ms["morton"] > 0 and ms["sort"] > 0.2 * front, ms
        if given:  # skipped; the triangles are read for the keys
            assert ms["bounds"] == 0.0 and ms["morton"] > 0.02 * front, ms
        else:
            assert ms["bounds"] > 0.02 * front, ms
        assert ms["tree"] > 0 and ms["upload"] < 0.1
        for k in ("nodes", "leaf_index", "morton"):  # profiling changes no result
            assert torch.equal(getattr(res, k), getattr(want[given], k)), k
    # a larger build's stages are its events again
    big = builder.build_soup(torch.from_numpy(scenes.uniform_soup(70000, seed=3)).cuda(), profile=True).stage_ms
    assert min(big["bounds"], big["morton"], big["sort"]) > 0
