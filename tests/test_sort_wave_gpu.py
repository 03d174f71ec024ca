"""The plain sort ranks by words while its tiles are one wave of the device and by ballots above.  At that
line, which moves with the number of SMs: the same words as the look-back sort of a one-mesh batch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "runs"])
@pytest.mark.parametrize("past", [-4096 * 3 - 7, -1, 0, 1, 4096 * 5 + 3])
def test_plain_equals_batch_of_one(builder, past, kind):
    import torch
    from lvbh import scenes
    n = 4096 * 4 * torch.cuda.get_device_properties(0).multi_processor_count + past
    tri = torch.from_numpy(scenes.uniform_soup(n, seed=n)).cuda()
    if kind == "runs":  # long runs of equal digits, where rows fall back to ballots
        tri = tri[torch.arange(n, device="cuda") // 37].contiguous()
    plain, batch = builder.build_soup(tri), builder.build_batched(tri, [0, n])
    for k in ("morton", "leaf_index", "nodes", "parents", "tris"):
        assert torch.equal(getattr(plain, k).view(torch.int32), getattr(batch, k).view(torch.int32)), k
