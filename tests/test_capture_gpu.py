"""Builds on a stream that the caller is capturing: refused, whatever their size and whatever was built
before, unless LVBH_NO_GRAPH asks for plain launches (a caller's graph would keep the context's buffers,
and a build that replays a graph of its own cannot be captured)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

VP = ctypes.c_void_p


def result(out):
    from lvbh import _native
    r = _native.Result()
    for k in ("nodes", "tris", "parents", "leaf_index", "morton"):
        setattr(r, k, out[k].data_ptr())
    return r


@pytest.mark.parametrize("n", [1, 1000, 70000, (1 << 22) + 5])  # one cluster kernel; launched directly; always a graph
@pytest.mark.parametrize("kind", ["soup", "indexed", "mesh", "batch"])
def test_a_captured_build_is_refused(builder, kind, n):
    import lvbh
    import torch
    from lvbh import _native
    lib, ctx = _native.lib, builder.ctx
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    v4 = torch.rand((3 * n, 4), generator=g, device="cuda")
    tri, xyz = v4.reshape(n, 12), v4[:, :3].contiguous()
    idx = torch.arange(3 * n, device="cuda", dtype=torch.int32)
    outs = [lvbh.empty_outputs(n, tri.device) for _ in range(2)]
    structs = [result(o) for o in outs]
    offs = (ctypes.c_uint32 * 3)(0, n // 2, n)
    stream = torch.cuda.Stream()
    p = lambda t: VP(t.data_ptr())  # noqa: E731

    def call(flags, o):
        flags |= _native.OUT_CALLER
        r, s = ctypes.byref(structs[o]), VP(stream.cuda_stream)
        if kind == "soup":
            return lib.lvbh_build_soup(ctx, p(tri), n, None, flags, r, s)
        if kind == "indexed":
            return lib.lvbh_build_indexed(ctx, p(xyz), 3 * n, p(idx), n, None, flags, r, s)
        if kind == "mesh":
            return lib.lvbh_build_mesh(ctx, p(v4), 3 * n, p(idx), n, None, flags, r, s)
        return lib.lvbh_build_batched(ctx, p(tri), offs, 2, None, None, flags, r, s)

    torch.cuda.synchronize()
    assert call(0, 0) == _native.OK  # the context's scratch is there, and a build in these buffers
    want = outs[0]["nodes"].clone()
    # buffers not seen before, seen, seen again; with a wait; plain launches
    for flags, o in ((_native.ASYNC, 1), (_native.ASYNC, 0), (_native.ASYNC, 0), (0, 0), (_native.ASYNC | _native.NO_GRAPH, 0)):
        graph, whole = torch.cuda.CUDAGraph(), True
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            rc = call(flags, o)
            try:
                graph.capture_end()
            except RuntimeError:
                whole = False
        assert rc == (_native.OK if flags & _native.NO_GRAPH else _native.ECUDA), (flags, o)
        assert whole, (flags, o)  # a refused call leaves the caller's capture as it was
        assert lib.lvbh_sync(ctx) == _native.OK
        del graph
    outs[0]["nodes"].fill_(-1)
    torch.cuda.synchronize()
    assert call(0, 0) == _native.OK  # outside a capture as before
    assert torch.equal(outs[0]["nodes"].view(torch.int32), want.view(torch.int32))
