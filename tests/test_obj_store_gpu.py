"""The two-call OBJ parse into memory of the caller knows where that memory ends."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TEXT = ("o m\n" + "".join("v %d %d %d\n" % (i, i * i % 7, -i) for i in range(12)) + "f 1 2 3 4 5 6 7 8 9 10 11 12\n").encode()


def begin(builder, n):
    from lvbh import _native
    line = ctypes.c_uint64()
    assert _native.lib.lvbh_parse_obj_begin(builder.ctx, TEXT, len(TEXT), _native.INPUT_HOST, ctypes.byref(n),
                                            ctypes.byref(line), None) == _native.OK
    return line


def test_store_refuses_a_short_buffer_and_takes_a_full_one(builder):
    import torch
    from lvbh import _native
    want = builder.parse_obj(TEXT)
    n, b6 = ctypes.c_uint32(), (ctypes.c_double * 6)()
    line = begin(builder, n)
    assert n.value == want["NUM_TRIS"] == 12
    store = lambda t, room: _native.lib.lvbh_parse_obj_store(builder.ctx, ctypes.c_void_p(t.data_ptr()), room, b6,  # noqa: E731
                                                             ctypes.byref(line), None)
    guard = torch.full((n.value + 1, 12), -5.0, device="cuda")
    for room in (0, 1, n.value - 1):
        assert store(guard, room) == _native.EINVAL
    assert torch.all(guard == -5.0)
    assert store(guard, n.value) == _native.OK  # the scan is still there
    assert torch.equal(guard[:-1].view(torch.int32), want["TRI_ARR"].view(torch.int32)) and torch.all(guard[-1] == -5.0)
    assert np.array_equal(np.array(b6), np.array(want["BOUNDS"]["min"] + want["BOUNDS"]["max"]))
    assert store(guard, n.value) == _native.EINVAL  # nothing scanned any more


def test_into_refuses_an_allocation_that_ends_too_early(builder):
    import torch
    from lvbh import _native
    n, b6 = ctypes.c_uint32(), (ctypes.c_double * 6)()
    line = begin(builder, n)
    keep = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")
    seg, = [s for s in torch.cuda.memory_snapshot() if s["address"] <= keep.data_ptr() < s["address"] + s["total_size"]]
    end = seg["address"] + seg["total_size"]
    into = lambda p: _native.lib.lvbh_parse_obj_into(builder.ctx, ctypes.c_void_p(p), b6, ctypes.byref(line), None)  # noqa: E731
    assert into(end - 48 * (n.value - 1)) == _native.EINVAL
    assert into(end - 48) == _native.EINVAL
    assert into(keep.data_ptr()) == _native.OK


def test_into_takes_pool_memory(builder):
    """Memory whose end is not told (a stream-ordered pool's) is the caller's word, as it was."""
    import lvbh
    here, pkg = os.path.dirname(os.path.abspath(__file__)), os.path.dirname(os.path.dirname(os.path.abspath(lvbh.__file__)))
    code = (
        "import sys, ctypes; sys.path[:0] = [%r, %r]\n"
        "import torch, lvbh\n"
        "from lvbh import _native\n"
        "from test_obj_store_gpu import TEXT, begin\n"
        "b = lvbh.BVHBuilder(0)\n"
        "want = b.parse_obj(TEXT)['TRI_ARR']\n"
        "n, b6 = ctypes.c_uint32(), (ctypes.c_double * 6)()\n"
        "line = begin(b, n)\n"
        "tri = torch.empty((n.value, 12), device='cuda')\n"
        "rc = _native.lib.lvbh_parse_obj_into(b.ctx, ctypes.c_void_p(tri.data_ptr()), b6, ctypes.byref(line), None)\n"
        "assert rc == _native.OK and torch.equal(tri.view(torch.int32), want.view(torch.int32))\n"
        "big = torch.empty((1 << 21, 12), device='cuda')\n"
        "line = begin(b, n)\n"
        "rc = _native.lib.lvbh_parse_obj_into(b.ctx, ctypes.c_void_p(big[(1 << 21) - 12].data_ptr()), b6, ctypes.byref(line), None)\n"
        "assert rc == _native.OK and torch.equal(big[-12:].view(torch.int32), want.view(torch.int32))\n"
        % (pkg, here))
    for conf in ("backend:cudaMallocAsync", "expandable_segments:True"):
        subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, PYTORCH_CUDA_ALLOC_CONF=conf), timeout=300)
