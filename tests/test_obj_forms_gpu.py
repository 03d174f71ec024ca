"""OBJ lines at the edges of the short loops for common forms, model ranges that cut blocks of 256
lines, and texts with many more lines than their size suggests - against the oracle, bit for bit."""
import numpy as np
import pytest

from test_obj_gpu import check_same

pytestmark = pytest.mark.gpu

V = "v 1.5 -2.25 .5\nv -0 +1 0.0\nv 123456789 -0.12345678 1e2\nv 1234567890 1. -.5\n"

VERTEX_LINES = ["v 1 2 3", "v  1   2    3  ", "v 1 2 3\r", "v\t1\t2\t3", "v 1 2", "v 1", "v", "v 1 2 3 4 5", "v 1 2 3#c", "v 1 2 #3",
                "v -.5 -0 -0.0", "v 1.2.3 4 5", "v 1e3 2E-2 3e", "v Infinity -Infinity 1", "v x 1 2", "v 999999999 0.99999999 1.00000000",
                "v 1234567890 12345.67891 0000000001", "V 1 2 3", " v 1 2 3", "v 1 2 3 \r", "v 1\r2 3", "v - 1 2", "v 1 2 3 4",
                "v 00000000012 1 2", "v 1 2 -"]
FACE_LINES = ["f 1 2 3", "f  1  2  3 ", "f 1 2 3\r", "f 1 2 3 \r", "f\t1 2\t3", "f 1 2 3 4 1", "f 1/1 2/2 3/3", "f 1//1 2//2 3//3",
              "f 1/2/3 2/3/4 3/4/5", "f 1/2/3/4 2 3", "f 1 2", "f 1", "f", "f -1 -2 -3", "f +1 2 3", "f 01 2 3", "f 0x1 2 3", "f 1 2 3 # c",
              "f 1 2 3#c", "f 1 2 0", "f 1 2 -0", "f 1 2 x", "f 1 2 3x", "f 1.5 2 3", "f 1 2 4", "f 1 2 5", "f 1 2 999999999",
              "f 1 2 9999999999", "f 1 2 3 4", "f 1/a#b 2 3", "F 1 2 3", " f 1 2 3", "f 1\r2 3", "f 1/ 2/ 3/", "f /1 2 3", "f 1 2 3 　"]


@pytest.mark.parametrize("where", ["host", "device", "device_odd"])
def test_line_forms(builder, where):
    for line in VERTEX_LINES:
        check_same(builder, V + line + "\nf 1 2 3\nf 1 2 5\n", where, repr(line))
        check_same(builder, V + line, where, repr(line) + " at the end")
    for line in FACE_LINES:
        check_same(builder, V + line + "\nf 3 2 1\n", where, repr(line))
        check_same(builder, V + line, where, repr(line) + " at the end")


@pytest.mark.parametrize("first,second", [(0, 255), (0, 256), (1, 257), (255, 511), (256, 700), (300, 301), (255, 256), (511, 5000)])
@pytest.mark.parametrize("default_model", [False, True])
def test_model_ranges(builder, first, second, default_model):
    """`o` lines at given line numbers; statements before the first one open the default model."""
    rng = np.random.default_rng(first * 7919 + second)
    lines, nv = [], 0
    for k in range(6000):
        if k in (first, second, 5500):
            lines.append("o part%d" % k)
            if not (default_model and first > 0):
                nv = 0
        elif k < first and not default_model:
            lines.append("# nothing yet")
        elif nv < 3 or rng.random() < 0.5:
            lines.append("v %.6f %.6f %.6f" % tuple(rng.normal(size=3)))
            nv += 1
        else:
            lines.append("f " + " ".join("-%d" % i for i in rng.integers(1, 4, int(rng.integers(3, 6)))))
    check_same(builder, "\n".join(lines) + "\n", "host", f"{first} {second}")


def test_many_short_lines(builder):
    """More lines than a sixteenth of the bytes: the line arrays grow and the passes run again."""
    body = V + "f 1 2 3\n"
    for text in ("\n" * 200000 + body, body + "\n" * 300001, "f 1 2 3\n" * 120000 + V, (V + "f -1 -2 -3\n") * 30000):
        check_same(builder, text, "device", "short lines")
        check_same(builder, body, "host", "after them")


def test_long_lines(builder):
    """A line longer than a block's window, between lines inside it."""
    long_face = "f " + " ".join("%d" % (1 + k % 4) for k in range(20000))
    check_same(builder, V + "f 1 2 3\n" + long_face + "\nf 2 3 4\n# " + "x" * 50000 + "\nf 4 3 2\nv 1 2 3" + " " * 40000 + "\nf 5 1 2", "host", "long")


def test_two_call_form(builder):
    """lvbh_parse_obj_begin / _into in caller memory equals lvbh_parse_obj; misuse is LVBH_EINVAL."""
    import ctypes
    import torch
    from lvbh import _native
    text = (V + "f 1 2 3 4\nf -1 -2 -3\n").encode()
    want = builder.parse_obj(text, stream=torch.cuda.Stream())  # the one-call form
    got = builder.parse_obj(text)
    assert torch.equal(got["TRI_ARR"].view(torch.int32), want["TRI_ARR"].view(torch.int32)) and got["BOUNDS"] == want["BOUNDS"]
    tri, b6, line = torch.empty(48 * 5, device="cuda"), (ctypes.c_double * 6)(), ctypes.c_uint64()
    into = lambda p: _native.lib.lvbh_parse_obj_into(builder.ctx, p, b6, ctypes.byref(line), None)  # noqa: E731
    assert into(ctypes.c_void_p(tri.data_ptr())) == _native.EINVAL  # nothing scanned
    assert into(None) == _native.EINVAL
    n = ctypes.c_uint32()
    assert _native.lib.lvbh_parse_obj_begin(builder.ctx, text, len(text), _native.INPUT_HOST, ctypes.byref(n),
                                            ctypes.byref(line), None) == _native.OK
    assert into(ctypes.c_void_p(tri.data_ptr() + 4)) == _native.EINVAL  # not on 16 bytes
    assert into(ctypes.c_void_p(tri.data_ptr())) == _native.OK and n.value == want["NUM_TRIS"]
    assert torch.equal(tri[:12 * n.value].view(torch.int32), want["TRI_ARR"].reshape(-1).view(torch.int32))
