"""What a chained kernel may touch before chain_wait: nothing that a kernel it can overtake writes.

A kernel launched with programmatic stream serialisation may start while the kernel before it on the
stream is finishing.  Every pointer-like parameter of every chained kernel that its body names before
the wait, helpers and structs of pointers included, has to be listed here with the reason why it is
final by then, and no block may leave before its wait: completion of a chained kernel stands for
completion of the one before it, whichever blocks had work.  Checked on the sources (no GPU)."""
import re

from test_chained_kernels import _kernel_body, _sources

# kernel -> parameters that it may name before the wait
ALLOWED = {
    # the text was on the device before k_nl_count, which k_scan_small's wait saw complete
    "k_nl_write": {"s"},
    # obj_scan waited on the host for everything that these were written by
    "k_faces": {"text", "line_start", "type", "fans", "pre"},
}
SCALARS = re.compile(r"^(const\s+)?(bool|int|float|double|uint8_t|uint32_t|uint64_t|size_t|U|int32_t|HostBounds|PtFrame)$")


def _split(params):
    """Top-level commas of a parameter list (template arguments keep theirs)."""
    out, depth, cur = [], 0, ""
    for ch in params:
        depth += {"<": 1, "(": 1, ">": -1, ")": -1}.get(ch, 0)
        if ch == "," and depth == 0:
            out.append(cur)
            cur = ""
        else:
            cur += ch
    return [p.strip() for p in out + [cur] if p.strip()]


def _memory_params(text, kernel):
    """Names of the kernel's parameters that are or may hold pointers (anything but plain values)."""
    m = re.search(r"__global__[^{;]*?\b" + kernel + r"\s*\(", text)
    i, depth = m.end(), 1
    while depth:
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        i += 1
    names = set()
    for p in _split(re.sub(r"//[^\n]*", "", text[m.end():i - 1])):
        p = re.sub(r"\b(__restrict__|__grid_constant__)\b", " ", p)
        typ, name = re.match(r"^(.*?)(\w+)$", p, flags=re.S).groups()
        if "*" in typ or not SCALARS.match(" ".join(typ.split())):
            names.add(name)
    return names


def _chained():
    src = _sources()
    kernels = {m.group(1) for t in src.values() for m in re.finditer(r"launch_chained\(\s*[^,]+,\s*(k_\w+)", t)}
    assert len(kernels) >= 12, kernels
    for k in sorted(kernels):
        text, = [t for t in src.values() if _kernel_body(t, k)]
        body = re.sub(r"//[^\n]*", "", _kernel_body(text, k))
        assert body.count("chain_wait();") == 1, k
        yield k, _memory_params(text, k), body[:body.index("chain_wait();")]


def test_only_final_memory_is_named_before_the_wait():
    for kernel, params, before in _chained():
        assert params, kernel
        used = {p for p in params if re.search(r"\b" + p + r"\b", before)}
        assert used <= ALLOWED.get(kernel, set()), (kernel, used)


def test_no_block_leaves_before_its_wait():
    for kernel, _, before in _chained():
        assert not re.search(r"\breturn\s*;", before), kernel  # (a lambda's returns a value)
