"""Kernels that launch_kernel starts may be resident while the kernel before
them, which may write their inputs, still runs.  Checked in the sources: each
of them waits (overlap_begin) before anything but declarations, and none names
its inputs read-only for the kernel's lifetime (__restrict__, __ldg,
ld.global.nc: such loads may go through the non-coherent path and be moved
across the wait)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qla_b200", "csrc")


def _sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(f) as fh:
            out[os.path.basename(f)] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def _closing(s, at, pair):
    """Index behind the bracket that closes the one at s[at]."""
    depth = 0
    for k in range(at, len(s)):
        depth += {pair[0]: 1, pair[1]: -1}.get(s[k], 0)
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced source")


def _kernels():
    """name -> (file, parameters, body) of every __global__ definition"""
    found = {}
    for f, s in _sources().items():
        for m in re.finditer(r"__global__\s+void\s+", s):
            k = m.end()
            if s.startswith("__launch_bounds__", k):
                k = _closing(s, s.index("(", k), "()")
            name = re.match(r"\s*(\w+)", s[k:])
            p0 = k + name.end()
            p1 = _closing(s, p0, "()")
            b0 = s.index("{", p1)
            found[name.group(1)] = (f, s[p0:p1], s[b0:_closing(s, b0, "{}")])
    return found


def test_overlapping_kernels_wait_and_read_coherently():
    kernels = _kernels()
    launched = set()
    for s in _sources().values():
        launched |= set(re.findall(r"launch_kernel\(\s*&?(\w+)", s))
    launched &= set(kernels)
    assert len(launched) >= 30, sorted(launched)
    for name in sorted(launched):
        f, params, body = kernels[name]
        assert "__restrict__" not in params, (f, name)
        assert not re.search(r"__ldg|ld\.global\.nc|__restrict__", body), (f, name)
        before = body[1:].split("overlap_begin();")
        assert len(before) == 2, (f, name, "waits once")
        # only declarations before the wait
        for line in before[0].split(";"):
            assert not line.strip() or re.match(r"\s*(constexpr|using|extern|__shared__)\b", line), (f, name, line)
