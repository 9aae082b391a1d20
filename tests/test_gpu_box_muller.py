"""QLA_gaussian's Box-Muller over every 24-bit deviate: states made so that the
two deviates of a site are given integers (the feedback register's words and a
zero multiplier), against the host's double log, sqrt and cos.

The device's functions and the host's are each good to a few units in the last
place of the double, and the result is rounded to float, so both sides give the
same float except where the double lies within that distance of the midpoint of
two floats: 16 ulps of the double are allowed for."""
import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu

ALL = 1 << 24


def _states(cuda, kv, kp):
    """States whose next two deviates are kv and kp (int64 tensors of 24-bit integers)."""
    t1, t2 = kv ^ 48, kp ^ 48  # 48: the congruential part, 12345 >> 8, with multiplier 0
    st = cuda.zeros((kv.numel(), 11), dtype=cuda.int32, device="cuda")
    st[:, 4] = (t1 << 1).to(cuda.int32)
    st[:, 3] = ((t2 ^ ((t1 << 1) >> 7)) << 1).to(cuda.int32)
    return st


def _check(qla, cuda, kv, kp, what):
    n = kv.numel()
    r = cuda.empty(n, dtype=cuda.float32, device="cuda")
    st = _states(cuda, kv, kp)
    qla.lib().QLA_F_R_veq_gaussian_S(T.ptr_dev(r), T.ptr_dev(st), n)
    qla.check("QLA_F_R_veq_gaussian_S")
    got = r.cpu().numpy()
    v, u = (k.cpu().numpy().astype(np.float64) / ALL for k in (kv, kp))
    d = np.sqrt(2.0 * -np.log(v + 1e-307)) * np.cos((u * 2.0) * 3.14159265358979323846)
    want = d.astype(np.float32)
    off = np.flatnonzero(got != want)
    mid = 0.5 * (got[off].astype(np.float64) + want[off].astype(np.float64))
    assert np.all(np.abs(got[off].astype(np.float64) - want[off]) <= np.spacing(np.abs(want[off]))), (what, off[:4])
    assert np.all(np.abs(d[off] - mid) <= 16 * np.spacing(np.abs(d[off]))), (what, off[:4])
    assert len(off) <= 64, (what, len(off))


@pytest.mark.parametrize("which", ["radius", "angle"])
def test_every_deviate(qla, cuda, which):
    step = 1 << 22
    for k0 in range(0, ALL, step):
        k = cuda.arange(k0, k0 + step, dtype=cuda.int64, device="cuda")
        # radius: cos 0 = 1; angle: a radius with no special digits
        other = cuda.full_like(k, 0 if which == "radius" else 5592407)
        _check(qla, cuda, *((k, other) if which == "radius" else (other, k)), (which, k0))


def test_pairs_and_edges(qla, cuda):
    """0, 1 and the largest deviates, both sides of the log table's change of octave
    (leading bits 52 / 53) at every power of two, and of the quadrants of cos."""
    edge = {0, 1, 2, 3, ALL - 1, ALL - 2}
    for e in range(7, 24):
        for lead in (127, 128 + 52, 128 + 53, 128 + 127):
            edge |= {(lead << e >> 7) + d for d in (-1, 0, 1)}
    for q in range(0, 9):
        edge |= {q * (ALL >> 3) + d for d in (-2, -1, 0, 1, 2)}
    edge = cuda.tensor(sorted(k for k in edge if 0 <= k < ALL), dtype=cuda.int64, device="cuda")
    a, b = cuda.meshgrid(edge, edge, indexing="ij")
    _check(qla, cuda, a.reshape(-1).contiguous(), b.reshape(-1).contiguous(), "edges")
    g = cuda.Generator(device="cuda").manual_seed(3)
    pick = [cuda.randint(0, ALL, (1 << 22,), dtype=cuda.int64, device="cuda", generator=g) for _ in range(2)]
    _check(qla, cuda, *pick, "pairs")
