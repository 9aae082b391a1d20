"""The warp-cooperative site kernel (gang-index forms and operands that are not
16-B aligned) at the edges of its 32-site tiles, against the oracle, bit for
bit: maps with 8-B and 16-B pieces, pointers whose records are only 8-B
aligned, sites outside the gang index left alone, and reductions."""
import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu

PCS = [("F3", np.float32), ("D3", np.float64)]
SIZES = [1, 31, 32, 33, 127, 128, 129, 2051, 70003]


@pytest.mark.parametrize("pc,dt", PCS)
@pytest.mark.parametrize("n", SIZES)
def test_gang_hop_term_and_norm2(qla, cuda, pc, dt, n):
    rng = np.random.default_rng(7 * n)
    rb, ns = (8 if pc == "F3" else 16), 2 * n + 3
    u, d = T.haar_su3(rng, ns, dt), T.gaussian_field(rng, ns, 12, dt)
    r0 = T.gaussian_field(rng, ns, 12, dt)
    idx = rng.integers(0, ns, ns).astype(np.int32)
    gang = np.sort(rng.permutation(ns)[:n]).astype(np.int32)
    ns_ = getattr(qla, pc)
    for shift in ((0, 8) if pc == "F3" else (0,)):  # bytes past a 16-B boundary
        flat = cuda.zeros(ns * 24 + 4, dtype=cuda.float32 if pc == "F3" else cuda.float64, device="cuda")
        k = shift // 4
        flat[k:k + d.size].copy_(cuda.from_numpy(d.reshape(-1)))
        ptrs = cuda.from_numpy(flat.data_ptr() + shift + idx.astype(np.int64) * (12 * rb)).cuda()
        ud, rd = T.to_dev(u), T.to_dev(r0)
        ns_.D_xpeq_spproj_M_times_pD(rd, ud, ptrs, 2, -1, T.to_dev(gang), n)
        want = r0.copy()
        T.ora_hop(want, u, d, n, 2, -1, "peq", "D", "spproj", idx_b=idx, gang=gang)
        assert T.bits_equal(T.to_host(rd), want), shift
    got = getattr(qla, "DF3" if pc == "F3" else "D3").r_xeq_norm2_D(None, T.to_dev(d), T.to_dev(gang), n)
    exact = T.ora_norm2(d, n, 12, exact=True, gang=gang)
    assert abs(got - exact) <= 1e-12 * exact


@pytest.mark.parametrize("n", SIZES)
def test_unaligned_records(qla, n):
    """F3 operands that start 8 bytes past a 16-B boundary, no gang index."""
    rng = np.random.default_rng(n)
    for dest, nc, ncol in (("V", 3, 1), ("H", 6, 2), ("D", 12, 4), ("M", 9, 3)):
        a, b = T.haar_su3(rng, n + 1, np.float32), T.gaussian_field(rng, n + 1, nc)
        buf = np.zeros((n + 2) * 2 * nc, np.float32)
        bd, rd, ad = T.to_dev(buf), T.to_dev(buf), T.to_dev(a)
        bd[2:2 + 2 * nc * n] = T.to_dev(b[:n].reshape(-1))
        getattr(qla.F3, f"{dest}_veq_M_times_{dest}")(rd.data_ptr() + 8, ad, bd.data_ptr() + 8, n)
        want = np.zeros((n, 2 * nc), np.float32)
        T.ora_lmult(want, a, b, n, ncol, "eq")
        got = T.to_host(rd)
        assert T.bits_equal(got[2:2 + 2 * nc * n].reshape(n, -1), want), dest
        assert not got[:2].any() and not got[2 + 2 * nc * n:].any(), dest
