"""Calls that the launcher sends one site per thread over global memory, at the
sizes where the choice or the block size changes, against the oracle."""
import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu


def _rows(rng, base, n):
    """n records drawn from `base` (host arrays of few distinct records)."""
    return rng.integers(0, len(base), n).astype(np.int32)


@pytest.mark.parametrize("lib,dt", [("FN", np.float32), ("DN", np.float64)])
@pytest.mark.parametrize("nc", [4, 8])
def test_matrix_functions_of_many_colours(qla, nc, lib, dt):
    """Contiguous, pointer and gang forms around the block sizes (32, 64, 128 and
    256 threads, by the sites per SM); every record is one of 64, computed once."""
    sms = qla.lib().qlagpu_sm_count()
    rng = np.random.default_rng(300 + nc)
    base = T.positive_hermitian_inputs(rng, 64, dt, nc=nc)
    vec = T.gaussian_field(rng, 64, nc, dt)
    ns_ = getattr(qla, lib)
    rec = 2 * nc * nc * np.dtype(dt).itemsize
    for fname in ("inverse", "sqrt", "invsqrt", "log", "exp", "expA", "eigenvals", "det"):
        dest = {"eigenvals": "V", "det": "C"}.get(fname, "M")
        want = T.ora_mfunc(base, 64, fname, nc=nc)
        for n in (1, 31, 33, 16 * sms, 16 * sms + 1) + ((64 * sms + 1, 128 * sms + 1) if fname == "inverse" else ()):
            row = _rows(rng, base, n)
            a = T.to_dev(base[row])
            r = T.to_dev(np.zeros((n, want.shape[1]), dt))
            getattr(ns_, f"{dest}_veq_{fname}_M")(nc, r, a, n)
            got = {"v": T.to_host(r)}
            pick = rng.permutation(n).astype(np.int32)
            getattr(ns_, f"{dest}_veq_{fname}_pM")(nc, r, T.ptr_array(a, pick, rec), n)
            got["p"] = T.to_host(r)
            gang = np.sort(rng.permutation(n)[:n // 2 + 1]).astype(np.int32)
            r.zero_()
            getattr(ns_, f"{dest}_xeq_{fname}_M")(nc, r, a, T.to_dev(gang), len(gang))
            got["x"] = T.to_host(r)
            only = np.zeros_like(got["x"])
            only[gang] = want[row[gang]]
            for form, w in (("v", want[row]), ("p", want[row[pick]]), ("x", only)):
                if fname == "log":  # the host libm's log of |A|_F, on the diagonal, may differ in the last place
                    scale = max(1.0, float(np.abs(w).max()))
                    assert np.abs(got[form] - w).max() <= 4 * np.finfo(dt).eps * scale, (fname, n, form)
                else:
                    assert T.bits_equal(got[form], w), (fname, n, form)
    # a^-1 b
    for n in (33, 16 * sms + 1):
        row = _rows(rng, base, n)
        a, b = base[row], vec[rng.integers(0, 64, n)]
        r = T.to_dev(np.zeros((n, 2 * nc), dt))
        ns_.V_veq_M_inverse_V(nc, r, T.to_dev(a), T.to_dev(b), n)
        assert T.bits_equal(T.to_host(r), T.ora_minv(a, b, n, 1, nc=nc)), n
        r = T.to_dev(np.zeros((n, 2 * nc * nc), dt))
        gang = rng.permutation(n).astype(np.int32)
        ns_.M_xeq_M_inverse_M(nc, r, T.to_dev(a), T.to_dev(a), T.to_dev(gang), n)
        assert T.bits_equal(T.to_host(r), T.ora_minv(a, a, n, nc, nc=nc)), n
    assert qla.device_error() == 0


@pytest.mark.parametrize("lib,dt", [("F3", np.float32), ("D3", np.float64)])
def test_scattered_log_and_eigenvalues(qla, lib, dt):
    sms = qla.lib().qlagpu_sm_count()
    rng = np.random.default_rng(311)
    base = T.positive_hermitian_inputs(rng, 64, dt)
    ns_ = getattr(qla, lib)
    for fname, dest, nout in (("log", "M", 9), ("eigenvals", "V", 3)):
        for n in (1, 33, 32 * sms + 1):
            a = T.to_dev(base[_rows(rng, base, n)])
            v, x = T.to_dev(np.zeros((n, 2 * nout), dt)), T.to_dev(np.zeros((n, 2 * nout), dt))
            getattr(ns_, f"{dest}_veq_{fname}_M")(v, a, n)
            gang = rng.permutation(n).astype(np.int32)
            getattr(ns_, f"{dest}_xeq_{fname}_M")(x, a, T.to_dev(gang), n)
            assert T.bits_equal(T.to_host(x), T.to_host(v)), (fname, n)


@pytest.mark.parametrize("lib,dt", [("FN", np.float32), ("DN", np.float64)])
def test_scattered_short_and_long_records(qla, cuda, lib, dt):
    """Gang-index calls around the sizes where they leave the warp-cooperative
    kernel: V of two colours (65,536 sites; reductions and products), and H and D
    of eight colours (one round of the few warps that fit)."""
    rng = np.random.default_rng(321)
    ns_ = getattr(qla, lib)
    red = getattr(qla, "DFN" if lib == "FN" else "DN")
    sms = qla.lib().qlagpu_sm_count()
    for nc, dest, ncol, sizes in ((2, "V", 1, (65535, 65536, 65537, 70001)),
                                  (8, "H", 2, (33, 96 * sms, 96 * sms + 1, 128 * sms, 128 * sms + 33)),
                                  (8, "D", 4, (33, 96 * sms, 96 * sms + 1, 128 * sms, 128 * sms + 33))):
        ncx, ns = nc * ncol, max(sizes) + 7
        a, b = T.gaussian_field(rng, ns, nc * nc, dt), T.gaussian_field(rng, ns, ncx, dt)
        ad, bd = T.to_dev(a), T.to_dev(b)
        for n in sizes:
            gang = np.sort(rng.permutation(ns)[:n]).astype(np.int32)
            gd = T.to_dev(gang)
            for eq in ("eq", "peq"):
                r0 = T.gaussian_field(rng, ns, ncx, dt)
                rd, want = T.to_dev(r0), r0.copy()
                getattr(ns_, f"{dest}_x{eq}_M_times_{dest}")(nc, rd, ad, bd, gd, n)
                T.ora_lmult(want, a, b, n, ncol, eq, gang=gang, nc=nc)
                assert T.bits_equal(T.to_host(rd), want), (nc, dest, eq, n)
            if dest == "V":
                exact = T.ora_norm2(b, n, ncx, exact=True, gang=gang)
                got = red.r_xeq_norm2_V(nc, None, bd, gd, n)
                assert abs(got - exact) <= 1e-12 * exact, n
                c = T.gaussian_field(rng, ns, ncx, dt)
                ed = T.ora_dot(b, c, n, ncx, exact=True, gang=gang)
                gotd = red.c_xeq_V_dot_V(nc, None, bd, T.to_dev(c), gd, n)
                assert abs(gotd - ed) <= 1e-12 * max(1.0, abs(ed)) * 4, n
    assert qla.device_error() == 0


@pytest.mark.parametrize("lib,dt,red", [("F3", np.float32, "DF3"), ("D3", np.float64, "D3")])
@pytest.mark.parametrize("n", [65536, 65537, 100003])
def test_scattered_vector_reductions(qla, lib, dt, red, n):
    rng = np.random.default_rng(331 + n)
    b = T.gaussian_field(rng, n + 5, 3, dt)
    gang = np.sort(rng.permutation(n + 5)[:n]).astype(np.int32)
    exact = T.ora_norm2(b, n, 3, exact=True, gang=gang)
    got = getattr(qla, red).r_xeq_norm2_V(None, T.to_dev(b), T.to_dev(gang), n)
    assert abs(got - exact) <= 1e-12 * exact
