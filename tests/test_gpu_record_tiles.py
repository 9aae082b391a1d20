"""Kernels that take 32 sites of a contiguous field per warp -- the site-local
products, the random fills -- and the padded-slot products of 4 and 8 colours,
at the edges of their tiles and for fields that start off a 16-B boundary,
against the oracle."""
import ctypes

import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 127, 129, 1000]
LOCAL = ["C_veq_V_dot_V", "C_vpeq_D_dot_D", "R_veq_norm2_P", "R_vmeq_re_M_dot_M", "C_veq_M_dot_Ma", "C_veqm_Pa_dot_P",
         "R_veq_norm2_H", "C_veq_Ma_dot_M", "M_vpeq_V_times_Va"]


def _shifted(cuda, arr, off):
    """Device copy of arr that starts `off` bytes past a 16-B boundary: (address, tensor)."""
    raw = np.ascontiguousarray(arr).view(np.uint8).reshape(-1)
    t = cuda.zeros(raw.size + 32, dtype=cuda.uint8, device="cuda")
    t[off:off + raw.size] = cuda.from_numpy(raw.copy()).cuda()
    return t.data_ptr() + off, t


def _back(t, off, like):
    raw = t[off:off + like.nbytes].cpu().numpy()
    return raw.view(like.dtype).reshape(like.shape)


def _call(qla, cuda, name, lead, e, ins, n, off):
    args, keep, r = list(lead), [], None
    for t, p in zip(e["ctypes"], e["params"]):
        if p == "n":
            args.append(n)
            continue
        a, dev = _shifted(cuda, ins[p][2], off)
        keep.append(dev)
        args.append(ctypes.c_void_p(a))
        if p == "r":
            r = dev
    getattr(qla.lib(), name)(*args)
    qla.check(name)
    return _back(r, off, ins["r"][2])


@pytest.mark.parametrize("pc,nc", [("F3", 3), ("D3", 3), ("FN", 2), ("FN", 4), ("DN", 2), ("DN", 4)])
def test_site_local_products(qla, cuda, pc, nc):
    byname = {e["name"]: e for e in qla.manifest()}
    rng = np.random.default_rng(31 + nc)
    dt = np.float32 if pc[0] == "F" else np.float64
    for n in SIZES:
        for short in LOCAL:
            name = f"QLA_{pc}_{short}"
            e = byname[name if nc == 3 else T.fixed_colour_twin(name)]
            ins, idx, gang = T.ewise_inputs(e, rng, dt, n, n, nc=nc)
            want = T.ewise_oracle(e, ins, idx, gang, n, nc=nc)
            for off in (0, 8, 4) if dt == np.float32 else (0, 8):  # bytes past a 16-B boundary
                got = _call(qla, cuda, name, [] if nc == 3 else [nc], e, ins, n, off)
                assert T.bits_equal(got, want), (name, n, off)


@pytest.mark.parametrize("pc,dest", [("F3", "V"), ("F3", "D"), ("F3", "P"), ("D3", "V"), ("D3", "M"), ("F", "R"),
                                     ("F", "C"), ("D", "R")])
@pytest.mark.parametrize("op", ["gaussian", "random"])
def test_random_fills(qla, cuda, pc, dest, op):
    if op == "random" and dest != "R":
        pytest.skip("uniform fills exist for real fields only")
    byname = {e["name"]: e for e in qla.manifest()}
    name = f"QLA_{pc}_{dest}_veq_{op}_S"
    e = byname[name]
    rng = np.random.default_rng(77)
    for n in SIZES:
        ins, idx, gang, ints, want_r, want_s = T.random_case(e, rng, n, n)
        for off_r, off_s in ((0, 0), (8, 4), (0, 12)):
            ra, rt = _shifted(cuda, ins["r"][2], off_r)
            sa, st = _shifted(cuda, ins["a"][2], off_s)
            getattr(qla.lib(), name)(ctypes.c_void_p(ra), ctypes.c_void_p(sa), n)
            qla.check(name)
            assert T.bits_equal(_back(st, off_s, want_s), want_s), (name, n, off_s)
            got = np.asarray(_back(rt, off_r, want_r), np.float32).ravel()
            w = np.asarray(want_r, np.float32).ravel()
            if op == "random":
                assert T.bits_equal(got, w), (name, n)
            else:  # the stated bound: one float ulp
                assert np.all(np.abs(got.astype(np.float64) - w) <= np.spacing(np.abs(w))), (name, n)


@pytest.mark.parametrize("pc", ["FN", "DN"])
@pytest.mark.parametrize("nc", [2, 4, 8])
def test_padded_slot_products(qla, cuda, pc, nc):
    rng = np.random.default_rng(nc)
    dt = np.float32 if pc == "FN" else np.float64
    L = qla.lib()
    for n in (1, 31, 33, 129, 515):
        a = T.gaussian_field(rng, n, nc * nc, dt)
        b, v = T.gaussian_field(rng, n, nc * nc, dt), T.gaussian_field(rng, n + 3, nc, dt)
        d, d2 = T.gaussian_field(rng, n, 4 * nc, dt), T.gaussian_field(rng, n, 4 * nc, dt)
        idx = rng.integers(0, n + 3, n).astype(np.int32)
        ad, bd, vd, xd = T.to_dev(a), T.to_dev(b), T.to_dev(v), T.to_dev(idx)
        rm, rv = T.to_dev(np.zeros_like(a)), T.to_dev(np.zeros((n, 2 * nc), dt))
        getattr(L, f"QLA_{pc}_M_veq_M_times_Ma")(nc, T.ptr_dev(rm), T.ptr_dev(ad), T.ptr_dev(bd), n)
        getattr(L, f"QLA_{pc}_V_eq_M_times_xV")(nc, T.ptr_dev(rv), T.ptr_dev(ad), T.ptr_dev(vd), T.ptr_dev(xd), n)
        wm, wv = np.zeros_like(a), np.zeros((n, 2 * nc), dt)
        T.ora_lmult(wm, a, b, n, nc, "eq", adjb=1, nc=nc)
        T.ora_lmult(wv, a, v, n, 1, "eq", idx_b=idx, nc=nc)
        assert T.bits_equal(T.to_host(rm), wm) and T.bits_equal(T.to_host(rv), wv), (nc, n)
        res = cuda.zeros(2, dtype=cuda.float64, device="cuda")
        dd, d2d = T.to_dev(d), T.to_dev(d2)
        getattr(L, "QLA_DFN_c_veq_D_dot_D" if pc == "FN" else "QLA_DN_c_veq_D_dot_D")(
            nc, T.ptr_dev(res), T.ptr_dev(dd), T.ptr_dev(d2d), n)
        z, z2 = (x.astype(np.float64).ravel().view(np.complex128) for x in (d, d2))
        got = complex(*res.cpu().tolist())
        assert abs(got - np.vdot(z, z2)) <= 1e-12 * np.abs(z).sum() * np.abs(z2).max(), (nc, n)
    qla.check("padded slots")


ADJOINT = ["M_veq_Ma", "M_vpeq_Ca_times_Ma", "M_vmeq_C_times_Ma", "M_veqm_c_times_Ma", "M_vpeq_r_times_Ma"]


@pytest.mark.parametrize("pc", ["F3", "D3"])
def test_adjoint_forms(qla, cuda, pc):
    byname = {e["name"]: e for e in qla.manifest()}
    rng = np.random.default_rng(61)
    dt = np.float32 if pc == "F3" else np.float64
    for n in SIZES + [2051]:
        for short in ADJOINT:
            e = byname[f"QLA_{pc}_{short}"]
            ins, idx, gang = T.ewise_inputs(e, rng, dt, n, n)
            want = T.ewise_oracle(e, ins, idx, gang, n)
            for off in (0, 4, 8) if pc == "F3" else (0, 8):  # bytes past a 16-B boundary
                assert T.bits_equal(_call(qla, cuda, e["name"], [], e, ins, n, off), want), (short, n, off)


@pytest.mark.parametrize("pc,dt", [("F3", np.float32), ("D3", np.float64)])
def test_small_field_tiles(qla, cuda, pc, dt):
    """Volumes on both sides of the points where the tile size changes (the
    64-site tiles, one usual tile per SM, one 64-site tile per SM of a
    reduction) and with partial last tiles."""
    sms = qla.lib().qlagpu_sm_count()
    rng = np.random.default_rng(5)
    top = 256 * sms + 65
    a, b = T.haar_su3(rng, top, dt), T.gaussian_field(rng, top, 3, dt)
    ad, bd = T.to_dev(a), T.to_dev(b)
    h = T.positive_hermitian_inputs(rng, top, dt)
    hd = T.to_dev(h)
    ns_ = getattr(qla, pc)
    want = np.zeros((top, 6), dt)
    T.ora_lmult(want, a, b, top, 1, "eq")
    for n in (1, 63, 64, 65, 64 * sms - 1, 64 * sms, 64 * sms + 33, 128 * sms, 256 * sms - 1, 256 * sms, top):
        rd = T.to_dev(np.zeros((top, 6), dt))
        ns_.V_veq_M_times_V(rd, ad, bd, n)
        got = T.to_host(rd)
        assert T.bits_equal(got[:n], want[:n]) and not got[n:].any(), n
        nrm = getattr(qla, "DF3" if pc == "F3" else "D3").r_veq_norm2_V(None, bd, n)
        exact = T.ora_norm2(b, n, 3, exact=True)
        assert abs(nrm - exact) <= 1e-12 * exact, n
        xd = T.to_dev(np.zeros((top, 18), dt))
        ns_.M_veq_inverse_M(xd, hd, n)
        inv = T.to_host(xd)
        if n <= 64 * sms:
            assert T.bits_equal(inv[:n], T.ora_mfunc(np.ascontiguousarray(h[:n]), n, "inverse")), n
        assert not inv[n:].any(), n


@pytest.mark.parametrize("pc,dt", [("F3", np.float32), ("D3", np.float64)])
@pytest.mark.parametrize("n", [63, 65, 18943, 18945, 19071, 37889])
def test_register_limited_operators_take_smaller_tiles(qla, pc, dt, n):
    """Matrix functions whose registers limit the blocks on an SM, contiguous and
    through a pointer array, around one and two 128-site tiles per SM."""
    rng = np.random.default_rng(91 + n)
    a = T.positive_hermitian_inputs(rng, n, np.float64).astype(dt)
    idx = rng.permutation(n).astype(np.int32)
    ns_ = getattr(qla, pc)
    a_d = T.to_dev(a)
    ptrs = T.ptr_array(a_d, idx, 9 * 2 * np.dtype(dt).itemsize)
    for fname in ("sqrt", "invsqrt"):
        r = T.to_dev(np.zeros_like(a))
        getattr(ns_, f"M_veq_{fname}_M")(r, a_d, n)
        want = T.ora_mfunc(a, n, fname)
        assert T.bits_equal(T.to_host(r), want), fname
        getattr(ns_, f"M_veq_{fname}_pM")(r, ptrs, n)
        assert T.bits_equal(T.to_host(r), want[idx]), fname + " pM"


@pytest.mark.parametrize("pc", ["F3", "D3"])
def test_partial_tiles_of_propagators(qla, cuda, pc):
    """Fields whose last tile of 32 sites is nearly empty, nearly full or the only
    one, on and off a 16-B boundary (P records: one bulk copy per lane)."""
    byname = {e["name"]: e for e in qla.manifest()}
    rng = np.random.default_rng(83)
    dt = np.float32 if pc == "F3" else np.float64
    for n in (1, 2, 31, 33, 63, 3000):
        for short in ("R_veq_re_P_dot_P", "R_vpeq_norm2_P", "C_veq_P_dot_P", "C_vmeq_P_dot_Pa", "C_veq_Pa_dot_P"):
            e = byname[f"QLA_{pc}_{short}"]
            ins, idx, gang = T.ewise_inputs(e, rng, dt, n, n)
            want = T.ewise_oracle(e, ins, idx, gang, n)
            for off in (0, 8):
                assert T.bits_equal(_call(qla, cuda, e["name"], [], e, ins, n, off), want), (short, n, off)


@pytest.mark.parametrize("pc,nc", [("F", 3), ("D", 3), ("F3", 3), ("D3", 3), ("FN", 2), ("DN", 2)])
def test_local_products_of_short_records(qla, cuda, pc, nc):
    """Records of 8 to 48 B around 65,536 sites, where the longer ones change kernel."""
    byname = {e["name"]: e for e in qla.manifest()}
    rng = np.random.default_rng(87 + nc)
    dt = np.float32 if pc[0] == "F" else np.float64
    L = qla.lib()
    for n in (65535, 65536, 65537):
        for letter in ("C",) if len(pc) == 1 else ("V", "H"):
            ne = {"C": 1, "V": nc, "H": 2 * nc}[letter]
            a, b = T.gaussian_field(rng, n, ne, dt), T.gaussian_field(rng, n, ne, dt)
            x, y = a.astype(np.float64), b.astype(np.float64)
            lead = [nc] if pc[1:] == "N" else []
            for short, want in ((f"R_veq_norm2_{letter}", (x, x)), (f"R_veq_re_{letter}_dot_{letter}", (x, y))):
                assert f"QLA_{pc}_{short}" in byname
                r = T.to_dev(np.zeros(n, dt))
                keep = [T.to_dev(a), T.to_dev(b)]
                args = [T.ptr_dev(r), T.ptr_dev(keep[0])] + ([T.ptr_dev(keep[1])] if "re_" in short else [])
                getattr(L, f"QLA_{pc}_{short}")(*lead, *args, n)
                s = np.zeros(n)
                for e in range(ne):  # the reference's order, in double
                    s = s + (want[0][:, 2 * e] * want[1][:, 2 * e] + want[0][:, 2 * e + 1] * want[1][:, 2 * e + 1])
                assert T.bits_equal(T.to_host(r), s.astype(dt)), (pc, short, n)
    qla.check("short records")


@pytest.mark.parametrize("pc", ["F3", "D3"])
def test_adjoint_and_outer_forms_change_kernel_with_size(qla, cuda, pc):
    byname = {e["name"]: e for e in qla.manifest()}
    rng = np.random.default_rng(67)
    dt = np.float32 if pc == "F3" else np.float64
    top = 128 * qla.lib().qlagpu_sm_count()
    for n in (top, top + 1, top + 33):
        for short in ADJOINT + ["M_veq_V_times_Va", "M_vmeq_V_times_Va"]:
            e = byname[f"QLA_{pc}_{short}"]
            ins, idx, gang = T.ewise_inputs(e, rng, dt, n, n)
            want = T.ewise_oracle(e, ins, idx, gang, n)
            for off in (0, 8):
                assert T.bits_equal(_call(qla, cuda, e["name"], [], e, ins, n, off), want), (short, n, off)
