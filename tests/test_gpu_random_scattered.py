"""Random fills through scattered states in fields larger than the L2, where
fewer blocks run (each thread then takes several sites): the same records and
states as the contiguous fill of the same states, which the oracle checks."""
import ctypes

import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc,dest,n", [("F3", "D", 950000), ("D3", "D", 540000), ("F3", "V", 2100000)])
def test_large_scattered_fills_equal_contiguous_ones(qla, cuda, pc, dest, n):
    ns_ = getattr(qla, pc)
    dt = cuda.float32 if pc == "F3" else cuda.float64
    nreal = 2 * T.NCPLX3[dest]
    assert n * (nreal * (4 if pc == "F3" else 8) + 44) > 126e6
    g = cuda.Generator(device="cuda").manual_seed(5)
    states = cuda.randint(0, 1 << 24, (n, 11), dtype=cuda.int32, device="cuda", generator=g)
    perm = cuda.randperm(n, device="cuda", generator=g)
    # contiguous: record i from state perm[i]
    s1 = states[perm].contiguous()
    r1 = cuda.zeros((n, nreal), dtype=dt, device="cuda")
    getattr(ns_, f"{dest}_veq_gaussian_S")(r1, s1, n)
    # the same through pointers
    s2, r2 = states.clone(), cuda.zeros_like(r1)
    ptrs = s2.data_ptr() + perm * 44
    getattr(ns_, f"{dest}_veq_gaussian_pS")(r2, ptrs, n)
    assert cuda.equal(r1.view(cuda.int32), r2.view(cuda.int32)) and cuda.equal(s2[perm], s1)
    # a gang index: every second site, states in place
    gang = cuda.arange(0, n, 2, dtype=cuda.int32, device="cuda")
    s3, r3 = s1.clone(), cuda.zeros_like(r1)
    s3[:] = states[perm]
    getattr(ns_, f"{dest}_xeq_gaussian_S")(r3, s3, gang, gang.numel())
    assert cuda.equal(r3[::2].contiguous().view(cuda.int32), r1[::2].contiguous().view(cuda.int32))
    assert not r3[1::2].any() and cuda.equal(s3[::2], s1[::2]) and cuda.equal(s3[1::2], states[perm][1::2])


def test_first_records_of_a_large_fill_match_the_oracle(qla):
    rng = np.random.default_rng(19)
    n, m = 950000, 2000
    st = np.zeros((n, 11), np.uint32)
    st[:m] = T.rng_states(rng, m)
    st[m:] = st[:m][rng.integers(0, m, n - m)]
    idx = np.arange(n)[::-1].astype(np.int32)  # record i from state n - 1 - i
    sd, rd = T.to_dev(st.view(np.int32)), T.to_dev(np.zeros((n, 24), np.float32))
    qla.F3.D_veq_gaussian_pS(rd, T.ptr_array(sd, idx, 44), n)
    want_s, want = st[idx[:m]].copy(), np.zeros((m, 24), np.float32)
    T.oracle().ora_rng_fill_f(24, 1, 0, T.ptr(want), T.ptr(want_s), ctypes.c_long(m), None, None)
    got = rd[:m].cpu().numpy().ravel()
    w = want.ravel()
    assert np.all(np.abs(got.astype(np.float64) - w) <= np.spacing(np.abs(w)))  # one float ulp
    assert np.array_equal(T.to_host(sd)[idx[:m]].view(np.uint32), want_s)
