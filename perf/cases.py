"""Performance cases: the level-1 work that lattice programs have this library do.

Every case runs through the C entry points of libqla_b200.so on device
arrays, called as a compiled program calls them: the argument lists are made
once in prepare(), and one pass of run() issues the case's calls in order on
the default stream.  Extents are those of the test and benchmark lattices,
or generic; draw() gives other lattices of the same ranges, odd and ragged
extents among them.
"""
import ctypes
import math

import torch

import qla_b200 as qla

# ---------------------------------------------------------------------------
# the cases


def listed():
    return [
        # the smallest lattices (tests, multigrid coarse levels, thermalisation
        # runs): 24 short calls, launch latency counts
        _lat("hop_8x8x8x8_f3", "hop", "F3", (8, 8, 8, 8), form="steps"),
        # the Wilson hop as separate level-1 calls on a production lattice
        _lat("hop_32x32x32x64_f3", "hop", "F3", (32, 32, 32, 64), form="steps"),
        # the even-odd preconditioned Wilson hop as a data-parallel layer calls
        # it: fused terms, neighbour pointers, a subset index, half the sites
        _lat("hop_eo_32x32x32x64_f3", "hop", "F3", (32, 32, 32, 64), form="subset"),
        # a staggered operator in double precision (forward and backward
        # multi-direction sums through pointers) on a ragged lattice
        _lat("staggered_21x25x27x45_d3", "staggered", "D3", (21, 25, 27, 45)),
        # a solver's vector updates and inner products: the largest lattice
        _lat("cg_48x48x48x96_f3", "cg", "F3", (48, 48, 48, 96), result="device"),
        # many fields of uneven volume, the same two-step sequence on each
        {"name": "batch_pairs_64", "kind": "batch", "mix": "pairs", "fields": 64, "lattices": 4, "emin": 8, "emax": 32},
        # many fields of uneven volume, each with its own sequence: link
        # products, hop terms, vector updates, staples
        {"name": "batch_mixed_48", "kind": "batch", "mix": "mixed", "fields": 48, "lattices": 7, "emin": 8, "emax": 26},
        # one gauge-link update: plaquette, its antihermitian part, exp,
        # reunitarisation
        _lat("links_24x24x24x48_f3", "links", "F3", (24, 24, 24, 48)),
        # colour-matrix functions in double precision (smeared-link
        # reunitarisation and its derivatives)
        _lat("mfunc_24x24x24x48_d3", "mfunc", "D3", (24, 24, 24, 48)),
        # propagator contractions
        _lat("prop_16x16x16x32_f3", "prop", "F3", (16, 16, 16, 32)),
        # stochastic estimator: noise fill, site-local products and norms
        _lat("noise_24x24x24x48_f3", "noise", "F3", (24, 24, 24, 48)),
        # the N-colour library at four colours
        _lat("ncolor4_20x20x20x40_fn", "ncolor", "FN", (20, 20, 20, 40), nc=4),
    ]


# most sites that draw() gives a kind (F3; half for D3)
_MOST = {"hop": 2097152, "staggered": 2097152, "cg": 4194304, "links": 663552, "mfunc": 663552, "prop": 131072,
         "noise": 663552, "ncolor": 320000}


def _lat(name, kind, pc, dims, **more):
    c = {"name": name, "kind": kind, "pc": pc, "lx": dims[0], "ly": dims[1], "lz": dims[2], "lt": dims[3]}
    c.update(more)
    return c


def draw(rng):
    kind = rng.choice(["hop", "hop", "staggered", "cg", "batch", "links", "mfunc", "prop", "noise", "ncolor"])
    if kind == "batch":
        emin = rng.randint(3, 9)
        return {"kind": "batch", "mix": rng.choice(["pairs", "mixed", "hops"]), "fields": rng.randint(5, 60),
                "lattices": rng.randint(100, 10 ** 6), "emin": emin, "emax": rng.randint(emin + 3, 25)}
    pc = "FN" if kind == "ncolor" else rng.choice(["F3", "D3"])
    more = {}
    if kind == "hop":
        more["form"] = rng.choice(["steps", "fused", "subset"])
    elif kind == "cg":
        more["result"] = rng.choice(["device", "host"])
    elif kind == "ncolor":
        more["nc"] = rng.choice([2, 4, 8])
    most = _MOST[kind] // (2 if pc == "D3" else 1)
    if kind == "ncolor":
        most = most * 16 // max(16, more["nc"] ** 2)
    sites = math.exp(rng.uniform(math.log(300), math.log(0.8 * most)))
    side = sites ** 0.25
    lx, ly, lz = (max(2, round(side * rng.uniform(0.75, 1.25))) for _ in range(3))
    lt = max(2, int(sites / (lx * ly * lz)))
    c = _lat("", kind, pc, (lx, ly, lz, lt), **more)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs, from the seed alone


def _dims(c):
    return [c["lx"], c["ly"], c["lz"], c["lt"]]


def _vol(dims):
    return dims[0] * dims[1] * dims[2] * dims[3]


def _real(pc):
    return torch.float64 if pc[0] == "D" else torch.float32


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(7919 * seed + 17)
    return g


def _gauss(g, n, ncplx, dt):
    """n records of ncplx complex N(0,1) numbers: [n, 2 ncplx] reals."""
    return torch.randn(n, 2 * ncplx, generator=g, device="cuda", dtype=dt)


def _field(z, dt):
    return torch.view_as_real(z).reshape(z.shape[0], -1).to(dt).contiguous()


def _su3(g, n, dt):
    """Random unitary 3x3 links (Gram-Schmidt rows, unit determinant)."""
    z = torch.view_as_complex(torch.randn(n, 2, 3, 2, generator=g, device="cuda", dtype=torch.float64 if dt ==
                                          torch.float64 else torch.float32))
    a = z[:, 0] / z[:, 0].abs().square().sum(1, keepdim=True).sqrt()
    b = z[:, 1] - (a.conj() * z[:, 1]).sum(1, keepdim=True) * a
    b = b / b.abs().square().sum(1, keepdim=True).sqrt()
    c = torch.linalg.cross(a, b).conj()
    return _field(torch.stack([a, b, c], 1).reshape(n, 9), dt)


def _neighbour(dims, mu, sign):
    """int32 table of x + sign mu on the periodic lattice, x0 fastest."""
    n = _vol(dims)
    i = torch.arange(n, device="cuda", dtype=torch.int64)
    stride = 1
    for k in range(mu):
        stride *= dims[k]
    x = (i // stride) % dims[mu]
    return (i + ((x + sign) % dims[mu] - x) * stride).to(torch.int32)


def _even(dims):
    i = torch.arange(_vol(dims), device="cuda", dtype=torch.int64)
    par = torch.zeros_like(i)
    stride = 1
    for d in dims:
        par += (i // stride) % d
        stride *= d
    return torch.nonzero(par % 2 == 0).flatten().to(torch.int32).contiguous()


def _pointers(t, idx):
    """Device array of record addresses t[idx[i]] (the pointer operands)."""
    return (t.data_ptr() + idx.long() * (t.shape[1] * t.element_size())).contiguous()


def _lattice_list(c):
    """The batch's lattices: extents from a fixed generator, by the case alone."""
    x, out = c["lattices"] * 2654435761 % 4294967296, []
    for _ in range(c["fields"]):
        d = []
        for _ in range(4):
            x = (1664525 * x + 1013904223) % 4294967296
            d.append(c["emin"] + (x >> 8) % (c["emax"] - c["emin"] + 1))
        out.append(d)
    return out


_MIXES = {"pairs": ("pair",), "hops": ("hop",), "mixed": ("pair", "hop", "axpy", "mma", "staple")}


def _batch_kinds(c):
    m = _MIXES[c["mix"]]
    return [m[k % len(m)] for k in range(c["fields"])]


def _inputs(c, seed):
    g = _gen(seed)
    kind = c["kind"]
    if kind == "batch":
        fields = []
        for k, (dims, what) in enumerate(zip(_lattice_list(c), _batch_kinds(c))):
            n, f = _vol(dims), {"what": what, "n": _vol(dims), "nbr": _neighbour(dims, k % 4, 1 if k % 3 else -1)}
            dt = torch.float32
            f["u"] = _su3(g, n, dt)
            if what in ("pair", "mma", "staple"):
                f["u2"] = _su3(g, n, dt)
            if what == "pair":
                f["v"] = _gauss(g, n, 3, dt)
            if what in ("hop", "axpy"):
                f["d"], f["o"] = _gauss(g, n, 12, dt), _gauss(g, n, 12, dt)
            if what == "mma":
                f["q"] = _gauss(g, n, 9, dt)
            f["mu"], f["sign"], f["r"] = k % 4, 1 if k % 2 else -1, 0.25 + 0.01 * k
            fields.append(f)
        return {"fields": fields}
    dims, pc = _dims(c), c["pc"]
    n, dt = _vol(dims), _real(pc)
    s = {"n": n}
    if kind == "hop":
        s["u"] = [_su3(g, n, dt) for _ in range(4)]
        s["d"] = _gauss(g, n, 12, dt)
        s["nbr"] = {(mu, sg): _neighbour(dims, mu, sg) for mu in range(4) for sg in (1, -1)}
        if c["form"] == "subset":
            s["even"] = _even(dims)
            s["o"] = _gauss(g, n, 12, dt)
    elif kind == "staggered":
        s["u"] = [_su3(g, n, dt) for _ in range(4)]
        s["v"] = _gauss(g, n, 3, dt)
        s["nbr"] = {(mu, sg): _neighbour(dims, mu, sg) for mu in range(4) for sg in (1, -1)}
    elif kind == "cg":
        s["x"], s["p"] = _gauss(g, n, 12, dt), _gauss(g, n, 12, dt)
    elif kind == "links":
        s["u"] = [_su3(g, n, dt) for _ in range(2)]
        s["nbr"] = [_neighbour(dims, 0, 1), _neighbour(dims, 1, 1)]
    elif kind == "mfunc":
        z = torch.view_as_complex(torch.randn(n, 3, 3, 2, generator=g, device="cuda", dtype=torch.float64)) * 0.5
        h = z.conj().transpose(1, 2) @ z + 0.1 * torch.eye(3, device="cuda", dtype=z.dtype)
        lo = torch.complex64 if dt == torch.float32 else torch.complex128
        h = h.to(lo)
        s["h"] = _field((0.5 * (h + h.conj().transpose(1, 2))).reshape(n, 9), dt)
        s["m"] = _gauss(g, n, 9, dt)
        s["v"] = _gauss(g, n, 3, dt)
    elif kind == "prop":
        s["m"] = _su3(g, n, dt)
        s["a"], s["b"] = _gauss(g, n, 144, dt), _gauss(g, n, 144, dt)
    elif kind == "noise":
        s["seeds"] = torch.arange(n, device="cuda", dtype=torch.int32)
        s["seed"] = 1000 + seed
        s["d"] = _gauss(g, n, 12, dt)
        s["m"], s["cf"] = _gauss(g, n, 9, dt), _gauss(g, n, 1, dt)
        s["p"] = _gauss(g, n // 8 + 1, 144, dt)
    else:
        nc = c["nc"]
        z = torch.view_as_complex(torch.randn(n, nc, nc, 2, generator=g, device="cuda", dtype=torch.float64))
        z = (0.5 / nc) * (z - z.conj().transpose(1, 2))
        s["q"] = _field(z.reshape(n, nc * nc), dt)
        s["m"], s["m2"] = _gauss(g, n, nc * nc, dt), _gauss(g, n, nc * nc, dt)
        s["v"] = _gauss(g, n, nc, dt)
        s["d"], s["d2"] = _gauss(g, n, 4 * nc, dt), _gauss(g, n, 4 * nc, dt)
        s["nbr"] = _neighbour(dims, 1, 1)
        s["c"] = torch.tensor([0.3, -0.7], device="cuda", dtype=dt)
    return s


# ---------------------------------------------------------------------------
# prepare: buffers, argument lists, plans


class _Int(int):
    """An argument passed as a C int (everything else is an address)."""


class _Calls(list):
    def add(self, name, *args):
        fn = getattr(qla.lib(), name)
        fn.restype = None
        self.append((fn, tuple(_arg(a) for a in args)))


def _arg(a):
    if isinstance(a, _Int):
        return ctypes.c_int(a)
    if isinstance(a, torch.Tensor):
        return ctypes.c_void_p(a.data_ptr())
    return a  # a ctypes object of the caller's


def prepare(case, seed):
    c = case
    s = _inputs(c, seed)
    if c["kind"] == "batch":
        return _prepare_batch(s)
    pc, n, dt = c["pc"], s["n"], _real(c["pc"])
    N, I = _Int(n), _Int
    calls, out = _Calls(), {}

    def new(ncplx, sites=n, like=dt):
        return torch.zeros(sites, 2 * ncplx, device="cuda", dtype=like)

    P = f"QLA_{pc}_"
    R = "QLA_DF3_" if pc == "F3" else P  # global reductions of F3 fields in double
    if c["kind"] == "hop":
        if c["form"] == "steps":
            o, h, h2 = new(12), new(6), new(6)
            first = True
            for mu in range(4):
                for sg in (1, -1):
                    calls.add(P + "H_veq_spproj_D", h, s["d"], I(mu), I(sg), N)
                    calls.add(P + "H_eq_M_times_xH", h2, s["u"][mu], h, s["nbr"][mu, sg], N)
                    calls.add(P + ("D_veq_sprecon_H" if first else "D_vpeq_sprecon_H"), o, h2, I(mu), I(sg), N)
                    first = False
            s["keep"] = (h, h2)
        elif c["form"] == "fused":
            o = new(12)
            first = True
            for mu in range(4):
                for sg in (1, -1):
                    calls.add(P + ("D_eq_spproj_M_times_xD" if first else "D_peq_spproj_M_times_xD"), o, s["u"][mu],
                              s["d"], s["nbr"][mu, sg], I(mu), I(sg), N)
                    first = False
        else:
            o = s["o"].clone()
            ev = s["even"]
            keep, first = [], True
            for mu in range(4):
                pd = _pointers(s["d"], s["nbr"][mu, 1])
                calls.add(P + ("D_xeq_spproj_M_times_pD" if first else "D_xpeq_spproj_M_times_pD"), o, s["u"][mu], pd,
                          I(mu), I(1), ev, I(len(ev)))
                first = False
                pb, pu = _pointers(s["d"], s["nbr"][mu, -1]), _pointers(s["u"][mu], s["nbr"][mu, -1])
                calls.add(P + "D_xpeq_spproj_pMa_times_pD", o, pu, pb, I(mu), I(-1), ev, I(len(ev)))
                keep += [pd, pb, pu]
            s["keep"] = keep
        out["o"] = o
    elif c["kind"] == "staggered":
        r = new(3)
        pf = [_pointers(s["v"], s["nbr"][mu, 1]) for mu in range(4)]
        pb = [_pointers(s["v"], s["nbr"][mu, -1]) for mu in range(4)]
        pu = [_pointers(s["u"][mu], s["nbr"][mu, -1]) for mu in range(4)]
        tab = [(ctypes.c_void_p * 4)(*[t.data_ptr() for t in ts]) for ts in (s["u"], pf, pu, pb)]
        calls.add(P + "V_veq_nM_times_npV", r, tab[0], tab[1], N, I(4))
        calls.add(P + "V_vmeq_npMa_times_npV", r, tab[2], tab[3], N, I(4))
        s["keep"] = (pf, pb, pu, tab)
        out["r"] = r
    elif c["kind"] == "cg":
        ct = ctypes.c_double if pc == "D3" else ctypes.c_float
        x, res = s["x"].clone(), []
        for k, a in enumerate(_CG):
            calls.add(P + "D_vpeq_r_times_D", x, ctypes.byref(ct(a)), s["p"], N)
            if c["result"] == "device":
                nr, dot = (torch.zeros(w, device="cuda", dtype=torch.float64) for w in (1, 2))
            else:
                nr, dot = (ctypes.c_double * 1)(), (ctypes.c_double * 2)()
            calls.add(R + "r_veq_norm2_D", nr, x, N)
            calls.add(R + "c_veq_D_dot_D", dot, s["p"], x, N)
            res += [nr, dot]
        out["x"], out["res"] = x, res
    elif c["kind"] == "links":
        u0, u1 = s["u"]
        t, w, f, q, e, u, v = (new(9) for _ in range(7))
        act = torch.zeros(1, device="cuda", dtype=torch.float64)
        calls.add(P + "M_eq_M_times_xM", t, u0, u1, s["nbr"][0], N)
        calls.add(P + "M_eq_M_times_xM", w, u1, u0, s["nbr"][1], N)
        calls.add(R + "r_veq_re_M_dot_M", act, t, w, N)
        calls.add(P + "M_veq_M_times_Ma", f, t, w, N)
        calls.add(P + "M_veq_antiherm_M", q, f, N)
        calls.add(P + "M_veq_exp_M", e, q, N)
        calls.add(P + "M_veq_M_times_M", u, e, u0, N)
        calls.add(f"qlagpu_{pc}_M_veq_reunit_M", v, u, N)
        s["keep"] = (t, w)
        out.update(action=act, f=f, q=q, e=e, u=u, v=v)
    elif c["kind"] == "mfunc":
        for name in ("sqrt", "invsqrt", "log", "sqrtPH", "invsqrtPH"):
            out[name] = new(9)
            calls.add(P + f"M_veq_{name}_M", out[name], s["h"], N)
        out["inverse"], out["det"], out["solve"] = new(9), new(1), new(3)
        calls.add(P + "M_veq_inverse_M", out["inverse"], s["m"], N)
        calls.add(P + "C_veq_det_M", out["det"], s["m"], N)
        calls.add(P + "V_veq_M_inverse_V", out["solve"], s["h"], s["v"], N)
    elif c["kind"] == "prop":
        mp, pm, pp, ap = (new(144) for _ in range(4))
        tr = new(9)
        dot = torch.zeros(2, device="cuda", dtype=torch.float64)
        calls.add(P + "P_veq_M_times_P", mp, s["m"], s["a"], N)
        calls.add(P + "P_veq_P_times_Ma", pm, s["a"], s["m"], N)
        calls.add(P + "P_veq_P_times_P", pp, s["a"], s["b"], N)
        calls.add(P + "P_veq_Pa_times_P", ap, s["a"], s["b"], N)
        calls.add(P + "M_veq_spintrace_P", tr, ap, N)
        calls.add(R + "c_veq_P_dot_P", dot, s["a"], s["b"], N)
        out.update(mp=mp, pm=pm, pp=pp, ap=ap, tr=tr, dot=dot)
    elif c["kind"] == "noise":
        st = torch.zeros(n, 11, device="cuda", dtype=torch.int32)
        fn = qla.lib().QLA_S_veq_seed_i_I
        fn(ctypes.c_void_p(st.data_ptr()), ctypes.c_int(s["seed"]), ctypes.c_void_p(s["seeds"].data_ptr()),
           ctypes.c_int(n))
        eta, loc = new(12), new(1)
        nd, npr = (torch.zeros(k, device="cuda", dtype=dt) for k in (n, len(s["p"])))
        ma, ou, np8 = new(9), new(9), _Int(len(s["p"]))
        v1, v2 = new(3), new(3)
        calls.add(P + "D_veq_gaussian_S", eta, st, N)
        calls.add(P + "V_veq_colorvec_D", v1, eta, I(1), N)
        calls.add(P + "V_veq_colorvec_D", v2, s["d"], I(2), N)
        calls.add(P + "C_veq_D_dot_D", loc, eta, s["d"], N)
        calls.add(P + "R_veq_norm2_D", nd, s["d"], N)
        calls.add(P + "R_veq_norm2_P", npr, s["p"], np8)
        calls.add(P + "M_veq_V_times_Va", ou, v1, v2, N)
        calls.add(P + "M_veq_Ca_times_Ma", ma, s["cf"], s["m"], N)
        s["keep"] = (v1, v2)
        out.update(state=st, eta=eta, loc=loc, nd=nd, np=npr, ou=ou, ma=ma)
    else:
        nc = c["nc"]
        v, mm, z, q = new(nc), new(nc * nc), new(4 * nc), new(nc * nc)
        loc, dot = new(1), torch.zeros(2, device="cuda", dtype=torch.float64)
        C = I(nc)
        calls.add(P + "V_eq_M_times_xV", C, v, s["m"], s["v"], s["nbr"], N)
        calls.add(P + "M_veq_M_times_Ma", C, mm, s["m"], s["m2"], N)
        calls.add(P + "D_veq_c_times_D_plus_D", C, z, s["c"], s["d"], s["d2"], N)
        calls.add(P + "C_veq_D_dot_D", C, loc, s["d"], s["d2"], N)
        calls.add("QLA_DFN_c_veq_D_dot_D", C, dot, s["d"], s["d2"], N)
        calls.add(P + "M_veq_exp_M", C, q, s["q"], N)
        out.update(v=v, mm=mm, z=z, loc=loc, dot=dot, q=q)
    s["calls"], s["out"] = calls, out
    return s


_CG = (0.37, -0.21)  # the step lengths of the two iterations of a pass


def _prepare_batch(s):
    progs, arena = [], _Arena(s["fields"], torch.float32)
    R0, R1 = qla.REG0, qla.REG1
    for f in s["fields"]:
        n = f["n"]

        def new(ncplx, like=None):
            t = arena.take(n, ncplx)
            return t if like is None else t.copy_(like)

        def st(base, kind, role="in", index=None):
            d = {"base": base, "kind": kind, "role": role}
            if index is not None:
                d["index"], d["nsrc"] = index, n
            return d

        if f["what"] == "pair":  # r = u u2[x+mu], w = r v
            r, w = new(9), new(3)
            streams = [st(f["u"], "M"), st(f["u2"], "M", index=f["nbr"]), st(f["v"], "V"), st(r, "M", "out"),
                       st(w, "V", "out")]
            steps = [{"op": "lmult", "a": 0, "b": 1, "dst": R0, "store": 3},
                     {"op": "lmult", "a": R0, "b": 2, "dst": R1, "store": 4}]
        elif f["what"] == "hop":  # o += sprecon(u spproj(d[x+mu]))
            o = new(12, f["o"])
            streams = [st(f["u"], "M"), st(f["d"], "D", index=f["nbr"]), st(o, "D", "inout")]
            steps = [{"op": "spproj", "a": 1, "dst": R0, "mu": f["mu"], "sign": f["sign"]},
                     {"op": "lmult", "a": 0, "b": R0, "dst": R1},
                     {"op": "sprecon", "eqop": "peq", "a": R1, "dst": R0, "store": 2, "mu": f["mu"],
                      "sign": f["sign"]}]
        elif f["what"] == "axpy":  # o += r d, w = u^+ o
            o, w = new(12, f["o"]), new(12)
            streams = [st(f["d"], "D"), st(f["u"], "M"), st(o, "D", "inout"), st(w, "D", "out")]
            steps = [{"op": "rtimes", "eqop": "peq", "a": 0, "dst": R0, "store": 2, "r": f["r"]},
                     {"op": "lmult", "a": 1, "b": R0, "dst": R1, "store": 3, "adja": 1}]
        elif f["what"] == "mma":  # r = u u2^+, q -= r
            r, q = new(9), new(9, f["q"])
            streams = [st(f["u"], "M"), st(f["u2"], "M"), st(r, "M", "out"), st(q, "M", "inout")]
            steps = [{"op": "lmult", "a": 0, "b": 1, "dst": R0, "store": 2, "adjb": 1},
                     {"op": "copy", "eqop": "meq", "a": R0, "dst": R1, "store": 3}]
        else:  # staple: r = u u2[x+mu], w = r u^+
            r, w = new(9), new(9)
            streams = [st(f["u"], "M"), st(f["u2"], "M", index=f["nbr"]), st(r, "M", "out"), st(w, "M", "out")]
            steps = [{"op": "lmult", "a": 0, "b": 1, "dst": R0, "store": 2},
                     {"op": "lmult", "a": R0, "b": 0, "dst": R1, "store": 3, "adjb": 1}]
        progs.append({"n": n, "streams": streams, "steps": steps})
    s["plan"] = qla.BatchProgramPlan(progs)
    s["out"] = arena.whole
    return s


class _Arena:
    """One array per record length that holds all output fields of a batch, in
    the fields' order, each padded to a multiple of 16 sites."""

    LENGTHS = {"pair": (9, 3), "hop": (12,), "axpy": (12, 12), "mma": (9, 9), "staple": (9, 9)}

    def __init__(self, fields, dt):
        rows = {}
        for f in fields:
            for k in self.LENGTHS[f["what"]]:
                rows[k] = rows.get(k, 0) + (f["n"] + 15) // 16 * 16
        self.whole = {"r%d" % k: torch.zeros(n, 2 * k, device="cuda", dtype=dt) for k, n in rows.items()}
        self.at = dict.fromkeys(rows, 0)

    def take(self, n, ncplx):
        a = self.at[ncplx]
        self.at[ncplx] = a + (n + 15) // 16 * 16
        return self.whole["r%d" % ncplx][a:a + n]


def run(state):
    if "plan" in state:
        state["plan"].run()
        return state["out"]
    for fn, args in state["calls"]:
        fn(*args)
    out = state["out"]
    if "res" in out:
        return {"x": out["x"], "res": [r if isinstance(r, torch.Tensor) else list(r) for r in out["res"]]}
    return out


# ---------------------------------------------------------------------------
# work: bytes and floating-point operations per site of each call


def work(case):
    c = case
    if c["kind"] == "batch":
        b = {"pair": 268, "hop": 364, "axpy": 456, "mma": 360, "staple": 292}
        fl = {"pair": 288, "hop": 264 + 24, "axpy": 48 + 288, "mma": 216 + 18, "staple": 432}
        kinds, lats = _batch_kinds(c), _lattice_list(c)
        return {"bytes": sum(b[k] * _vol(d) for k, d in zip(kinds, lats)),
                "flops": sum(fl[k] * _vol(d) for k, d in zip(kinds, lats))}
    n = _vol(_dims(c))
    z = 16 if c["pc"][0] == "D" else 8  # bytes of a complex number
    if c["kind"] == "hop":
        if c["form"] == "steps":
            by, fl = 8 * ((18 + 21 + 30) * z + 4) - 12 * z, 8 * (24 + 144 + 24)
        elif c["form"] == "fused":
            by, fl = 8 * (45 * z + 4) - 12 * z, 8 * 192
        else:  # half the sites: index 4, pointers 8 (forward) or 16 (backward)
            by, fl = (8 * (45 * z + 4) - 12 * z + 4 * 8 + 4 * 16) // 2, 4 * 192
    elif c["kind"] == "staggered":
        by, fl = 2 * 4 * (12 * z + 8) + 4 * 8 + 3 * 3 * z, 8 * 72
    elif c["kind"] == "cg":
        by, fl = 2 * 72 * z, 2 * (48 + 48 + 96)
    elif c["kind"] == "links":
        by, fl = (27 * 2 + 18 + 27 + 18 + 18 + 27 + 18) * z + 8, 4 * 216 + 36 + 1000 + 700
    elif c["kind"] == "mfunc":
        by, fl = (5 * 18 + 18 + 10 + 15) * z, 3 * 3000 + 2 * 700 + 300
    elif c["kind"] == "prop":
        by, fl = (2 * (9 + 288) + 2 * 432 + 153 + 288) * z, 2 * 432 * 8 + 2 * 1728 * 8 + 1152
    elif c["kind"] == "noise":
        by, fl = 88 + (12 + 2 * 15 + 25 + 12.5 + 18 + 15 + 19) * z + 144.5 * z / 8, 12 * 80 + 96 + 48 + 72 + 72
    else:
        nc = c["nc"]
        by = (nc * nc + 2 * nc + 3 * nc * nc + 12 * nc + 8 * nc + 1 + 8 * nc + 2 * nc * nc) * z + 4
        fl = 8 * nc * nc + 8 * nc ** 3 + 32 * nc * 3 + 8 * nc ** 3 * 12
    return {"bytes": n * by, "flops": n * fl}


# ---------------------------------------------------------------------------
# exact: the same results in 64 bits, plain torch

# spin components of the projection (value = first + coefficient * second) and
# of the reconstruction (coefficient, half-spin), by (mu, sign)
_PROJ = {(0, 1): ((0, 1j, 3), (1, 1j, 2)), (0, -1): ((0, -1j, 3), (1, -1j, 2)),
         (1, 1): ((0, -1, 3), (1, 1, 2)), (1, -1): ((0, 1, 3), (1, -1, 2)),
         (2, 1): ((0, 1j, 2), (1, -1j, 3)), (2, -1): ((0, -1j, 2), (1, 1j, 3)),
         (3, 1): ((0, 1, 2), (1, 1, 3)), (3, -1): ((0, -1, 2), (1, -1, 3))}
_RECON = {(0, 1): ((-1j, 1), (-1j, 0)), (0, -1): ((1j, 1), (1j, 0)),
          (1, 1): ((1, 1), (-1, 0)), (1, -1): ((-1, 1), (1, 0)),
          (2, 1): ((-1j, 0), (1j, 1)), (2, -1): ((1j, 0), (-1j, 1)),
          (3, 1): ((1, 0), (1, 1)), (3, -1): ((-1, 0), (-1, 1))}


def _z(x, *shape):
    x = x.double().reshape(x.shape[0], -1, 2)
    return torch.view_as_complex(x.contiguous()).reshape(x.shape[0], *shape)


def _r(z):
    return torch.view_as_real(z.contiguous()).reshape(z.shape[0], -1)


def _proj(d, mu, sg):
    """[n, 3, 4] -> [n, 3, 2]"""
    return torch.stack([d[:, :, a] + k * d[:, :, b] for a, k, b in _PROJ[mu, sg]], 2)


def _recon(h, mu, sg):
    return torch.cat([h, torch.stack([k * h[:, :, s] for k, s in _RECON[mu, sg]], 2)], 2)


def _dag(m):
    return m.conj().transpose(-1, -2)


def _mm(a, b):
    """Batched product as sums of broadcast products."""
    o = a[:, :, 0, None] * b[:, None, 0, :]
    for k in range(1, a.shape[2]):
        o = o + a[:, :, k, None] * b[:, None, k, :]
    return o


def exact(case, seed):
    c = case
    s = _inputs(c, seed)
    kind = c["kind"]
    if kind == "batch":
        return _exact_batch(s)
    if kind == "hop":
        d = _z(s["d"], 3, 4)
        o = torch.zeros_like(d)
        for mu in range(4):
            u = _z(s["u"][mu], 3, 3)
            for sg in (1, -1):
                nb = s["nbr"][mu, sg].long()
                if c["form"] == "subset" and sg < 0:
                    o += _recon(_mm(_dag(u[nb]), _proj(d[nb], mu, sg)), mu, sg)
                else:
                    o += _recon(_mm(u, _proj(d[nb], mu, sg)), mu, sg)
        if c["form"] == "subset":
            full = _z(s["o"], 3, 4)
            ev = s["even"].long()
            full[ev] = o[ev]
            o = full
        return {"o": _r(o)}
    if kind == "staggered":
        v = _z(s["v"], 3, 1)
        r = torch.zeros_like(v)
        for mu in range(4):
            u, nf, nb = _z(s["u"][mu], 3, 3), s["nbr"][mu, 1].long(), s["nbr"][mu, -1].long()
            r = r + _mm(u, v[nf]) - _mm(_dag(u[nb]), v[nb])
        return {"r": _r(r)}
    if kind == "cg":
        ct = torch.float64 if c["pc"] == "D3" else torch.float32
        x, p = s["x"].double(), s["p"].double()
        res = []
        for a in _CG:
            x += torch.tensor(a, dtype=ct).double().item() * p
            nr = (x * x).sum().reshape(1)
            re = (p * x).sum()
            im = (p[:, 0::2] * x[:, 1::2]).sum() - (p[:, 1::2] * x[:, 0::2]).sum()
            res += [nr, torch.stack([re, im])]
        if c["result"] == "host":
            res = [[float(v) for v in t] for t in res]
        return {"x": x, "res": res}
    if kind == "links":
        u0, u1 = _z(s["u"][0], 3, 3), _z(s["u"][1], 3, 3)
        t, w = _mm(u0, u1[s["nbr"][0].long()]), _mm(u1, u0[s["nbr"][1].long()])
        act = (t.conj() * w).real.sum().reshape(1)
        f = _mm(t, _dag(w))
        q = 0.5 * (f - _dag(f))
        q = q - torch.diagonal(q, dim1=1, dim2=2).sum(1)[:, None, None] / 3 * torch.eye(3, device="cuda")
        e = torch.linalg.matrix_exp(q)
        u = _mm(e, u0)
        v = u  # unitary in exact arithmetic
        return {"action": act, "f": _r(f), "q": _r(q), "e": _r(e), "u": _r(u), "v": _r(v)}
    if kind == "mfunc":
        h, m, v = _z(s["h"], 3, 3), _z(s["m"], 3, 3), _z(s["v"], 3, 1)
        part = [torch.linalg.eigh(x) for x in h.split(8192)]  # the batched solver takes limited batches
        w, q = torch.cat([x[0] for x in part]), torch.cat([x[1] for x in part])

        def of(x):
            return _r(_mm(q * x[:, None, :], _dag(q)))

        rt, irt = of(w.sqrt()), of(w.rsqrt())
        return {"sqrt": rt, "invsqrt": irt, "log": of(w.log()), "sqrtPH": rt, "invsqrtPH": irt,
                "inverse": _r(torch.linalg.inv(m)), "det": _r(torch.linalg.det(m)[:, None]),
                "solve": _r(_mm(_mm(q / w[:, None, :], _dag(q)), v))}
    if kind == "prop":
        n = s["n"]
        m, a, b = _z(s["m"], 3, 3), _z(s["a"], 12, 12), _z(s["b"], 12, 12)
        mp = _mm(m, a.reshape(n, 3, 48))
        pm = torch.einsum("nricj,ndc->nridj", a.reshape(n, 3, 4, 3, 4), m.conj())  # columns times m^+
        pp, ap = _mm(a, b), _mm(_dag(a), b)
        tr = torch.einsum("nisjs->nij", ap.reshape(n, 3, 4, 3, 4))
        dot = (a.conj() * b).sum()
        return {"mp": _r(mp), "pm": _r(pm), "pp": _r(pp), "ap": _r(ap), "tr": _r(tr),
                "dot": torch.stack([dot.real, dot.imag])}
    if kind == "noise":
        d, m, cf, p = _z(s["d"], 12), _z(s["m"], 3, 3), _z(s["cf"], 1), _z(s["p"], 144)
        # the deviates and what is made of them have no independent value here
        return {"state": None, "eta": None, "loc": None, "nd": d.abs().square().sum(1), "np": p.abs().square().sum(1),
                "ou": None, "ma": _r(cf.conj()[:, :, None] * _dag(m))}
    nc = c["nc"]
    m, m2, q = _z(s["m"], nc, nc), _z(s["m2"], nc, nc), _z(s["q"], nc, nc)
    v, d, d2 = _z(s["v"], nc, 1), _z(s["d"], 4 * nc), _z(s["d2"], 4 * nc)
    k = complex(*s["c"].double().tolist())
    loc = (d.conj() * d2).sum(1, keepdim=True)
    dot = loc.sum()
    return {"v": _r(_mm(m, v[s["nbr"].long()])), "mm": _r(_mm(m, _dag(m2))), "z": _r(k * d + d2), "loc": _r(loc),
            "dot": torch.stack([dot.real, dot.imag]), "q": _r(torch.linalg.matrix_exp(q))}


def _exact_batch(s):
    arena = _Arena(s["fields"], torch.float64)
    for f in s["fields"]:
        nb, u = f["nbr"].long(), _z(f["u"], 3, 3)
        r = torch.tensor(f["r"], dtype=torch.float32).double().item()
        if f["what"] == "pair":
            t = _mm(u, _z(f["u2"], 3, 3)[nb])
            got = [t, _mm(t, _z(f["v"], 3, 1))]
        elif f["what"] == "hop":
            h = _mm(u, _proj(_z(f["d"], 3, 4)[nb], f["mu"], f["sign"]))
            got = [_z(f["o"], 3, 4) + _recon(h, f["mu"], f["sign"])]
        elif f["what"] == "axpy":
            o = _z(f["o"], 3, 4) + r * _z(f["d"], 3, 4)
            got = [o, _mm(_dag(u), o)]
        elif f["what"] == "mma":
            t = _mm(u, _dag(_z(f["u2"], 3, 3)))
            got = [t, _z(f["q"], 3, 3) - t]
        else:
            t = _mm(u, _z(f["u2"], 3, 3)[nb])
            got = [t, _mm(t, _dag(u))]
        for t in got:
            x = _r(t)
            arena.take(f["n"], x.shape[1] // 2).copy_(x)
    return arena.whole
