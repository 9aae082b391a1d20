"""Random batched programs (qlagpu_F3_batch_plan_program) against the oracle's
functions applied step by step, bit for bit: registers read by later steps,
results that take the place of values read for the last time, INOUT streams
still read after their store, gathers, aligned and 8-B aligned fields, and
volumes at the edges of the 32-site tiles."""
import numpy as np
import pytest

import qla_testlib as T

pytestmark = pytest.mark.gpu

NC = {"V": 3, "H": 6, "D": 12, "M": 9}
NCOL = {"V": 1, "H": 2, "D": 4, "M": 3}
EQ = ["eq", "peq", "meq", "eqm"]


def _apply(step, val, n):
    """The step's result from the operand values, by the oracle."""
    op, eq, a = step["op"], step["eqop"], val["a"]
    kind = step["kind"]
    r = np.ascontiguousarray(val["old"]) if "old" in val else np.zeros((n, 2 * NC[kind]), np.float32)
    r = r.copy()
    if op == "lmult":
        T.ora_lmult(r, a, val["b"], n, NCOL[kind], eq, adja=step["adja"], adjb=step["adjb"])
    elif op == "spproj":
        T.ora_spproj(r, a, n, step["mu"], step["sign"], eq)
    elif op == "sprecon":
        T.ora_sprecon(r, a, n, step["mu"], step["sign"], eq)
    else:
        x = a if op == "copy" else np.float32(step["r"]) * a
        r = {"eq": x, "eqm": -x, "peq": r + x, "meq": r - x}[eq]
    return r


def _program(rng, qla, n):
    """A random valid program: (streams, steps); each step carries its result kind."""
    streams = [{"kind": "M", "role": "in", "gather": bool(rng.integers(2))}]
    for _ in range(int(rng.integers(1, 4))):
        streams.append({"kind": str(rng.choice(list("VHDM"))), "role": "in", "gather": bool(rng.integers(2))})
    for _ in range(int(rng.integers(0, 3))):
        streams.append({"kind": str(rng.choice(list("VHDM"))), "role": "inout", "gather": False})
    steps, regs, stored = [], {}, set()
    want = int(rng.integers(2, 9))
    while len(steps) < want or any(s["role"] != "in" and j not in stored for j, s in enumerate(streams)):
        refs = [(j, s["kind"]) for j, s in enumerate(streams) if s["role"] != "out"]
        refs += [(qla.REG0 + k, v) for k, v in regs.items()] * 2
        a, ka = refs[int(rng.integers(len(refs)))]
        ops = ["copy", "rtimes"] + {"M": ["lmult"] * 6, "D": ["spproj"] * 3, "H": ["sprecon"] * 3}.get(ka, [])
        st = {"op": str(rng.choice(ops)), "a": a, "b": 0, "adja": 0, "adjb": 0, "kind": ka, "r": float(rng.normal()),
              "mu": int(rng.integers(5)), "sign": int(rng.choice([1, -1]))}
        if st["op"] == "lmult":
            st["b"], st["kind"] = refs[int(rng.integers(len(refs)))]
            st["adja"] = int(rng.integers(2))
            st["adjb"] = int(rng.integers(2)) if st["kind"] == "M" else 0
        elif st["op"] in ("spproj", "sprecon"):
            st["kind"] = "H" if st["op"] == "spproj" else "D"
        dst = int(rng.integers(2))
        open_ = [j for j, s in enumerate(streams) if s["role"] != "in" and j not in stored and s["kind"] == st["kind"]]
        left = [j for j, s in enumerate(streams) if s["role"] != "in" and j not in stored]
        st["store"] = -1
        if open_:
            st["store"] = int(rng.choice(open_))
        elif len(streams) < 8 and rng.integers(2):
            streams.append({"kind": st["kind"], "role": "out", "gather": False})
            st["store"] = len(streams) - 1
        inout = st["store"] >= 0 and streams[st["store"]]["role"] == "inout"
        st["old"] = st["store"] if inout else (qla.REG0 + dst if regs.get(dst) == st["kind"] else None)
        st["eqop"] = str(rng.choice(EQ if st["old"] is not None else ["eq", "eqm"]))
        st["dst"] = qla.REG0 + dst
        if len(steps) == 8 or (len(steps) >= want and not open_ and left):
            return None  # an output of a kind that no step made: draw another program
        steps.append(st)
        regs[dst] = st["kind"]
        if st["store"] >= 0:
            stored.add(st["store"])
    return (streams, steps) if stored else None


@pytest.mark.parametrize("seed", range(6))
def test_random_programs_match_the_oracle(qla, cuda, seed):
    rng = np.random.default_rng(900 + seed)
    sizes = [1, 31, 32, 33, 64, 127, 0, 2049, 5000]
    progs, checks, keep = [], [], []
    while len(progs) < 24:
        n = sizes[len(progs) % len(sizes)]
        made = _program(rng, qla, n)
        if made is None:
            continue
        streams, steps = made
        off = 8 if len(progs) % 4 == 3 else 0  # bytes past a 16-B boundary
        cur, devs, spec = {}, [], []
        for s in streams:
            nsrc = n + 5
            host = (T.haar_su3(rng, nsrc, np.float32) if s["kind"] == "M" else
                    T.gaussian_field(rng, nsrc, NC[s["kind"]], np.float32))
            buf = cuda.zeros(host.size + 4, dtype=cuda.float32, device="cuda")
            buf[off // 4:off // 4 + host.size] = cuda.from_numpy(host.reshape(-1)).cuda()
            d = {"base": buf.data_ptr() + off, "kind": s["kind"], "role": s["role"]}
            j = len(spec)
            cur[j] = host[:n].copy()
            if s["gather"]:
                idx = rng.integers(0, nsrc, max(n, 1)).astype(np.int32)
                d["index"], d["nsrc"] = T.to_dev(idx), nsrc if rng.integers(2) else 0
                cur[j] = host[idx[:n]].copy()
                keep.append(d["index"])
            devs.append(buf)
            spec.append(d)
        reg, results = {}, {}
        for st in steps:
            def value(ref):
                return reg[ref] if ref >= qla.REG0 else cur[ref]
            val = {"a": np.ascontiguousarray(value(st["a"]))}
            if st["op"] == "lmult":
                val["b"] = np.ascontiguousarray(value(st["b"]))
            if st["old"] is not None:
                val["old"] = value(st["old"])
            out = _apply(st, val, n) if n else np.zeros((0, 2 * NC[st["kind"]]), np.float32)
            reg[st["dst"]] = out
            if st["store"] >= 0:
                results[st["store"]] = out
        progs.append({"n": n, "streams": spec, "steps": [
            {k: st[k] for k in ("op", "eqop", "a", "b", "dst", "store", "adja", "adjb", "mu", "sign", "r")}
            for st in steps]})
        checks.append((devs, off, n, results, streams, steps))
        keep.append(devs)
    plan = qla.BatchProgramPlan(progs)
    plan.run()
    cuda.cuda.synchronize()
    for f, (devs, off, n, results, streams, steps) in enumerate(checks):
        for j, want in results.items():
            got = devs[j][off // 4:off // 4 + want.size].cpu().numpy().reshape(want.shape)
            assert T.bits_equal(got, want), (f, n, j, streams, steps)
    plan.close()
    assert qla.device_error() == 0
