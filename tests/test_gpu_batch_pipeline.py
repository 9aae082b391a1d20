"""The steady state of the batched kernel: plans with well over sixteen tiles a
warp, hundreds of fields of many programs (full and ragged, empty, tiny, 8-B
aligned between 16-B aligned ones), so that every warp goes through many
tiles, changes field and takes a second run, in two-stage plans (short
programs) and in one-stage plans (long ones), against the oracle, bit for bit.
Several fields share a program's inputs: the oracle runs once per program."""
import ctypes

import numpy as np
import pytest

import qla_testlib as T
from test_gpu_batch_programs import EQ, NC, _apply, _program

pytestmark = pytest.mark.gpu

NMAX = 6016  # 188 tiles of 32 sites
SIZES = [6016, 5003, 33, 6016, 4096, 0, 5984, 31, 6000, 64, 5985, 1, 6015, 32, 4097]


class _PlanHead(ctypes.Structure):  # the start of struct BatchPlan (qla_batch.cu)
    _fields_ = [("dfields", ctypes.c_void_p), ("dstart", ctypes.c_void_p), ("nfields", ctypes.c_int),
                ("threads", ctypes.c_int), ("grid", ctypes.c_int), ("stages", ctypes.c_int), ("runs", ctypes.c_int),
                ("ntiles", ctypes.c_longlong)]


def _short_program(rng, qla):
    """r (eqop) s U v or U^+ v: few enough bytes a tile for two stages."""
    inout = bool(rng.integers(2))
    streams = [{"kind": "M", "role": "in", "gather": bool(rng.integers(2))},
               {"kind": "V", "role": "in", "gather": bool(rng.integers(2))},
               {"kind": "V", "role": "inout" if inout else "out", "gather": False}]
    base = {"b": 0, "adja": 0, "adjb": 0, "mu": 0, "sign": 1, "kind": "V", "r": float(rng.normal()), "old": None}
    steps = [dict(base, op="lmult", a=0, b=1, adja=int(rng.integers(2)), eqop=str(rng.choice(["eq", "eqm"])),
                  dst=qla.REG0, store=-1),
             dict(base, op=str(rng.choice(["copy", "rtimes"])), a=qla.REG0, dst=qla.REG1, store=2,
                  eqop=str(rng.choice(EQ if inout else ["eq", "eqm"])), old=2 if inout else None)]
    return streams, steps


def _oracle(streams, steps, cur, qla):
    reg, results = {}, {}
    for st in steps:
        def value(ref):
            return reg[ref] if ref >= qla.REG0 else cur[ref]
        val = {"a": np.ascontiguousarray(value(st["a"]))}
        if st["op"] == "lmult":
            val["b"] = np.ascontiguousarray(value(st["b"]))
        if st["old"] is not None:
            val["old"] = value(st["old"])
        reg[st["dst"]] = _apply(st, val, NMAX)
        if st["store"] >= 0:
            results[st["store"]] = reg[st["dst"]]
    return results


@pytest.mark.parametrize("programs,stages", [("short", 2), ("long", 1)])
@pytest.mark.parametrize("seed", [0, 1])
def test_many_tiles_and_fields_per_warp(qla, cuda, programs, stages, seed):
    rng = np.random.default_rng(1700 + seed)
    made, nfields = [], 400
    while len(made) < 20:
        pr = _short_program(rng, qla) if programs == "short" else _program(rng, qla, NMAX)
        if pr is not None:
            made.append(pr)
    dev, wants = [], []  # per program: the streams' device data at byte offsets 0 and 8, the results
    for streams, steps in made:
        cur, at = {}, []
        for j, s in enumerate(streams):
            nsrc = NMAX + 5
            host = T.gaussian_field(rng, nsrc, NC[s["kind"]], np.float32)
            idx = rng.integers(0, nsrc, NMAX).astype(np.int32) if s["gather"] else None
            cur[j] = host[:NMAX] if idx is None else host[idx]
            both = {}
            for off in (0, 8):
                buf = cuda.zeros(host.size + 4, dtype=cuda.float32, device="cuda")
                buf[off // 4:off // 4 + host.size] = cuda.from_numpy(host.reshape(-1)).cuda()
                both[off] = buf
            at.append((both, None if idx is None else T.to_dev(idx), nsrc if rng.integers(2) else 0))
        dev.append(at)
        wants.append({j: cuda.from_numpy(w).cuda() for j, w in _oracle(streams, steps, cur, qla).items()})
    fields, outs = [], []
    for f in range(nfields):
        q, n, off = f % len(made), SIZES[(f + f // len(SIZES)) % len(SIZES)], 8 if f % 9 == 4 else 0
        streams, steps = made[q]
        spec = []
        for j, s in enumerate(streams):
            both, idx, nsrc = dev[q][j]
            buf = both[off]
            if s["role"] != "in":  # its own copy, with the values from before the launch
                buf = buf.clone()
                outs.append((f, j, buf, both[off], n, off, wants[q][j]))
            d = {"base": buf.data_ptr() + off, "kind": s["kind"], "role": s["role"]}
            if idx is not None:
                d["index"], d["nsrc"] = idx, nsrc
            spec.append(d)
        fields.append({"n": n, "streams": spec, "steps": [
            {k: st[k] for k in ("op", "eqop", "a", "b", "dst", "store", "adja", "adjb", "mu", "sign", "r")}
            for st in steps]})
    plan = qla.BatchProgramPlan(fields)
    head = _PlanHead.from_address(plan.handle)
    assert head.nfields == nfields and head.ntiles == sum((p["n"] + 31) // 32 for p in fields)
    assert head.stages == stages and head.runs == 2 * head.grid
    assert head.ntiles >= 16 * head.grid * head.threads // 32
    for _ in range(3):
        for _, _, buf, before, _, _, _ in outs:
            buf.copy_(before)
        plan.run()
        for f, j, buf, before, n, off, want in outs:
            k, rec = off // 4, want.shape[1]
            got = buf[k:k + n * rec].view(cuda.int32)
            assert cuda.equal(got, want[:n].reshape(-1).view(cuda.int32)), (f, j, n, made[f % len(made)])
            # records behind the field's last one, and the bytes around the array, are untouched
            assert cuda.equal(buf[k + n * rec:], before[k + n * rec:]) and cuda.equal(buf[:k], before[:k]), (f, j, n)
    plan.close()
    assert qla.device_error() == 0
