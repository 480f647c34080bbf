"""Performance cases of the prover's public entry points.

Proofs (`Context.prove`, `Context.prove_device`), a batch of queued proofs
(`Context.submit` / `wait` over 16 lanes), `Context.evaluate`, `Context.verify` and
`Context.eval_multilinear`, over M31 and BN254, from a few kilobytes to layers of 2^20 gates
at 1024 copies.  A program keeps its contexts and loaded circuits for as long as it runs, so
both are made once per process; a case's witnesses, points and proofs come from the seed.
"""
import functools
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "expander-cpp_gb300"))

from gkr_gb300 import circuit as gc  # noqa: E402
from gkr_gb300.prover import Context, DeviceBuffer, HostBuffer  # noqa: E402

GRINDING = 10


def listed():
    return [
        # the small plain workload: 8 layers of 2^10 gates, one packed lane set; launches and
        # round trips count
        _prove("m31 small", "10 10 10 10 10 10 10 10 10", 16),
        # a small circuit of uneven layers at a copy count that no tile divides evenly, with
        # the Keccak-256 transcript
        _prove("m31 ragged keccak", "7 9 6 8 5 3", 20, fs_hash="Keccak256"),
        # the average proof of the mixed batched workload, alone
        _prove("m31 middle", "13 13 13 13 13 13 13 13 13 13 13 13", 112),
        # wide layers at 268 = 4 * 67 copies: no power of two divides the rows beyond 4
        _prove("m31 wide odd copies", "11 16 15 17 14", 268, p_mul=0.6, out="buffer"),
        # the large workload's layers (2^18 / 2^20 gates, window-local wiring, 1024 copies)
        # behind a narrow committed input, which is already on the device
        _prove("m31 large", "12 18 20 18 20 18", 1024, p_mul=0.6, p_local=0.8, where="device", out="buffer"),
        # continuous batching: 16 proofs of the mixed workload's depths and copies in flight
        {"name": "m31 batch", "kind": "batch", "proofs": 16, "lanes": 16, "mix": 3, "min_width": 8, "max_width": 15},
        # BN254, a small proof and layers of the BN254 workload (2^16 gates, 64 copies)
        _prove("bn254 small", "9 9 9 9 9 9", 16, field="BN254"),
        _prove("bn254 large", "10 14 16 16 16 15", 64, field="BN254", out="buffer"),
        # Circuit::evaluate from host memory to host memory
        {"name": "m31 evaluate", "kind": "evaluate", "field": "M31", "widths": "13 15 17 17 16 13", "copies": 256,
         "p_mul": 0.6, "p_local": 0.8},
        # eight proofs to check, some of them forged
        {"name": "m31 verify", "kind": "verify", "field": "M31", "widths": "10 12 11 12 9", "copies": 64, "proofs": 8},
        # the RAW commitment's opening check: a large input at three points, a small odd one at one
        {"name": "m31 eval large", "kind": "eval", "vars": 18, "copies": 1024, "points": 3},
        {"name": "m31 eval small", "kind": "eval", "vars": 9, "copies": 36, "points": 1},
    ]


def _prove(name, widths, copies, field="M31", p_mul=0.5, p_local=0.0, where="host", out="bytes", fs_hash="SHA256"):
    c = {"kind": "prove", "field": field, "widths": widths, "copies": copies, "p_mul": p_mul, "p_local": p_local,
         "where": where, "out": out, "fs_hash": fs_hash}
    return dict(c, name=name) if name else c


def draw(rng):
    kind = rng.choice(["prove"] * 6 + ["bn"] * 3 + ["batch", "evaluate", "verify", "eval", "eval"])
    if kind == "eval":
        return {"kind": "eval", "vars": rng.randint(4, 18), "copies": 4 * _log(rng, 1, 256), "points": rng.randint(1, 3)}
    if kind == "batch":
        lo = rng.randint(5, 9)
        return {"kind": "batch", "proofs": rng.randint(5, 16), "lanes": rng.choice([4, 8, 16]), "mix": rng.randint(1, 999),
                "min_width": lo, "max_width": rng.randint(lo + 2, 14)}
    if kind == "bn":
        base, copies = rng.randint(3, 14), _log(rng, 1, 96)
        widths = _widths(rng, base, 2, 15, rng.randint(2, 8), (1 << 22) // copies)
        return _prove(None, widths, copies, field="BN254", p_mul=rng.choice([0.3, 0.5, 1.0]),
                      where=rng.choice(["host", "device"]), out=rng.choice(["bytes", "buffer"]))
    if kind == "evaluate":
        copies = 4 * _log(rng, 1, 128)
        widths = _widths(rng, rng.randint(5, 15), 3, 17, rng.randint(2, 8), (1 << 26) // copies)
        return {"kind": "evaluate", "field": "M31", "widths": widths, "copies": copies, "p_mul": rng.choice([0.4, 0.6]),
                "p_local": rng.choice([0.0, 0.8])}
    if kind == "verify":
        copies = 4 * _log(rng, 1, 32)
        widths = _widths(rng, rng.randint(5, 12), 3, 13, rng.randint(2, 6), (1 << 21) // copies)
        return {"kind": "verify", "field": "M31", "widths": widths, "copies": copies, "proofs": rng.randint(4, 10)}
    copies = 4 * _log(rng, 1, 256)
    base = rng.randint(4, 18)
    widths = _widths(rng, base, 3, 19, rng.randint(2, 12), (1 << 28) // copies)
    return _prove(None, widths, copies, p_mul=rng.choice([0.0, 0.5, 0.6, 1.0]), p_local=rng.choice([0.0, 0.8]),
                  where=rng.choice(["host", "device"]), out=rng.choice(["bytes", "buffer"]),
                  fs_hash=rng.choice(["SHA256", "SHA256", "SHA256", "Keccak256"]))


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return min(hi, int(lo * (float(hi + 1) / lo) ** rng.random()))


def _widths(rng, base, lo, hi, layers, rows):
    """Layer widths around `base`: at most `rows` rows and 2^20 gates in all, a committed
    input of at most a sixteenth of the rows where the layers allow it."""
    w = [min(hi, max(lo, base + rng.randint(-2, 2))) for _ in range(layers + 1)]
    while sum(1 << x for x in w) > min(rows, 1 << 20) and max(w) > lo:
        w[w.index(max(w))] -= 1
    if w[0] > 12:
        w[0] = 12
    return " ".join(str(x) for x in w)


# ------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _context(lanes):
    ctx = Context(0)
    if lanes > 1:
        ctx.set_concurrency(lanes)
    return ctx


@functools.lru_cache(maxsize=48)
def _loaded(lanes, field, widths, p_mul, p_local):
    """A circuit on the device; its wiring is the case's, whatever the witness."""
    circ = gc.random_circuit(2024, [int(x) for x in widths.split()], p_mul=p_mul, p_local=p_local)
    return _context(lanes).load(circ, field)


@functools.lru_cache(maxsize=8)
def _mix(mix, proofs, lo, hi):
    """The mixed workload's (seed, depth, width, copies) of each proof."""
    return gc.mixed_batch_specs(seed=mix, n_proofs=proofs, width=(lo, hi))


@functools.lru_cache(maxsize=8)
def _loaded_mix(lanes, mix, proofs, lo, hi):
    return [_context(lanes).load(gc.uniform_circuit(s, d, w)) for s, d, w, _ in _mix(mix, proofs, lo, hi)]


def _values(rng, field, rows, copies):
    """Uniform canonical field elements as the library takes them."""
    if field == "BN254":
        v = rng.integers(0, 1 << 64, (rows, copies, 4), dtype=np.uint64)
        v[..., 3] %= np.uint64(gc.BN254_R >> 192)
        return v
    return rng.integers(0, gc.P, (rows, copies), dtype=np.uint32)


def _pinned(values):
    b = HostBuffer(values.nbytes)
    a = b.array.view(values.dtype).reshape(values.shape)
    a[...] = values
    return a


def _device(ctx, values):
    d = DeviceBuffer(ctx, values.nbytes)
    d.upload(values)
    return d


# ------------------------------------------------------------------ one state, one pass
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "eval":
        ctx = _context(1)
        table = _values(rng, "M31", 1 << case["vars"], case["copies"])
        return {"case": case, "ctx": ctx, "table": _device(ctx, table),
                "points": _values(rng, "M31", case["points"], case["vars"])}
    if kind == "batch":
        lanes, key = case["lanes"], (case["mix"], case["proofs"], case["min_width"], case["max_width"])
        jobs = []
        for dc, (_, _, width, copies) in zip(_loaded_mix(lanes, *key), _mix(*key)):
            jobs.append((dc, _pinned(_values(rng, "M31", 1 << width, copies)),
                         HostBuffer(dc.proof_size(copies, GRINDING)).array,
                         np.empty((dc.num_repetitions(GRINDING), copies), np.uint32)))
        return {"case": case, "ctx": _context(lanes), "jobs": jobs}
    ctx, field, copies = _context(1), case["field"], case["copies"]
    dc = _loaded(1, field, case["widths"], case.get("p_mul", 0.5), case.get("p_local", 0.0))
    ctx.set_fs_hash(case.get("fs_hash", "SHA256"))
    if kind == "verify":
        proofs = []
        for _ in range(case["proofs"]):
            cv, proof = ctx.prove(dc, _values(rng, field, 1 << dc.log_input_size, copies), GRINDING)
            if rng.integers(2):  # forged: the last claim is another one
                proof = proof[:-4] + bytes(np.uint32((int.from_bytes(proof[-4:], "little") + 1) % gc.P).tobytes())
            proofs.append((cv, proof))
        return {"case": case, "ctx": ctx, "dc": dc, "proofs": proofs}
    w = _values(rng, field, 1 << dc.log_input_size, copies)
    st = {"case": case, "ctx": ctx, "dc": dc}
    if kind == "prove" and case["out"] == "buffer":
        st["out"] = HostBuffer(dc.proof_size(copies, GRINDING)).array
    if case.get("where") == "device":
        st["d_input"] = _device(ctx, w)
        if "out" not in st:
            st["out"] = np.empty(dc.proof_size(copies, GRINDING), np.uint8)
    else:
        st["witness"] = _pinned(w)
    return st


def _plain(a):
    """Field elements and digests as signed integers of their size (torch's own types)."""
    return a.view(np.int32) if a.dtype == np.uint32 else a.view(np.int64) if a.dtype == np.uint64 else a


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "eval":
        return _plain(ctx.eval_multilinear(state["table"].ptr, case["vars"], case["copies"], state["points"]))
    if kind == "batch":
        jobs = [ctx.submit(dc, w, proof, cv, GRINDING) for dc, w, proof, cv in state["jobs"]]
        lengths = [ctx.wait(j) for j in jobs]
        return {"proofs": [p[:n] for n, (_, _, p, _) in zip(lengths, state["jobs"])],
                "claimed": [_plain(cv) for _, _, _, cv in state["jobs"]]}
    if kind == "verify":
        return [int(ctx.verify(state["dc"], proof, cv, GRINDING)) for cv, proof in state["proofs"]]
    if kind == "evaluate":
        return _plain(ctx.evaluate(state["dc"], state["witness"]))
    ctx.set_fs_hash(case["fs_hash"])
    if "d_input" in state:
        cv, n = ctx.prove_device(state["dc"], state["d_input"].ptr, case["copies"], state["out"], GRINDING)
        return {"claimed": _plain(cv), "proof": state["out"][:n]}
    if "out" in state:
        cv, n = ctx.prove(state["dc"], state["witness"], GRINDING, out=state["out"])
        return {"claimed": _plain(cv), "proof": state["out"][:n]}
    cv, proof = ctx.prove(state["dc"], state["witness"], GRINDING)
    return {"claimed": _plain(cv), "proof": np.frombuffer(proof, np.uint8)}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: the inputs, the circuit's gates and the results once each.  Flops: two per
    32 x 32-bit multiplication of the field products (64 of them in a BN254 product)."""
    kind = case["kind"]
    if kind == "eval":
        rows, n, k = 1 << case["vars"], case["copies"], case["points"]
        return {"bytes": 4 * (rows * n + k * (case["vars"] + n)), "flops": 2 * k * rows * (n + 1)}
    if kind == "batch":
        parts = [_work_of([w] * (d + 1), n, 0.5, "M31", True)
                 for _, d, w, n in _mix(case["mix"], case["proofs"], case["min_width"], case["max_width"])]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    widths = [int(x) for x in case["widths"].split()]
    if kind == "verify":
        b, _ = _work_of(widths, case["copies"], 0.5, "M31", True)
        muls = 6 * sum(1 << x for x in widths) + 6 * case["copies"] * (1 << widths[0])
        return {"bytes": case["proofs"] * b, "flops": 2 * case["proofs"] * muls}
    b, f = _work_of(widths, case["copies"], case["p_mul"], case["field"], kind == "prove")
    return {"bytes": b, "flops": f}


def _work_of(widths, copies, p_mul, field, prove):
    size, limbs, reps = (32, 64, 1) if field == "BN254" else (4, 1, 3)
    b = size * copies * (1 << widths[0])
    muls = 0
    for n_in, n_out in zip(widths[:-1], widths[1:]):
        rows, gates = 1 << n_in, 1 << n_out
        b += gates * (16 * p_mul + 24 * (1 - p_mul))
        muls += copies * gates * 2  # evaluate
        if prove:
            b += size * copies * reps * (6 * n_in + 2)
            # both phases: two sums a pair and one fold a pair and table, halving each round;
            # phase one gathers a product for each mul gate
            muls += copies * reps * (gates * p_mul + rows * (2 + 2) + rows * (2 + 1))
    if prove:
        b += size * copies * (1 << widths[0])  # the commitment in the proof
    else:
        b += size * copies * (1 << widths[-1])
    return float(b), 2.0 * limbs * muls


def exact(case, seed):
    """Every output is a whole number or a byte: none is rounded."""
    return None
