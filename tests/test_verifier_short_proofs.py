"""A proof that runs out is rejected, and the verifiers write nothing past the transcript's end and
leave nothing in flight, wherever it was cut (the verifiers compiled for the host, and on the
GPU)."""
import os
import shutil
import subprocess

import pytest

from gkr_gb300 import build as libbuild
from gkr_gb300 import circuit as gc

HERE = os.path.dirname(os.path.abspath(__file__))
GRINDING_BYTES = 32


@pytest.fixture(scope="module")
def verifier(tmp_path_factory):
    nvcc = shutil.which(libbuild.NVCC) or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path_factory.mktemp("verifier") / "verifier_on_host")
    subprocess.check_call([os.environ.get("CXX", "g++"), *libbuild.CXXFLAGS, "-w", "-I", cuda, "-I", libbuild.CSRC, "-I",
                           libbuild.INCLUDE, os.path.join(HERE, "adapter", "verifier_on_host.cpp"),
                           *[os.path.join(libbuild.CSRC, f) for f in ("sha256.cpp", "keccak.cpp")], "-o", exe])

    def run(field, copies, reps, length, widths):
        layers = [str(x) for pair in zip(widths[:-1], widths[1:]) for x in pair]
        out = subprocess.check_output([exe, str(int(field == "BN254")), str(copies), str(reps), str(length), *layers])
        return [int(x) for x in out.split()]
    return run


def cuts(widths, reps, copies, elem):
    """Proof lengths: at the commitment and the grinding bytes, then for each layer from the top at
    its first row, in its first rounds, at vx, in phase two, at vy, and one byte short of a row."""
    row = copies * elem
    at = (row << widths[0]) + GRINDING_BYTES
    yield from (0, at - GRINDING_BYTES, at - 1, at)
    for n in reversed(widths[:-1]):
        rows = reps * (6 * n + 2)
        for r in sorted({0, 1, 3 * reps, 3 * reps * n + 1, rows // 2, rows - reps, rows - 1}):
            yield at + r * row
            yield at + r * row + row - 1
        at += rows * row


@pytest.mark.parametrize("field,widths,copies,reps", [
    ("M31", [3, 4, 2, 5, 1], 8, 3), ("M31", [1, 1], 4, 1), ("M31", [6, 7], 20, 2), ("BN254", [3, 4, 2, 5, 1], 3, 1),
    ("BN254", [2, 0], 1, 1),
])
def test_short_proofs_stay_inside_the_transcript(verifier, field, widths, copies, reps):
    elem = 32 if field == "BN254" else 4
    for length in cuts(widths, reps, copies, elem):
        accepted, overrun, _, in_flight = verifier(field, copies, reps, length, widths)
        assert (accepted, overrun, in_flight) == (0, 0, 0), length
    # all rows there (and some more): read to the end, with the input's evaluations
    whole = (copies * elem << widths[0]) + GRINDING_BYTES + sum(reps * (6 * n + 2) for n in widths[:-1]) * copies * elem
    for length in (whole, whole + 5):
        accepted, overrun, launches, in_flight = verifier(field, copies, reps, length, widths)
        assert (accepted, overrun, in_flight) == (0, 0, 0), length
        assert launches == 1 + 2 * (len(widths) - 1) + 2


@pytest.mark.gpu
@pytest.mark.parametrize("field,widths,copies", [("M31", [5, 7, 6, 4], 12), ("BN254", [4, 5, 3], 3)])
def test_short_proofs_are_rejected(ctx, field, widths, copies):
    circ = gc.random_circuit(701, widths, p_mul=0.6)
    make = gc.random_witness_bn254 if field == "BN254" else gc.random_witness
    dc = ctx.load(circ, field)
    cv, proof = ctx.prove(dc, make(701, circ.log_input_size, copies))
    for length in cuts(widths, dc.num_repetitions(), copies, 32 if field == "BN254" else 4):
        if length == 0:
            continue  # no buffer to pass
        assert length < len(proof) and not ctx.verify(dc, proof[:length], cv), length
    assert ctx.verify(dc, proof, cv) and ctx.verify(dc, proof + bytes(5), cv)
    assert ctx.prove(dc, make(701, circ.log_input_size, copies))[1] == proof
