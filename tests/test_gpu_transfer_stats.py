"""gkrgpu_transfer_stats counts what a call moves between host and device: its input, and its
results, also where kernels write them into mapped host memory."""
import pytest

from gkr_gb300 import circuit as gc

pytestmark = pytest.mark.gpu


def moved(ctx, f):
    """(host -> device, device -> host) bytes of f()."""
    before = ctx.transfer_stats()
    f()
    after = ctx.transfer_stats()
    return after[0] - before[0], after[1] - before[1]


@pytest.mark.parametrize("field,widths,n", [("M31", [6, 13, 3, 1], 20), ("M31", [16, 9], 1024), ("BN254", [6, 12, 1, 4], 5)])
def test_a_proof_and_its_verification(field, widths, n):
    from gkr_gb300.prover import Context
    ctx = Context(0)
    circ = gc.random_circuit(721, widths)
    make = gc.random_witness if field == "M31" else gc.random_witness_bn254
    w = make(721, circ.log_input_size, n)
    dc = ctx.load(circ, field)
    reps, row = dc.num_repetitions(), n * (4 if field == "M31" else 32)
    # three evaluations a round, two rows at the end of a phase, the claims
    results = reps * row * (sum(6 * x + 4 for x in widths[:-1]) + 1)
    assert moved(ctx, lambda: ctx.prove(dc, w)) == (w.nbytes, results)
    ctx.set_round_tail(False)
    assert moved(ctx, lambda: ctx.prove(dc, w)) == (w.nbytes, results)
    cv, proof = ctx.prove(dc, w)
    # two gate sums a layer and repetition, the input's evaluations at two points
    sums = reps * (2 * (len(widths) - 1) * (row // n) + 2 * row)
    assert moved(ctx, lambda: ctx.verify(dc, proof, cv)) == (w.nbytes, sums)
    ctx.close()


@pytest.mark.parametrize("nb_vars,n,points", [(9, 36, 1), (10, 256, 3)])
def test_eval_multilinear(ctx, nb_vars, n, points):
    from gkr_gb300.prover import DeviceBuffer
    st = gc.Stream(731)
    table = st.field((1 << nb_vars) * n).reshape(1 << nb_vars, n)
    d = DeviceBuffer(ctx, table.nbytes)
    d.upload(table)
    pts = st.field(points * nb_vars).reshape(points, nb_vars)
    assert moved(ctx, lambda: ctx.eval_multilinear(d.ptr, nb_vars, n, pts)) == (0, 4 * points * n)
