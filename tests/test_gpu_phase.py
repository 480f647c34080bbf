"""GPU tests of the persistent sumcheck phases at the edges of their rule and tiles: layers of
exactly, just over and far over the rows a CTA takes, one-row-pair layers, copy counts that
leave part of the last CTA idle (516 = 4 * 129 at two quads a CTA), that need CTAs of 8 quads
(4096), 16 (4100 to 8192) and 32 (to 16384), and that are beyond the widest (20000, every round
launched alone).  The proof bytes equal the
oracle's and those with the phases off (exact arithmetic: tolerance zero)."""
import numpy as np
import pytest

from gkr_gb300 import circuit as gc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,widths,n,p_mul", [
    (601, [12, 13, 12], 16, 0.6), (602, [13, 12], 16, 0.6), (603, [14, 9], 8, 0.5), (604, [1, 1, 1, 1], 4, 0.5),
    (605, [2, 1, 3, 0], 20, 0.5), (606, [11, 10], 516, 0.6), (607, [12, 5], 268, 1.0), (608, [9, 10, 7], 1024, 0.0),
    (609, [6, 7], 4096, 0.5), (610, [5, 4], 20000, 0.5), (611, [3, 9, 3], 28, 1.0),
])
def test_phases_give_the_oracle_proof(ctx, oracle, seed, widths, n, p_mul):
    circ = gc.random_circuit(seed, widths, p_mul=p_mul)
    w = gc.random_witness(seed, circ.log_input_size, n)
    dc = ctx.load(circ)
    cv, proof = ctx.prove(dc, w)
    try:
        ctx.set_round_tail(False)
        assert ctx.prove(dc, w)[1] == proof
    finally:
        ctx.set_round_tail(True)
    ocv, op = oracle.prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)


def test_many_gates_on_one_row(ctx, oracle):
    # every mul gate's first input is row 0: one thread sums 2^9 gates of full-range weights
    st = gc.Stream(612)
    layer = gc.random_layer(st, 9, 9, p_mul=1.0)
    layer.mul[:, 1] = 0
    layer.mul[:, 3] = gc.P - 1
    circ = gc.Circuit([layer])
    w = np.full((512, 8), gc.P - 1, np.uint32)
    dc = ctx.load(circ)
    assert ctx.prove(dc, w)[1] == oracle.prove(circ, w)[1]


@pytest.mark.parametrize("seed,widths,n", [
    (621, [11, 10], 3), (622, [12, 11], 2), (623, [13, 4], 1), (624, [1, 1, 1], 5), (625, [2, 0], 1), (626, [5, 4], 310),
    (627, [8, 9, 7], 33),
])
def test_bn254_phases_give_the_oracle_proof(ctx, seed, widths, n):
    # the whole phase in one launch (2^11 rows), its start at a later round, one-pair layers, and
    # more copies than resident CTAs (310: every round launched alone)
    from oracle.oracle import OracleBn254
    circ = gc.random_circuit(seed, widths, p_mul=0.6)
    w = gc.random_witness_bn254(seed, circ.log_input_size, n)
    dc = ctx.load(circ, "BN254")
    cv, proof = ctx.prove(dc, w)
    try:
        ctx.set_round_tail(False)
        assert ctx.prove(dc, w)[1] == proof
    finally:
        ctx.set_round_tail(True)
    ocv, op = OracleBn254().prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)


@pytest.mark.parametrize("seed,widths,n", [
    (631, [13, 14], 268), (632, [14, 13], 148), (633, [12, 14], 44), (634, [10, 15], 36), (635, [13, 14, 13], 1036),
    (636, [5, 4], 4084),
])
def test_row_tiles_that_do_not_divide_the_copies(ctx, oracle, seed, widths, n):
    # n / 4 = 67, 37, 11, 9, 259, 1021: the last lane group of a row is partly idle; every round
    # as its own launch, so that every row-tiled kernel runs on such tiles
    circ = gc.random_circuit(seed, widths, p_mul=0.6)
    w = gc.random_witness(seed, circ.log_input_size, n)
    dc = ctx.load(circ)
    try:
        ctx.set_round_tail(False)
        cv, proof = ctx.prove(dc, w)
    finally:
        ctx.set_round_tail(True)
    assert ctx.prove(dc, w)[1] == proof
    ocv, op = oracle.prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)
    assert np.array_equal(ctx.evaluate(dc, w), oracle.evaluate(circ, w)[-1])
    assert ctx.verify(dc, proof, cv)


@pytest.mark.parametrize("seed,widths,n,p_mul,tails", [
    # the smallest tables whose rounds are taken in pairs, with a partly idle last lane group: six
    # pairs and a round, seven pairs, and a phase that takes over two rounds behind
    (641, [16, 14], 2052, 0.3, False), (642, [17, 16], 1024, 1.0, False), (643, [16, 16], 2048, 0.6, True),
    (644, [17, 15], 1028, 0.5, True),
])
def test_rounds_in_pairs_give_the_oracle_proof(ctx, oracle, seed, widths, n, p_mul, tails):
    circ = gc.random_circuit(seed, widths, p_mul=p_mul)
    w = gc.random_witness(seed, circ.log_input_size, n)
    dc = ctx.load(circ)
    try:
        ctx.set_round_tail(tails)
        cv, proof = ctx.prove(dc, w)
    finally:
        ctx.set_round_tail(True)
    ocv, op = oracle.prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)


@pytest.mark.parametrize("widths,n", [([13, 3], 250), ([14, 4], 128), ([12, 2], 1000)])
def test_bn254_sums_of_many_products(ctx, widths, n):
    # more than ten pairs a thread in the first rounds (sums reduced and gone on from), with input
    # elements whose Montgomery form is r - 1, the largest factor of a product
    from oracle.oracle import OracleBn254
    r = gc.BN254_R
    x = (r - 1) * pow(2, -256, r) % r
    circ = gc.random_circuit(651, widths, p_mul=0.6)
    w = gc.random_witness_bn254(651, circ.log_input_size, n)
    w[...] = np.frombuffer(x.to_bytes(32, "little"), np.uint64)
    cv, proof = ctx.prove(ctx.load(circ, "BN254"), w)
    ocv, op = OracleBn254().prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)


@pytest.mark.parametrize("seed,widths,n,p_mul,ctas", [
    # no mul gates at all; a step and a part of one; a row's copies and the last 64 partly past the end
    (661, [9, 8], 64, 0.0, 0), (662, [3, 4, 5], 128, 1.0, 0), (663, [13, 12], 60, 0.6, 0), (664, [10, 11], 452, 0.4, 0),
    # one CTA for all groups: sums that are reduced between conversions, of the largest inputs
    (665, [15, 16], 64, 1.0, 1),
])
def test_first_rounds_of_phase_two(oracle, seed, widths, n, p_mul, ctas):
    from gkr_gb300.prover import Context
    ctx = Context(0)
    circ = gc.random_circuit(seed, widths, p_mul=p_mul)
    w = gc.random_witness(seed, circ.log_input_size, n)
    if ctas:
        w[...] = gc.P - 1
    ctx.set_round_tail(False)
    ctx.set_tile(ctas=ctas)
    cv, proof = ctx.prove(ctx.load(circ), w)
    ocv, op = oracle.prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)
    ctx.close()


@pytest.mark.parametrize("name", ["NV_COMPUTE_PROFILER_PERFWORKS_DIR", "NV_NSIGHT_INJECTION_PORT_BASE"])
def test_no_persistent_phase_under_a_profiler(monkeypatch, ctx, name):
    # a profiler may block the launching thread until a kernel ends; a phase waits for that thread
    from gkr_gb300.prover import Context
    monkeypatch.setenv(name, "1")
    profiled = Context(0)
    circ = gc.random_circuit(671, [7, 8])
    w = gc.random_witness(671, circ.log_input_size, 16)
    cv, proof = profiled.prove(profiled.load(circ), w)
    assert profiled.kernel_stats()["round_tail"]["launches"] == 0
    profiled.close()
    assert proof == ctx.prove(ctx.load(circ), w)[1]


@pytest.mark.parametrize("seed,widths,n", [
    # 16 quads a CTA (4100 and 8192 copies) and 32 (8196 and 16384) on tables of 2 to 8 rows, and
    # on the last rounds of a layer that starts its phase at round 4
    (681, [1, 2, 3, 3, 2, 1, 0], 4100), (682, [1, 2, 3, 3, 2, 1, 0], 8192), (683, [1, 2, 3, 3, 2, 1, 0], 8196),
    (684, [1, 2, 3, 3, 2, 1, 0], 16384), (685, [10, 3, 1], 4100), (686, [10, 3, 1], 16384),
])
def test_phases_whose_finishers_are_in_several_warps(ctx, oracle, seed, widths, n):
    # with more than 8 quads a CTA its copies' sums are all warp 0's on small tables, and are read
    # by two or four warps
    circ = gc.random_circuit(seed, widths, p_mul=0.6)
    w = gc.random_witness(seed, circ.log_input_size, n)
    dc = ctx.load(circ)
    cv, proof = ctx.prove(dc, w)
    try:
        ctx.set_round_tail(False)
        assert ctx.prove(dc, w)[1] == proof
    finally:
        ctx.set_round_tail(True)
    ocv, op = oracle.prove(circ, w)
    assert proof == op and np.array_equal(cv, ocv)


@pytest.mark.parametrize("copies", [1, 152, 153, 304])
def test_bn254_phases_of_up_to_two_ctas_an_sm(copies):
    # a CTA a copy: from 153 on more of them than SMs (with a split of an SM's memory that holds two)
    from gkr_gb300.prover import Context
    from oracle.oracle import OracleBn254
    ctx = Context(0)
    circ = gc.random_circuit(695, [11, 3, 2], p_mul=0.6)
    w = gc.random_witness_bn254(695, circ.log_input_size, copies)
    proof = ctx.prove(ctx.load(circ, "BN254"), w)[1]
    assert ctx.kernel_stats()["bn254_phase"]["launches"] == 4
    ctx.close()
    assert proof == OracleBn254().prove(circ, w)[1]


def test_phases_of_both_fields_together(oracle):
    # two contexts whose phases would take several times the device: CTAs of 16 to 98 KB
    from gkr_gb300.prover import Context
    from oracle.oracle import OracleBn254
    jobs = []
    for field, lanes, widths, n, count in (("M31", 16, [13, 12, 9], 64, 48), ("BN254", 6, [11, 9, 10], 96, 24)):
        ctx = Context(0)
        ctx.set_concurrency(lanes)
        circ = gc.random_circuit(696, widths, p_mul=0.6)
        make = gc.random_witness if field == "M31" else gc.random_witness_bn254
        w = make(696, circ.log_input_size, n)
        want = (oracle if field == "M31" else OracleBn254()).prove(circ, w)[1]
        dc = ctx.load(circ, field)
        for _ in range(count):
            pb = np.empty(dc.proof_size(n), np.uint8)
            cb = np.empty((3, n), np.uint32) if field == "M31" else np.empty((1, n, 4), np.uint64)
            jobs.append((ctx, ctx.submit(dc, w, pb, cb), pb, want))
    for ctx, job, pb, want in jobs:
        assert pb[:ctx.wait(job)].tobytes() == want


@pytest.mark.parametrize("seed,widths,n", [(691, [3, 2, 3, 1, 2, 1], 512), (692, [7, 3, 2, 6], 512)])
def test_wide_tiles_on_a_full_device(oracle, seed, widths, n):
    # 64 lanes of phases that would take 128 CTAs each: the device's share of later ones is down to
    # tiles of 8, 16 and 32 quads
    from gkr_gb300.prover import Context
    ctx = Context(0)
    ctx.set_concurrency(64)
    circ = gc.random_circuit(seed, widths, p_mul=0.6)
    dc = ctx.load(circ)
    witnesses = [gc.random_witness(seed + k, circ.log_input_size, n) for k in range(8)]
    want = [oracle.prove(circ, w)[1] for w in witnesses]
    jobs = []
    for k in range(192):
        pb, cb = np.empty(dc.proof_size(n), np.uint8), np.empty((3, n), np.uint32)
        jobs.append((k % 8, ctx.submit(dc, witnesses[k % 8], pb, cb), pb))
    wrong = [k for k, job, pb in jobs if pb[:ctx.wait(job)].tobytes() != want[k]]
    ctx.close()
    assert not wrong
