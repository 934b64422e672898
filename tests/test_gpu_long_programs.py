"""GPU: the row form where a run does not take it by itself -- narrow programs of
many thousand measurements, each with a column of its own, alone and many in
one launch, and small programs by the hundred -- and runs whose programs take
different routes, against the oracle."""
import numpy as np
import pytest

from sdim_gb300.batch import BatchRunner
from sdim_gb300.encode import DeviceProgram, encode_program
from sdim_gb300.workloads import CircuitSpec, all_gates_random, random_hpc
from tests.conftest import oracle_run

pytestmark = pytest.mark.gpu


def _long(n, d, measurements, seed):
    """Random gates and measurements, a measurement every other instruction."""
    rng = np.random.default_rng(seed)
    ops = []
    for k in range(measurements):
        g = ("H", "P", "CNOT")[int(rng.integers(3))]
        q, t = (int(x) for x in rng.permutation(n)[:2])
        ops += [(g, q, t if g == "CNOT" else None, {}), ("M", k % n, None, {})]
    return CircuitSpec(n, d, ops, "long")


def _program(br, spec):
    return DeviceProgram(br.ctx, encode_program([spec.build()], spec.num_qudits, spec.dimension))


@pytest.mark.parametrize("d", [2, 5])
def test_long_program_alone(d):
    spec = _long(4, d, 3000, seed=d)
    br = BatchRunner()
    br.add_program(_program(br, spec), 37, 11)
    assert np.array_equal(br.run(engine="rows")[0], oracle_run([spec], 11, 0, 37)["records"])


def test_many_long_programs_in_one_launch():
    """80 programs of more column words (517) than a CTA has threads."""
    spec = _long(4, 2, 16500, seed=1)
    br = BatchRunner()
    dp = _program(br, spec)
    for k in range(80):
        br.add_program(dp, 1 + k % 3, 100 + k)
    outs = br.run(engine="rows")
    for k in (0, 1, 41, 79):
        assert np.array_equal(outs[k], oracle_run([spec], 100 + k, 0, 1 + k % 3)["records"]), k


@pytest.mark.parametrize("d", [2, 3, 7])
def test_one_long_program_among_small_ones(d):
    long, small = _long(4, d, 16500 if d == 2 else 2000, seed=d), random_hpc(3, d, 20, seed=2)
    br = BatchRunner()
    br.add_program(_program(br, long), 2, 7)
    dp = _program(br, small)
    for k in range(100):
        br.add_program(dp, 3, 20 + k)
    outs = br.run(engine="rows")
    assert np.array_equal(outs[0], oracle_run([long], 7, 0, 2)["records"])
    assert np.array_equal(outs[100], oracle_run([small], 119, 0, 3)["records"])


def _repeats(n, d, seed):
    """Sweeps of M on all qudits with gates in front of some: panels without a random row."""
    rng = np.random.default_rng(seed)
    meas = [("M", q, None, {}) for q in range(n)]
    gates = all_gates_random(n, d, 3 * n, seed=rng, noise_probs=(0.3,)).ops[:-n]
    k = 1 + 124 // n
    ops = gates + meas * k + [("H", int(rng.integers(n)), None, {})] + meas * k
    return CircuitSpec(n, d, ops, "repeats")


@pytest.mark.parametrize("d", [2, 3, 5, 7])
def test_rows_in_a_batch_of_more_programs_than_sms(d):
    br = BatchRunner()
    specs = [_repeats(4 + k % 7, d, k) for k in range(160)]
    for k, spec in enumerate(specs):
        br.add_spec(spec, 1 + k % 3, 90 + k)
    for k, (spec, out) in enumerate(zip(specs, br.run(engine="rows"))):
        if k % 8 == 0:
            assert np.array_equal(out, oracle_run([spec], 90 + k, 0, 1 + k % 3)["records"]), k


@pytest.mark.parametrize("engine", [None, "trace", "rows", "tableau"])
def test_a_run_of_different_routes(engine):
    """Small programs by the hundred, a few wide ones and a long narrow one, for
    every d, with and without noise, in one run."""
    br, specs = BatchRunner(), []
    for d in (2, 3, 5, 7, 11):
        specs += [random_hpc(3 + k % 9, d, 30, seed=10 * d + k) for k in range(60)]
        specs += [all_gates_random(5, d, 60, seed=d, noise_probs=(0.2,)), random_hpc(170, d, 300, seed=d),
                  _long(3, d, 700, seed=d)]
    shots = [1 + (37 * k) % 150 for k in range(len(specs))]
    for k, spec in enumerate(specs):
        br.add_spec(spec, shots[k], 300 + k)
    for k, (spec, out) in enumerate(zip(specs, br.run(engine=engine))):
        if k % 60 in (0, 7) or spec.num_qudits > 100 or len(spec.ops) > 1000:
            assert np.array_equal(out, oracle_run([spec], 300 + k, 0, shots[k])["records"]), k


@pytest.mark.parametrize("captured", [False, True])
def test_without_room_for_the_rows(captured):
    """A device whose memory is taken: 40 programs of 33 MB of rows each, with
    160 MB left, take the routes that need none."""
    import torch
    from sdim_gb300 import _lib
    spec = _long(4, 2, 16500, seed=2)
    br = BatchRunner(_lib.Context(0))
    dp = _program(br, spec)
    for k in range(40):
        br.add_program(dp, 2, 60 + k)
    out = torch.zeros(40 * 2 * dp.num_records, dtype=torch.uint8, device="cuda")
    ptrs = [out.data_ptr() + 2 * k * dp.num_records for k in range(40)]
    torch.cuda.synchronize()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        if captured:
            run = br.capture(ptrs, engine="rows")
            run.launch()
            run.sync()
            run.close()
        else:
            br.run_device(ptrs, engine="rows")
    finally:
        del taken
        torch.cuda.empty_cache()
    got = out.cpu().numpy().reshape(40, 2, dp.num_records)
    for k in (0, 39):
        assert np.array_equal(got[k], oracle_run([spec], 60 + k, 0, 2)["records"]), k
