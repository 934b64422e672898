"""GPU: narrow programs of many thousand measurements, each with a column of its
own in the row form, alone and many in one launch, against the oracle."""
import numpy as np
import pytest

from sdim_gb300.batch import BatchRunner
from sdim_gb300.encode import DeviceProgram, encode_program
from sdim_gb300.workloads import CircuitSpec, random_hpc
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
    assert np.array_equal(br.run(engine="trace")[0], oracle_run([spec], 11, 0, 37)["records"])


def test_many_long_programs_in_one_launch():
    """80 programs of more column words (517) than a CTA has threads."""
    spec = _long(4, 2, 16500, seed=1)
    br = BatchRunner()
    dp = _program(br, spec)
    for k in range(80):
        br.add_program(dp, 1 + k % 3, 100 + k)
    outs = br.run(engine="trace")
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
    outs = br.run(engine="trace")
    assert np.array_equal(outs[0], oracle_run([long], 7, 0, 2)["records"])
    assert np.array_equal(outs[100], oracle_run([small], 119, 0, 3)["records"])
