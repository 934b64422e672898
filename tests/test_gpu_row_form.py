"""GPU: the row form's passes named by SDIM_FLAG_ROWS, whatever a run's estimate,
over the sizes and batches of test_gpu_rows.py, against the oracle."""
import numpy as np
import pytest

from sdim_gb300 import Program
from sdim_gb300.batch import BatchRunner
from tests.conftest import oracle_run
from tests.test_gpu_rows import _repeats, _sweeps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("n,sweeps", [(1, 3), (2, 20), (7, 12), (9, 8), (33, 5), (64, 3), (65, 2), (130, 2)])
def test_alone(n, d, sweeps):
    spec = _sweeps(n, d, 1000 * n + d, sweeps)
    for shots in (3, 40, 200):
        got = Program(spec.build()).sample(shots, seed=5 + n, engine="rows")
        assert np.array_equal(got, oracle_run([spec], 5 + n, 0, shots)["records"]), shots


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("count", [20, 60, 170])
def test_batches_of_every_cluster_size(d, count):
    """Clusters of four and two CTAs a program, and one: with a chain pass of more than two panels."""
    br, specs = BatchRunner(), [_repeats(9 + k % 24, d, k) for k in range(10)]
    for k in range(count):
        br.add_spec(specs[k % 10], 1 + k % 3, 90 + k)
    outs = br.run(engine="rows")
    for k in (0, 7, count // 2, count - 1):
        assert np.array_equal(outs[k], oracle_run([specs[k % 10]], 90 + k, 0, 1 + k % 3)["records"]), k
