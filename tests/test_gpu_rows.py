"""GPU: the row form of the x / z pass (the trace engines' default for d = 2,
3, 5, 7) against the oracle, bit for bit: qudit counts on both sides of a
packed element and of a lane group, one to several panels of 32 measurements
(one CTA and clusters), pivots used again within a panel, every gate, RESET
and N1 rows; programs in one batch; and two-qudit gates on one qudit, which
keep the tableau pass."""
import numpy as np
import pytest

from sdim_gb300 import Program, workloads
from sdim_gb300.batch import BatchRunner
from tests.conftest import oracle_run

pytestmark = pytest.mark.gpu


def _sweeps(n, d, seed, sweeps):
    """Random gates, then M / RESET on a part of the qudits, several times; M on all."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(sweeps):
        ops += workloads.all_gates_random(n, d, 3 * n + 6, seed=rng, noise_probs=(0.0, 0.4, 1.0)).ops[:-n]
        for q in rng.permutation(n)[: max(1, n // 2)]:
            ops.append((("M", "RESET")[int(rng.integers(2))], int(q), None, {}))
    ops += [("M", q, None, {}) for q in range(n)] * 2
    return workloads.CircuitSpec(n, d, ops, "sweeps")


def _check(spec, shots, seed):
    got = Program(spec.build()).sample(shots, seed=seed, engine="trace")
    want = oracle_run([spec], seed, 0, shots)["records"]
    assert np.array_equal(got, want), (spec.num_qudits, spec.dimension)


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("n,sweeps", [(1, 3), (2, 20), (7, 12), (8, 1), (9, 8), (31, 3), (33, 5), (64, 3), (65, 2),
                                      (130, 2)])
def test_rows_match_oracle(n, d, sweeps):
    _check(_sweeps(n, d, 1000 * n + d, sweeps), 40, seed=5 + n)


@pytest.mark.parametrize("n,d", [(300, 2), (1030, 2), (257, 3), (200, 5), (290, 7)])
def test_rows_match_oracle_wide(n, d):
    _check(workloads.random_hpc(n, d, 5 * n, seed=n, mr_every=n, mr_fraction=0.1), 3, seed=2)


@pytest.mark.parametrize("d", [2, 3, 5, 7])
def test_rows_batch_matches_oracle(d):
    br = BatchRunner()
    items = [(_sweeps(n, d, 7 * n + d, s), 33 + n) for n, s in ((3, 4), (40, 3), (17, 6), (90, 2), (33, 1))]
    for k, (spec, shots) in enumerate(items):
        br.add_spec(spec, shots, 50 + k)
    for k, ((spec, shots), out) in enumerate(zip(items, br.run(engine="trace"))):
        assert np.array_equal(out, oracle_run([spec], 50 + k, 0, shots)["records"]), k


@pytest.mark.parametrize("d", [2, 3, 5])
def test_gates_on_one_qudit_twice(d):
    spec = _sweeps(6, d, 3, 2)
    ops = list(spec.ops)
    ops[5:5] = [("CNOT", 2, 2, {}), ("CZ", 1, 1, {}), ("SWAP", 3, 3, {})]
    _check(workloads.CircuitSpec(6, d, ops, "aliased"), 40, seed=9)


def test_mixed_batch_matches_oracle():
    """Programs with and without fires, in row form and not, of one trace-row
    width, in one launch: each kind has its own replay."""
    twice = workloads.CircuitSpec(9, 2, [("H", 0, None, {}), ("CNOT", 3, 3, {})] + [("M", q, None, {}) for q in range(9)],
                                  "aliased")
    odd = workloads.CircuitSpec(8, 5, [("H", 0, None, {}), ("CNOT", 3, 3, {})] + [("M", q, None, {}) for q in range(8)],
                                "aliased")
    specs = [workloads.random_hpc(30, 2, 100, seed=3), workloads.surface_memory(3, 2, prob=0.05), twice,
             workloads.random_hpc(12, 5, 60, seed=1), odd, workloads.random_hpc(21, 2, 80, seed=4),
             workloads.random_hpc(9, 5, 60, seed=6)]
    br = BatchRunner()
    for k, spec in enumerate(specs):
        br.add_spec(spec, 150 + 40 * k, 60 + k)
    for k, (spec, out) in enumerate(zip(specs, br.run())):
        assert np.array_equal(out, oracle_run([spec], 60 + k, 0, 150 + 40 * k)["records"]), k


def _repeats(n, d, seed):
    """Sweeps of M on all qudits with gates only before some: whole panels of
    deterministic rows, after a random panel, at the end and up to a lone random row."""
    rng = np.random.default_rng(seed)
    meas = [("M", q, None, {}) for q in range(n)]
    gates = workloads.all_gates_random(n, d, 3 * n, seed=rng, noise_probs=(0.3,)).ops[:-n]
    more = workloads.all_gates_random(n, d, 2 * n, seed=rng).ops[:-n]
    k = 1 + 124 // n
    ops = gates + meas * k + [("H", int(rng.integers(n)), None, {})] + meas * k + more + meas * (k + 1)
    return workloads.CircuitSpec(n, d, ops, "repeats")


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("n", [9, 33, 130])
def test_deterministic_panels_match_oracle(n, d):
    _check(_repeats(n, d, 10 * n + d), 5, seed=n)


@pytest.mark.parametrize("d", [2, 5])
def test_deterministic_panels_in_a_batch(d):
    """More programs than SMs: one CTA each."""
    br = BatchRunner()
    specs = [_repeats(4 + k % 7, d, k) for k in range(160)]
    for k, spec in enumerate(specs):
        br.add_spec(spec, 1 + k % 3, 90 + k)
    for k, (spec, out) in enumerate(zip(specs, br.run(engine="trace"))):
        if k % 8 == 0:
            assert np.array_equal(out, oracle_run([spec], 90 + k, 0, 1 + k % 3)["records"]), k
