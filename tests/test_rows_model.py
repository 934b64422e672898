"""CPU: the row form of the x / z pass (tests/rows_model.py) -- all gates
first, then the measurements eliminated on their rows -- gives the trace of
the one-at-a-time pass over the stabilizer half (odd d), and records that
equal the oracle's (every d), for sweeps that measure qudits several times
with gates between."""
import numpy as np
import pytest

import oracle
from sdim_gb300 import workloads
from tests.conftest import oracle_run
from tests.rows_model import eliminate, raw_rows, replay
from tests.test_xz_model import _ops, _spec
from tests.xz_model import sequential_xz


@pytest.mark.parametrize("d", [3, 5, 7, 11])
@pytest.mark.parametrize("n,kind", [(1, "twice"), (2, "hpc"), (5, "twice"), (17, "hpc"), (40, "twice")])
def test_rows_match_sequential(n, d, kind):
    ops = _ops(_spec(n, d, seed=n * 31 + d, kind=kind))
    seq, _ = sequential_xz(n, d, ops)
    rec, _ = eliminate(raw_rows(n, d, ops))
    assert len(seq) == len(rec)
    for i, ((h1, r1, z1), (kind2, p, e, a, row, zrow)) in enumerate(zip(seq, rec)):
        assert h1 == (kind2, p, e, a), (i, h1)
        assert np.array_equal(r1[:n], row), i
        assert (z1 is None) == (zrow is None) and (z1 is None or np.array_equal(z1[:n], zrow)), i


def _words(spec):
    """Device instructions of a spec's plain gates (CZ, SWAP, M_X expanded as the encoder does)."""
    out = []
    for g, q, t, _ in spec.op_table():
        g, q, t = int(g), int(q), int(t)
        if g == 0:
            continue
        if g in (11, 12):
            out += [(6, t, -1), (9 if g == 11 else 10, q, t), (5, t, -1)]
        elif g == 13:
            out += [(9, q, t), (5, q, -1), (5, t, -1)] * 2 + [(9, q, t), (5, t, -1), (5, t, -1)]
        elif g == 15:
            out += [(6, q, -1), (14, q, -1)]
        else:
            out.append((g, q, t))
    return out


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("n", [1, 2, 4, 9, 33])
def test_rows_records_match_oracle(n, d):
    rng = np.random.default_rng(100 * n + d)
    for case in range(6):
        ops = []
        for _ in range(12 * n + 10):
            g = ("X", "X_INV", "Z", "Z_INV", "H", "H_INV", "P", "P_INV", "M", "M_X", "RESET", "CNOT", "CNOT_INV",
                 "CZ", "CZ_INV", "SWAP", "CNOT", "H", "P")[int(rng.integers(19))]
            q = int(rng.integers(n))
            if g in ("CNOT", "CNOT_INV", "CZ", "CZ_INV", "SWAP"):
                if n == 1:
                    continue
                t = int(rng.integers(n - 1))
                ops.append((g, q, t + (t >= q), {}))
            else:
                ops.append((g, q, None, {}))
        ops += [("M", q, None, {}) for q in range(n)]
        spec = workloads.CircuitSpec(n, d, ops, "rows")
        rec, _ = eliminate(raw_rows(n, d, _words(spec)))
        seed = 77 + case
        want = oracle_run([spec], seed, 0, 4)["records"]
        for s in range(4):
            draw = lambda k: int(oracle.philox.measurement_outcome(seed, s, k, d))  # noqa: E731
            assert np.array_equal(replay(rec, n, d, draw), want[s]), (case, s)
