"""CPU: which programs of a run take the row form (route_cost.cuh, through the
host-only sdim_row_choice), against runs measured on GB300 on both routes."""
import numpy as np
import pytest

from sdim_gb300 import _lib, workloads
from sdim_gb300.encode import encode_program
from sdim_gb300.workloads import CircuitSpec

SMS = 152


def _narrow(n, d, measurements, seed=1):
    """Three random gates, then M or RESET on a random qudit, over and over."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(measurements):
        for _ in range(3):
            g, q = ("H", "P", "CNOT")[int(rng.integers(3))], int(rng.integers(n))
            t = int(rng.integers(n - 1))
            ops.append((g, q, t + (t >= q) if g == "CNOT" else None, {}))
        ops.append((("RESET" if rng.random() < 0.1 else "M"), int(rng.integers(n)), None, {}))
    return CircuitSpec(n, d, ops, "narrow")


def _choice(specs, shots, flags=0):
    """1 for each program of the run that takes the row form; equal specs may repeat."""
    seen = {}
    for s in specs:
        if id(s) not in seen:
            seen[id(s)] = encode_program([s.build()], s.num_qudits, s.dimension)
    encs = [seen[id(s)] for s in specs]
    begin = np.concatenate([[0], np.cumsum([e.ops.shape[0] for e in encs])]).astype(np.int64)
    rows, probs = np.concatenate([e.ops for e in encs]), np.concatenate([e.probs for e in encs])
    n = np.array([s.num_qudits for s in specs], np.int32)
    d = np.array([s.dimension for s in specs], np.int32)
    ns = np.broadcast_to(np.asarray(shots, np.int64), (len(specs),)).copy()
    out = np.zeros(len(specs), np.uint8)
    rc = _lib.load().sdim_row_choice(len(specs), rows.ctypes.data, begin.ctypes.data, probs.ctypes.data, n.ctypes.data,
                                     d.ctypes.data, ns.ctypes.data, flags, SMS, out.ctypes.data)
    assert rc == _lib.SDIM_OK
    return out


# (n, d, measurements, shots, programs, us in row form, us without); one route at least 1.8 times the other
MEASURED = [
    (3, 2, 2000, 1000, 1, 2442, 6817), (31, 2, 8000, 1, 1, 5511, 12499), (100, 3, 8000, 1, 1, 19788, 129381),
    (3, 7, 20000, 1, 1, 170496, 51700), (8, 5, 20000, 1000, 1, 158627, 64667), (31, 3, 500, 100, 1, 459, 2235),
    (100, 5, 2000, 200, 15, 2621, 10990), (31, 7, 200, 1, 100, 298, 848), (3, 3, 2000, 1, 100, 10952, 4721),
    (100, 7, 500, 1, 100, 941, 7894), (3, 2, 2000, 1, 300, 8588, 3175), (3, 5, 1000, 1, 300, 11929, 2489),
    (31, 7, 2000, 1, 300, 44978, 9389), (100, 5, 2000, 200, 300, 42306, 15060), (31, 3, 200, 200, 300, 531, 1078),
    (100, 2, 200, 1, 300, 257, 536), (3, 2, 8, 1, 1000, 216, 29), (31, 2, 62, 200, 1000, 326, 871),
    (8, 7, 62, 1, 1000, 393, 207), (60, 7, 124, 64, 1000, 701, 1923), (31, 2, 8, 1, 4000, 846, 37),
    (31, 3, 31, 1, 4000, 952, 238), (3, 7, 250, 1, 4000, 9892, 1648), (8, 2, 124, 200, 4000, 2132, 6444),
]


@pytest.mark.parametrize("n,d,measurements,shots,programs,row,other", MEASURED)
def test_the_measured_faster_route_is_taken(n, d, measurements, shots, programs, row, other):
    got = _choice([_narrow(n, d, measurements)] * min(programs, 4000), shots)
    assert (got == (1 if row < other else 0)).all()


def test_lone_programs_of_ordinary_size_take_it():
    for d in (2, 3, 5, 7):
        for n in (8, 32, 64, 128, 256, 517, 1024):
            for shots in (1, 100, 10000):
                assert _choice([workloads.random_hpc(n, d, 8 * n, seed=n)], shots)[0] == 1, (n, d, shots)
    assert _choice([workloads.surface_memory(7, 7)], 100000)[0] == 1


def test_a_wide_program_takes_it_beside_thousands_of_small_ones():
    small = workloads.random_hpc(6, 2, 24, seed=1)
    # (ms on GB300: all in row form 1.13, none 1.46, the wide ones alone 0.24)
    got = _choice([workloads.random_hpc(300, 2, 1200, seed=2)] * 8 + [small] * 4000, 1)
    assert got[:8].all() and not got[8:].any()


def test_millions_of_shots_of_a_tiny_odd_d_program():
    """The row form's replay costs more a shot there: 2 qudits of d = 7, 20,000 shots
    28 and 30 us, 3,000,000 shots 168 and 86 us.  Not for qubits, or with noise."""
    tiny = workloads.random_hpc(2, 7, 12, seed=2)
    assert _choice([tiny], 20000)[0] == 1 and _choice([tiny], 3000000)[0] == 0
    assert _choice([workloads.random_hpc(2, 2, 12, seed=2)], 3000000)[0] == 1
    assert _choice([workloads.random_hpc(300, 7, 1800, seed=2)], 3000000)[0] == 1


def test_mixed_sizes_keep_one_route():
    """Batches of many sizes, whose small programs would do as well as shot groups:
    splits took up to 2.2 times as long as the row form for all."""
    for programs, top, shots in ((241, 200, 25), (175, 20, 64), (449, 276, 200), (1277, 69, 8)):
        rng = np.random.default_rng(programs)
        n = np.round(np.exp(rng.uniform(np.log(12), np.log(top), programs))).astype(int)
        specs = [workloads.random_hpc(int(k), (2, 3, 5, 7)[i % 4], 4 * int(k), seed=i) for i, k in enumerate(n)]
        assert _choice(specs, rng.integers(1, shots + 1, programs)).all(), programs


def test_flags_and_programs_without_a_row_form():
    small = [workloads.random_hpc(6, 2, 24, seed=1)] * 2000
    assert _choice(small, 1, _lib.FLAG_ROWS).all() and not _choice(small, 1).any()
    for flag in (_lib.FLAG_NO_ROWS, _lib.FLAG_FORCE_GMEM, _lib.FLAG_NO_TRACE, _lib.FLAG_PER_SHOT, _lib.FLAG_PLAIN):
        assert not _choice([workloads.random_hpc(64, 3, 500, seed=1)], 1000, flag).any()
    twice = CircuitSpec(4, 3, [("CNOT", 1, 1, {}), ("M", 0, None, {})], "aliased")
    assert not _choice([twice, workloads.random_hpc(64, 11, 500, seed=1)], 1000, _lib.FLAG_ROWS).any()
    assert not _choice(small[:1], 0, _lib.FLAG_ROWS).any()
