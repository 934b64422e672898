"""CPU: which kernel the frame route's shots take (route_cost.cuh, through the
host-only sdim_frame_route), against frame runs measured on GB300 on both."""
import numpy as np
import pytest

from sdim_gb300 import _lib, workloads
from sdim_gb300.encode import encode_program
from sdim_gb300.workloads import CircuitSpec


def _noisy(n, d, ordinals, prob):
    """A CNOT (H) and an N1 over and over, a measurement in every twentieth part, M on all."""
    rng = np.random.default_rng(1)
    ops = []
    for k in range(ordinals):
        a, b = (int(x) for x in rng.integers(0, n, 2))
        ops.append(("CNOT", a, b, {}) if a != b else ("H", a, None, {}))
        ops.append(("N1", a, None, {"prob": prob, "noise_channel": "d"}))
        if k % (ordinals // 20) == 0:
            ops.append(("M", b, None, {}))
    return CircuitSpec(n, d, ops + [("M", q, None, {}) for q in range(n)], "noisy")


def _route(spec, shots, flags=0):
    enc = encode_program([spec.build()], spec.num_qudits, spec.dimension)
    ops, probs = np.ascontiguousarray(enc.ops), np.ascontiguousarray(enc.probs)
    got = _lib.load().sdim_frame_route(ops.ctypes.data, int(ops.shape[0]), probs.ctypes.data, spec.num_qudits,
                                       spec.dimension, shots, flags, 232448, 233472, 1024, 152)
    assert got in (0, 1)
    return got


# (n, d, ordinals, probability, [(shots, ms on planes, ms as bytes)])
MEASURED = [
    (7, 2, 10000, 1e-3, [(2000, 1.35, 7.01), (300000, 7.95, 15.73)]),
    (7, 2, 60000, 1e-3, [(20000, 16.52, 41.24), (300000, 144.91, 95.47)]),
    (7, 2, 120000, 1e-3, [(20000, 50.47, 82.38), (100000, 218.34, 97.36), (300000, 624.14, 190.71)]),
    (100, 2, 60000, 1e-3, [(2000, 1.63, 29.88), (300000, 39.34, 95.34)]),
    (7, 3, 5000, 1e-3, [(20000, 2.42, 4.27), (100000, 8.79, 4.84), (300000, 24.78, 8.93)]),
    (100, 3, 5000, 1e-3, [(2000, 0.29, 5.57), (300000, 8.05, 11.23)]),
    (7, 7, 2500, 1e-3, [(20000, 1.54, 2.25), (100000, 5.57, 2.56), (300000, 15.68, 4.64)]),
    (100, 7, 2500, 1e-3, [(20000, 0.51, 3.33), (300000, 4.94, 6.23)]),
]


@pytest.mark.parametrize("n,d,ordinals,prob,runs", MEASURED)
def test_the_measured_faster_kernel_is_taken(n, d, ordinals, prob, runs):
    spec = _noisy(n, d, ordinals, prob)
    for shots, planes, byte in runs:
        assert _route(spec, shots) == (1 if planes < byte else 0), shots


def test_ordinary_programs_take_planes():
    for shots in (2, 1000, 100000, 1000000):
        assert _route(workloads.surface_memory(7, 7, prob=0.001), shots) == 1
        for d in (2, 3, 5, 7):
            assert _route(workloads.random_hpc(60, d, 600, seed=1), shots) == 1


def test_flags_and_programs_without_planes():
    slow = _noisy(7, 7, 2500, 1e-3)
    assert _route(slow, 100000, _lib.FLAG_ROWS) == 1 and _route(slow, 100000) == 0
    spec = workloads.random_hpc(60, 3, 600, seed=1)
    assert not any(_route(spec, 1000, f) for f in (_lib.FLAG_NO_ROWS, _lib.FLAG_FORCE_GMEM)) and _route(spec, 1) == 0
    assert _route(workloads.random_hpc(60, 11, 600, seed=1), 1000, _lib.FLAG_ROWS) == 0
    twice = CircuitSpec(4, 3, [("CNOT", 1, 1, {}), ("M", 0, None, {})], "aliased")
    assert _route(twice, 1000, _lib.FLAG_ROWS) == 0
