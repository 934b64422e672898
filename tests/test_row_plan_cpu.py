"""CPU: the launch shape of the row form's raw pass (abi.cu: plan_row_group,
through the host-only sdim_row_plan).  A thread of a raw-pass CTA serves one
column word and strides over a layer's ops in steps of threads / words, so a CTA
needs whole multiples of its words in threads, whatever the number of
measurements (each owns a column) and of programs in the launch."""
import ctypes as C

import numpy as np
import pytest

from sdim_gb300 import _lib, workloads

OPTIN, SMS = 232448, 152
E_BYTES = {2: 16, 3: 8, 5: 16, 7: 16}  # a column word in the raw pass


def _row_program(spec):
    ops = np.ascontiguousarray(spec.op_table(), dtype=np.int32)
    out = (C.c_int64 * 6)()
    rc = _lib.load().sdim_row_program(ops.ctypes.data, int(ops.shape[0]), None, spec.num_qudits, spec.dimension, out)
    assert rc == _lib.SDIM_OK
    return list(out)


def _plan(d, ns, programs):
    n = np.ascontiguousarray(ns, dtype=np.int32)
    p = np.ascontiguousarray(programs, dtype=np.int64)
    out = (C.c_int32 * 8)()
    rc = _lib.load().sdim_row_plan(d, len(ns), n.ctypes.data, p.ctypes.data, OPTIN, SMS, out)
    return rc, dict(zip(("ctas", "cblock", "rawt", "lg", "block", "tiles", "units", "xctas"), out))


def _sound(plan, ns, d):
    words, threads = 1 << plan["lg"], plan["rawt"] or plan["block"]
    assert 32 <= threads <= 512 and threads % words == 0, plan
    if plan["rawt"]:
        assert plan["rawt"] <= plan["cblock"], plan
        assert plan["ctas"] * words >= plan["units"], plan
    else:
        assert plan["tiles"] * words >= plan["units"], plan
    assert 2 * max(ns) * words * E_BYTES[d] <= OPTIN, plan


def _repeated(n, d, measurements):
    """M on every qudit over and over, with a gate in front of the last."""
    ops = [("H", q, None, {}) for q in range(n)] + [("CNOT", 0, n - 1, {})]
    ops += [("M", k % n, None, {}) for k in range(measurements)]
    return workloads.CircuitSpec(n, d, ops + [("H", 0, None, {}), ("M", 0, None, {})], "repeated")


@pytest.mark.parametrize("programs,measurements", [(80, 16500), (40, 33000), (152, 16500)])
def test_long_narrow_programs_in_one_launch(programs, measurements):
    info = _row_program(_repeated(4, 2, measurements))
    info = info if info[0] else [measurements + 7, 33, measurements + 1, 0, measurements, 0]
    rc, plan = _plan(2, [4] * programs, [info] * programs)
    assert rc == _lib.SDIM_OK and plan["units"] > 512
    _sound(plan, [4], 2)


@pytest.mark.parametrize("d", [2, 3, 5, 7])
def test_one_long_program_among_small_ones(d):
    small = _row_program(workloads.random_hpc(3, d, 20, seed=1))
    for columns in (200, 5000, 16500, 60000):
        for others in (0, 1, 15, 76, 151, 152, 400):
            long = [columns + 9, 40, columns + 1, 0, columns, 0]
            rc, plan = _plan(d, [4] + [3] * others, [long] + [small] * others)
            assert rc == _lib.SDIM_OK
            _sound(plan, [4], d)


@pytest.mark.parametrize("d", [2, 3, 5, 7])
def test_plans_over_sizes(d):
    for n in (1, 32, 33, 64, 65, 128, 129, 256, 257, 768, 769, 2048):
        for columns in (0, 31, 700, 9000):
            for count in (1, 2, 19, 38, 76, 77, 152, 153, 1000):
                for layers in (1, 30, 4000):
                    rc, plan = _plan(d, [n] * count, [[4 * n + columns, layers, columns + 1, 7, columns, 0]] * count)
                    assert rc == _lib.SDIM_OK
                    _sound(plan, [n], d)


def test_row_program_of_tables():
    assert _row_program(workloads.random_hpc(8, 3, 60, seed=2))[0] > 0
    twice = workloads.CircuitSpec(4, 3, [("CNOT", 1, 1, {}), ("M", 0, None, {})], "aliased")
    assert _row_program(twice)[0] == 0
    assert _row_program(workloads.random_hpc(8, 11, 60, seed=2))[0] == 0
    assert _row_program(workloads.CircuitSpec(4, 2, [("H", 1, None, {})], "unmeasured"))[0] == 0
    ops = np.array([[9, 0, 5, 0]], dtype=np.int32)
    assert _lib.load().sdim_row_program(ops.ctypes.data, 1, None, 2, 2, (C.c_int64 * 6)()) == _lib.SDIM_EINVAL


def test_plan_refuses_mixed_groups():
    one = [10, 3, 4, 0, 0, 0]
    assert _plan(2, [4, 300], [one, one])[0] == _lib.SDIM_EINVAL
    assert _plan(11, [4], [one])[0] == _lib.SDIM_EINVAL
    assert _plan(2, [4], [[0] * 6])[0] == _lib.SDIM_EINVAL
