"""GPU: sdim_program_bytes holds the row form's memory and the trace that it
writes, for every d that has one."""
import ctypes as C

import numpy as np
import pytest

from sdim_gb300 import _lib, workloads
from sdim_gb300.encode import DeviceProgram, encode_program

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("n", [3, 40, 300])
def test_row_form_memory_is_counted(d, n):
    ctx = _lib.Context.default(0)
    spec = workloads.random_hpc(n, d, 6 * n, seed=n, mr_every=n, mr_fraction=0.2)
    enc = encode_program([spec.build()], n, d)
    prog = DeviceProgram(ctx, enc)
    info, out = (C.c_int64 * 6)(), (C.c_int64 * 2)()
    ops = np.ascontiguousarray(enc.ops)
    assert ctx.lib.sdim_row_program(ops.ctypes.data, int(ops.shape[0]), None, n, d, info) == _lib.SDIM_OK
    assert ctx.lib.sdim_program_bytes(prog.ptr, 10, out) == _lib.SDIM_OK
    trace = prog.num_records * (16 + 2 * n // 8)  # a header and a bit per residue of the factor row at least
    assert out[0] == 10 * prog.num_records and out[1] >= prog.group_slot_bytes + trace + info[5]
