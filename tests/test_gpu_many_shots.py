"""GPU: the row form's phase pass at the largest shot count of a call, 2^31 - 1
(its blocks were counted in 32 bits, past the last 127 shots of that range):
pieces of the records equal runs of those shots alone."""
import numpy as np
import pytest
import torch

from sdim_gb300 import _lib
from sdim_gb300.encode import DeviceProgram, encode_program
from sdim_gb300.workloads import CircuitSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,flags", [(3, _lib.FLAG_ROWS), (2, _lib.FLAG_ROWS | _lib.FLAG_PHASE_REPLAY)])
def test_the_largest_shot_count(d, flags):
    ctx = _lib.Context.default(0)
    spec = CircuitSpec(1, d, [("H", 0, None, {}), ("M", 0, None, {})], "one")
    prog = DeviceProgram(ctx, encode_program([spec.build()], 1, d))
    shots = 2**31 - 1
    out = torch.full((shots + 1,), 99, dtype=torch.uint8, device="cuda")

    def run(first, count, dst):
        rc = ctx.lib.sdim_run_device(ctx.ptr, prog.ptr, 77, first, count, dst.data_ptr(), None, flags)
        _lib.check(rc, ctx.ptr, "run")

    run(0, shots, out)
    assert int(out[shots]) == 99
    piece = torch.empty(1000, dtype=torch.uint8, device="cuda")
    for first in (0, 2**30, shots - 1000):
        run(first, 1000, piece)
        assert torch.equal(out[first : first + 1000], piece), first
    head = np.bincount(out[: 1 << 20].cpu().numpy(), minlength=d)
    assert (abs(head[:d] / head.sum() - 1 / d) < 0.01).all()
    del out
    torch.cuda.empty_cache()
