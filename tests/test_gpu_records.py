"""GPU: the record pass's output (trace_cols.cuh) -- 16 bytes at a time cut out
of the shots' record bits -- at record widths on both sides of 16 bytes and of
a record word, output pointers off the 16-byte boundary, a partial last group,
and a shot group across a multiple of 2^32, against the phase replay."""
import numpy as np
import pytest
import torch

from sdim_gb300 import Program, _lib
from sdim_gb300.batch import BatchRunner
from sdim_gb300.workloads import CircuitSpec

pytestmark = pytest.mark.gpu

REPLAY = _lib.FLAG_TRACE | _lib.FLAG_PHASE_REPLAY


def _program(nm, seed):
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(nm):
        for g in ("H", "P", "N1"):
            ops.append((g, int(rng.integers(4)), None, {"prob": 0.05, "noise_channel": "d"} if g == "N1" else {}))
        a, b = rng.permutation(4)[:2]
        ops += [("CNOT", int(a), int(b), {}), (("M", "RESET")[int(rng.integers(2))], int(rng.integers(4)), None, {})]
    return Program(CircuitSpec(4, 2, ops, "records").build())


def _replay(prog, shots, seed, shot0):
    dp, ctx = prog.compile(), prog.context
    out = np.zeros((shots, dp.num_records), dtype=np.uint8)
    _lib.check(ctx.lib.sdim_run(ctx.ptr, dp.ptr, seed, shot0, shots, out.ctypes.data, REPLAY), ctx.ptr, "run")
    return out


@pytest.mark.parametrize("nm", [1, 2, 7, 15, 16, 17, 31, 32, 33, 63, 64, 65, 96, 250, 513])
@pytest.mark.parametrize("off,shot0", [(0, 0), (5, 3), (16, 2**32 - 10020)])
def test_record_bytes_at_any_width_and_address(nm, off, shot0):
    prog, shots = _program(nm, 10 * nm + off), 20011
    br = BatchRunner(prog.context)
    br.add_program(prog.compile(), shots, 7, shot0)
    out = torch.full((off + shots * nm + 16,), 99, dtype=torch.uint8, device="cuda")
    br.run_device([out.data_ptr() + off], engine="trace", time_kernels=True)
    assert prog.context.last_passes_ms()[2] > 0.0, "the column pass did not run"
    got = out.cpu().numpy()
    assert np.array_equal(got[off : off + shots * nm].reshape(shots, nm), _replay(prog, shots, 7, shot0))
    assert (got[:off] == 99).all() and (got[off + shots * nm :] == 99).all()


@pytest.mark.parametrize("d,nms", [(2, (1, 15, 16, 17, 33, 385, 3100)), (3, (1, 16, 31, 65, 1600)),
                                   (5, (1, 17, 64, 1100)), (7, (1, 16, 33, 1100))])
def test_frame_records_at_any_width(d, nms):
    """The frame route's output pass: whole rows in shared memory and, past
    its limit, a byte at a time; a partial last group; against the frame oracle."""
    import oracle
    from oracle import frame
    rng = np.random.default_rng(d)
    for nm in nms:
        ops = [("H", 0, None, {}), ("CNOT", 0, 1, {}), ("H", 2, None, {}), ("N1", 1, None, {"prob": 0.3, "noise_channel": "d"})]
        for k in range(nm):
            ops.append((("M", "RESET")[int(rng.integers(8) == 0)], int(rng.integers(4)), None, {}))
            if k % 5 == 0:
                ops += [("H", int(rng.integers(4)), None, {}), ("N1", 2, None, {"prob": 0.1, "noise_channel": "f"})]
        spec = CircuitSpec(4, d, ops, "widths")
        rec = Program(spec.build()).sample_frames(70, seed=nm)
        want = frame.simulate(oracle.OracleProgram([spec], 4, d), nm, 70)
        assert np.array_equal(rec, want), nm
