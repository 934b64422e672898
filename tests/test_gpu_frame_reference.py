"""GPU: the frame route's reference shot runs beside the frames, so it shares no
buffer with them: a reference program that holds N1 instructions itself (of
probability 0, or the noisy program as its own reference) gives the records of
the byte-per-shot route, which runs the two one behind the other; and frames in
more than one part of the mask budget."""
import ctypes as C

import numpy as np
import pytest

from sdim_gb300 import _lib, workloads
from sdim_gb300.encode import DeviceProgram, encode_program
from sdim_gb300.workloads import CircuitSpec

pytestmark = pytest.mark.gpu


def _frames(ctx, prog, ref, seed, shots, flags=0):
    out = np.zeros((shots, prog.num_records), dtype=np.uint8)
    rc = ctx.lib.sdim_frame_run(ctx.ptr, prog.ptr, ref.ptr, C.c_uint64(seed), shots, out.ctypes.data, flags)
    _lib.check(rc, ctx.ptr, "frames")
    return out


def _noisy(d):
    if d == 2:
        return workloads.surface_memory(3, 3, prob=0.02)
    return workloads.all_gates_random(9, d, 400, seed=d, noise_probs=(0.02,), name="noisy")


@pytest.mark.parametrize("d", [2, 3, 5, 7])
@pytest.mark.parametrize("shots", [40, 20000])
def test_reference_programs_with_noise(d, shots):
    ctx = _lib.Context(0)  # fresh buffers: they grow while both run
    spec = _noisy(d)
    noisy = DeviceProgram(ctx, encode_program([spec.build()], spec.num_qudits, d))
    quiet = DeviceProgram(ctx, encode_program([spec.build()], spec.num_qudits, d, noise=False))
    off_spec = CircuitSpec(spec.num_qudits, d, [(g, q, t, dict(p, prob=0.0) if g == "N1" else p) for g, q, t, p in spec.ops],
                           "off")
    off = DeviceProgram(ctx, encode_program([off_spec.build()], spec.num_qudits, d))
    for seed in range(3):
        want = _frames(ctx, noisy, quiet, seed, shots, _lib.FLAG_FORCE_GMEM)
        assert np.array_equal(_frames(ctx, noisy, quiet, seed, shots), want)
        for _ in range(4):
            assert np.array_equal(_frames(ctx, noisy, off, seed, shots), want), "N1 of probability 0"
        own = _frames(ctx, noisy, noisy, seed, shots, _lib.FLAG_FORCE_GMEM)
        for flags in (0, _lib.FLAG_COLUMNS, _lib.FLAG_PHASE_REPLAY, _lib.FLAG_REUSE_XZ, _lib.FLAG_REUSE_XZ):
            assert np.array_equal(_frames(ctx, noisy, noisy, seed, shots, flags), own), flags
    ctx.close()


def test_a_reference_with_more_masks_than_the_frames():
    """The reference holds more N1 ordinals than the program itself."""
    ctx = _lib.Context(0)
    spec = _noisy(2)
    more = []
    for op in spec.ops:
        more += [op] * (30 if op[0] == "N1" else 1)
    noisy = DeviceProgram(ctx, encode_program([spec.build()], spec.num_qudits, 2))
    ref = DeviceProgram(ctx, encode_program([CircuitSpec(spec.num_qudits, 2, more, "more").build()], spec.num_qudits, 2))
    want = _frames(ctx, noisy, ref, 4, 9000, _lib.FLAG_FORCE_GMEM)
    assert np.array_equal(_frames(ctx, noisy, ref, 4, 9000), want)
    ctx.close()


def test_frames_in_two_parts():
    """20,000 N1 ordinals: about 5 KB of masks a shot, so 115,000 shots pass
    the 512 MB of a part."""
    rng = np.random.default_rng(5)
    ops = []
    for k in range(20000):
        a, b = (int(x) for x in rng.permutation(6)[:2])
        if k % 4 == 0:
            ops.append(("CNOT", a, b, {}) if k % 8 else ("H", a, None, {}))
        ops.append(("N1", a, None, {"prob": 0.0005, "noise_channel": "dfp"[k % 3]}))
        if k % 1500 == 0:
            ops.append((("M", "RESET")[k % 2], b, None, {}))
    ops += [("M", q, None, {}) for q in range(6)]
    spec = CircuitSpec(6, 2, ops, "parts")
    ctx = _lib.Context.default(0)
    noisy = DeviceProgram(ctx, encode_program([spec.build()], 6, 2))
    quiet = DeviceProgram(ctx, encode_program([spec.build()], 6, 2, noise=False))
    shots = 115000
    assert np.array_equal(_frames(ctx, noisy, quiet, 9, shots), _frames(ctx, noisy, quiet, 9, shots, _lib.FLAG_FORCE_GMEM))


@pytest.mark.parametrize("d", [2, 3, 5, 7])
def test_both_kernels_give_the_records(d):
    """On bit planes, as bytes, and as the run's estimate has it, for a program of
    so many ordinals that it takes both by the number of its shots."""
    rng = np.random.default_rng(d)
    ops = []
    for k in range(60000 if d == 2 else 2400):
        a, b = (int(x) for x in rng.permutation(7)[:2])
        ops += [("CNOT", a, b, {}), ("N1", a, None, {"prob": 0.001, "noise_channel": "dfp"[k % 3]})]
        if k % 400 == 0:
            ops.append((("M", "RESET")[k // 400 % 2], b, None, {}))
    spec = CircuitSpec(7, d, ops + [("M", q, None, {}) for q in range(7)], "many")
    ctx = _lib.Context.default(0)
    noisy = DeviceProgram(ctx, encode_program([spec.build()], 7, d))
    quiet = DeviceProgram(ctx, encode_program([spec.build()], 7, d, noise=False))
    for shots in (50, 130000):
        want = _frames(ctx, noisy, quiet, 3, shots, _lib.FLAG_NO_ROWS)
        for flags in (0, _lib.FLAG_ROWS, _lib.FLAG_FORCE_GMEM):
            assert np.array_equal(_frames(ctx, noisy, quiet, 3, shots, flags), want), (shots, flags)


def test_frames_without_room_for_the_masks():
    """A device whose memory is taken: the masks of a part (about 350 MB) do not
    fit, and the byte kernel takes the run."""
    import torch
    rng = np.random.default_rng(3)
    ops = []
    for k in range(40000):
        a, b = (int(x) for x in rng.permutation(6)[:2])
        ops += [("CNOT", a, b, {})] * (k % 3 == 0) + [("N1", a, None, {"prob": 0.0005, "noise_channel": "d"})]
    spec = CircuitSpec(6, 2, ops + [("M", q, None, {}) for q in range(6)], "room")
    ctx = _lib.Context(0)
    noisy = DeviceProgram(ctx, encode_program([spec.build()], 6, 2))
    quiet = DeviceProgram(ctx, encode_program([spec.build()], 6, 2, noise=False))
    shots = 34000
    want = _frames(ctx, noisy, quiet, 5, shots, _lib.FLAG_NO_ROWS)
    torch.cuda.synchronize()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = _frames(ctx, noisy, quiet, 5, shots, _lib.FLAG_ROWS)
    finally:
        del taken
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
    ctx.close()
