"""GPU: the trace engines' tableau x / z passes for the programs that the row form
takes by default (SDIM_FLAG_NO_ROWS): the d = 2 pass over every row width, with
its snapshots, and every form of the odd-d pass, alone and in one batch, against
the oracle and the shot-group engine.  Each test first asserts the form."""
import numpy as np
import pytest

from sdim_gb300 import Program, _lib, workloads
from sdim_gb300.batch import BatchRunner
from tests.conftest import oracle_run

pytestmark = pytest.mark.gpu

TABLEAU = _lib.FLAG_TRACE | _lib.FLAG_NO_ROWS


def _takes_rows(prog, shots, flags):
    enc, ctx = prog.compile().enc, prog.context
    ops, probs = np.ascontiguousarray(enc.ops), np.ascontiguousarray(enc.probs)
    begin = np.array([0, ops.shape[0]], np.int64)
    n, d, s = np.array([enc.n], np.int32), np.array([enc.d], np.int32), np.array([shots], np.int64)
    out = np.zeros(1, np.uint8)
    _lib.check(ctx.lib.sdim_row_choice(1, ops.ctypes.data, begin.ctypes.data, probs.ctypes.data, n.ctypes.data,
                                       d.ctypes.data, s.ctypes.data, flags, ctx.num_sms, out.ctypes.data))
    return bool(out[0])


def _tableau(spec, shots, seed, shot0=0):
    prog = Program(spec.build())
    assert _takes_rows(prog, shots, _lib.FLAG_ROWS) and not _takes_rows(prog, shots, TABLEAU)
    return prog, prog.sample(shots, seed=seed, shot0=shot0, engine="tableau")


@pytest.mark.parametrize("n", [1, 5, 32, 33, 65, 97, 129])
def test_d2_row_widths_against_oracle(n):
    spec = workloads.random_hpc(n, 2, 6 * n + 20, seed=700 + n, mr_every=max(1, n // 2), mr_fraction=0.3)
    _, rec = _tableau(spec, 70, n)
    assert np.array_equal(rec, oracle_run([spec], n, 0, 70)["records"])


@pytest.mark.parametrize("n", [160, 257, 512, 700, 1500])
def test_d2_wide_rows_against_group_engine(n):
    base = workloads.random_hpc(n, 2, 3 * n, seed=950 + n, mr_every=n, mr_fraction=0.1)
    ops = []
    for op in base.ops:
        ops += [op] + [("N1", op[1], None, {"noise_channel": "d", "prob": 0.01})] * (op[0] in ("H", "CNOT"))
    prog, rec = _tableau(workloads.CircuitSpec(n, 2, ops, f"wide_n{n}"), 70, n)
    assert np.array_equal(rec, prog.sample(70, seed=n, engine="group"))


@pytest.mark.parametrize("seed", [1, 2])
def test_d2_every_gate_and_channel(seed):
    spec = workloads.all_gates_random(7, 2, 300, seed=seed, noise_probs=(0.0, 0.35, 1.0))
    _, rec = _tableau(spec, 130, seed, shot0=11)
    assert np.array_equal(rec, oracle_run([spec], seed, 11, 130)["records"])


@pytest.mark.parametrize("shots", [300, 100000])
def test_d2_memory_with_replay_and_with_columns(shots):
    spec = workloads.surface_memory(7, 7, prob=1e-3)
    prog, rec = _tableau(spec, shots, 2)
    assert np.array_equal(rec, prog.sample(shots, seed=2, engine="rows"))
    assert np.array_equal(rec[:32], oracle_run([spec], 2, 0, 32)["records"])


def test_d2_snapshot_slots_run_out():
    """n = 2048: a deterministic snapshot is 1 MB, so the 64 MB budget holds 64 of
    80 runs of deterministic measurements; the pass sums the rest's cross terms."""
    ops = [("H", q, None, {}) for q in range(160)]
    ops += [("CNOT", q, q + 1, {}) for q in range(0, 159, 2)]
    ops += [("P", q, None, {}) for q in range(1, 160, 3)]
    for q in range(80):
        ops += [("M", 2 * q, None, {}), ("M", 2 * q, None, {})]
    prog, rec = _tableau(workloads.CircuitSpec(2048, 2, ops), 64, 3)
    det = rec[0] >> 7
    assert det[1::2].all() and not det[0::2].any(), "the pairs should alternate random / deterministic"
    assert np.array_equal(rec, prog.sample(64, seed=3, engine="group"))


@pytest.mark.parametrize("d", [3, 5, 7])
@pytest.mark.parametrize("n", [1, 5, 33, 100])
def test_odd_d_against_oracle(d, n):
    spec = workloads.random_hpc(n, d, 5 * n + 20, seed=31 * d + n, mr_every=max(1, n // 2), mr_fraction=0.3)
    _, rec = _tableau(spec, 70, d + n, shot0=3)
    assert np.array_equal(rec, oracle_run([spec], d + n, 3, 70)["records"])


@pytest.mark.parametrize("d", [3, 5, 7])
@pytest.mark.parametrize("n", [170, 256, 700])
def test_odd_d_wide_against_group_engine(d, n):
    spec = workloads.random_hpc(n, d, 3 * n, seed=17 * d + n, mr_every=n, mr_fraction=0.1)
    prog, rec = _tableau(spec, 66, n)
    assert np.array_equal(rec, prog.sample(66, seed=n, engine="group"))


@pytest.mark.parametrize("large,modes", [(False, {0, 3, 4, 5, 7}), (True, {5, 6, 7, 8})], ids=["latency", "throughput"])
def test_a_batch_of_every_odd_d_form(large, modes):
    """One CTA, clusters in shared memory and streamed (few programs), or packed
    tableaux in shared and global memory (76 or more); and the bytes of d = 11."""
    sizes = [(40, 3), (300, 5), (500, 7), (700, 3), (260, 7), (190, 5), (800, 5), (331, 3), (200, 3), (60, 11), (250, 11)]
    if large:
        sizes += [(232 + 3 * i, (3, 5, 7)[i % 3]) for i in range(72)]
    br = BatchRunner()
    optin, sms = br.ctx.smem_optin, br.ctx.num_sms
    got = {br.ctx.lib.sdim_trace_xz_mode(n, d, len(sizes), 0, optin, sms) for n, d in sizes if d != 11}
    assert got == modes
    specs = [workloads.random_hpc(n, d, 3 * n, seed=i, mr_every=n, mr_fraction=0.2) for i, (n, d) in enumerate(sizes)]
    for i, s in enumerate(specs):
        br.add_spec(s, 16 + 8 * (i % 30), seed=30 + i, shot0=i)
    for e, s, out in zip(br.entries, specs, br.run(engine="tableau")):
        prog = Program(s.build())
        assert np.array_equal(out, prog.sample(e.shots, seed=e.seed, shot0=e.shot0, engine="group")), s.name


def test_flags_of_the_row_form_are_exclusive():
    prog = Program(workloads.random_hpc(20, 3, 100, seed=1).build())
    assert not _takes_rows(prog, 1000, _lib.FLAG_ROWS | _lib.FLAG_NO_ROWS)
    for flag in (_lib.FLAG_SPLIT_XZ, _lib.FLAG_CLUSTER_XZ, _lib.FLAG_U8_XZ, _lib.FLAG_PACKED_XZ, _lib.FLAG_UNLAYERED):
        assert not _takes_rows(prog, 1000, _lib.FLAG_ROWS | flag)
