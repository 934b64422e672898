"""Measured cases: what a user of this framework has it do, through its public entry points.

Every case is a dict of plain values whose ``kind`` names the call:

* ``sample``  -- ``Program.sample``: records of the tableau route in host memory;
* ``frames``  -- ``Program.sample_frames``: records of the Pauli-frame route in host memory;
* ``device``  -- ``BatchRunner.run_device``: one program's tableau-route records into device memory;
* ``frames_device`` -- ``sdim_frame_run`` of the C ABI with a device output (``SDIM_FLAG_OUT_DEVICE``);
* ``batch``   -- ``BatchRunner.run_device`` of many uneven programs;
* ``serve``   -- ``Server.submit`` of a burst of requests and their results;
* ``graph``   -- ``BatchRunner.capture`` once, then ``CapturedRun.launch`` with fresh seeds.

Circuits come from ``sdim_gb300.workloads`` and are drawn from the seed (the surface-code memory is one
circuit per size; its shots are drawn from the seed; the sizes of a batch are the case's own).  All outputs are
whole records, one byte per measurement and shot (value | deterministic << 7): whole numbers, so there is
nothing for ``exact`` to say.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from sdim_gb300 import Program, _lib, workloads
from sdim_gb300.batch import BatchRunner
from sdim_gb300.encode import DeviceProgram, encode_program, encode_table
from sdim_gb300.serving import Server


def listed():
    return [
        # one shot of a small program: the first thing every user runs; launches and host work only
        {"name": "one_shot_small", "kind": "sample", "circuit": "random", "d": 3, "n": 6, "gates": 40, "mr": 0,
         "shots": 1},
        # a small error-correction experiment sampled into host memory
        {"name": "surface3_host", "kind": "sample", "circuit": "surface", "d": 2, "distance": 3, "rounds": 3,
         "prob": 0.001, "shots": 2000},
        # the headline: distance-7 memory, 100,000 noisy shots left on the device for a decoder
        {"name": "surface7_device", "kind": "device", "circuit": "surface", "d": 2, "distance": 7, "rounds": 7,
         "prob": 0.001, "shots": 100000},
        # the single-circuit qutrit workload of the benchmark
        {"name": "qutrit32_device", "kind": "device", "circuit": "random", "d": 3, "n": 32, "gates": 640, "mr": 0,
         "shots": 1024},
        # the odd-d workload of the benchmark: mid-circuit MEASURE + RESET, then MEASURE on all
        {"name": "odd5_256_device", "kind": "device", "circuit": "random", "d": 5, "n": 256, "gates": 2560,
         "mr": 256, "shots": 4096},
        # a wide program with a few shots, as the request stream holds them; ragged qudit count
        {"name": "odd7_517_few", "kind": "device", "circuit": "random", "d": 7, "n": 517, "gates": 4136, "mr": 0,
         "shots": 19},
        # a wide qubit program without structure
        {"name": "qubit_451_device", "kind": "device", "circuit": "random", "d": 2, "n": 451, "gates": 3608,
         "mr": 0, "shots": 1500},
        # the multi-shot route of simulate() (Pauli frames) at the headline size
        {"name": "frames_surface7", "kind": "frames_device", "circuit": "surface", "d": 2, "distance": 7,
         "rounds": 7, "prob": 0.001, "shots": 100000},
        # the same route for a noisy qudit circuit, records in host memory
        {"name": "frames_qutrit_host", "kind": "frames", "circuit": "noisy", "d": 3, "n": 48, "gates": 480,
         "mr": 120, "prob": 0.01, "shots": 10000},
        # many independent programs of uneven size and few shots in one call
        {"name": "uneven_batch_384", "kind": "batch", "programs": 384, "n_min": 8, "n_max": 1024, "shots_max": 64,
         "mix": 1},
        # a burst of requests to the serving loop
        {"name": "serve_burst_40", "kind": "serve", "requests": 40, "n_min": 16, "n_max": 512, "shots_max": 10000,
         "mix": 2},
        # a sampling loop that replays one captured step over fresh seeds
        {"name": "graph_surface5", "kind": "graph", "circuit": "surface", "d": 2, "distance": 5, "rounds": 5,
         "prob": 0.003, "shots": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample", "device", "device", "device", "surface", "frames", "frames_device", "batch",
                       "serve", "graph"])
    if kind == "batch":
        return {"kind": "batch", "programs": _log(rng, 12, 384), "n_min": rng.randint(4, 16),
                "n_max": _log(rng, 48, 1024), "shots_max": rng.randint(1, 64), "mix": rng.randint(10, 10**6)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(4, 40), "n_min": rng.randint(8, 24),
                "n_max": _log(rng, 48, 512), "shots_max": _log(rng, 100, 10000), "mix": rng.randint(10, 10**6)}
    if kind in ("surface", "graph"):
        L = rng.choice([3, 4, 5, 6, 7])
        return {"kind": "graph" if kind == "graph" else rng.choice(["sample", "device", "frames_device"]),
                "circuit": "surface", "d": 2, "distance": L, "rounds": rng.randint(1, L),
                "prob": rng.choice([0.0005, 0.001, 0.003, 0.01]), "shots": _log(rng, 100, 100000)}
    d = rng.choice([2, 3, 5, 7])
    if kind == "sample":
        n = _log(rng, 2, 48)
        return {"kind": kind, "circuit": "random", "d": d, "n": n, "gates": n * rng.randint(4, 12),
                "mr": rng.choice([0, 0, 2 * n]), "shots": _log(rng, 1, 4000)}
    if kind == "device":
        n = _log(rng, 8, 600)
        # records times shots stay below the headline's
        return {"kind": kind, "circuit": "random", "d": d, "n": n, "gates": n * rng.randint(4, 10),
                "mr": rng.choice([0, 0, n]), "shots": _log(rng, 1, max(2, min(8192, 2000000 // n)))}
    n = _log(rng, 4, 160)
    return {"kind": kind, "circuit": "noisy", "d": d, "n": n, "gates": n * rng.randint(4, 12),
            "mr": rng.choice([0, 2 * n]), "prob": rng.choice([0.001, 0.01, 0.05]), "shots": _log(rng, 100, 20000)}


# --------------------------------------------------------------------------------------------------------
def _spec(case, seed):
    """The case's circuit: a random one is drawn from the seed."""
    if case["circuit"] == "surface":
        return workloads.surface_memory(case["distance"], case["rounds"], prob=case["prob"])
    spec = workloads.random_hpc(case["n"], case["d"], case["gates"], seed=seed, mr_every=case["mr"],
                                mr_fraction=0.1)
    if case["circuit"] == "noisy":  # depolarizing noise after every gate, on each qudit that it touches
        ops = []
        for name, q, t, params in spec.ops:
            ops.append((name, q, t, params))
            if name in ("H", "P", "CNOT"):
                for x in (q,) if t is None else (q, t):
                    ops.append(("N1", x, None, {"prob": case["prob"], "noise_channel": "d"}))
        spec = workloads.CircuitSpec(case["n"], case["d"], ops, "noisy")
    return spec


def _mix(case):
    """(n, d, shots) of every program of a batch or burst: n log-uniform, d uniform; fixed by the case."""
    rng = np.random.Generator(np.random.PCG64(case["mix"]))
    batch = case["kind"] == "batch"
    sizes = []
    for _ in range(case["programs"] if batch else case["requests"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        d = int(rng.choice((2, 3, 5, 7) if batch else (2, 3, 5)))
        top = case["shots_max"]
        shots = rng.integers(1, top + 1) if batch else round(math.exp(rng.uniform(0, math.log(top))))
        sizes.append((n, d, int(shots)))
    return sizes


def _uneven(case, seed):
    """The programs of a batch (4 gates per qudit) or burst (8), drawn from the seed."""
    rng = np.random.Generator(np.random.PCG64(seed))
    per = 4 if case["kind"] == "batch" else 8
    return [workloads.BatchItem(workloads.random_hpc(n, d, per * n, seed=rng), shots, 1000003 * (seed % 1000003) + i)
            for i, (n, d, shots) in enumerate(_mix(case))]


def _device_program(ctx, spec, noise=True):
    if spec.table is not None:
        return DeviceProgram(ctx, encode_table(spec.table, spec.num_qudits, spec.dimension))
    return DeviceProgram(ctx, encode_program([spec.build()], spec.num_qudits, spec.dimension, noise=noise))


_server = None  # a serving program keeps its server running


def prepare(case, seed):
    global _server
    kind = case["kind"]
    s = {"kind": kind, "seed": 1000003 * (seed % 1000003) + 17}
    if kind in ("sample", "frames"):
        s["program"] = Program(_spec(case, seed).build())
        s["program"].compile()
        if kind == "frames":
            s["program"].compile(False)
        s["shots"] = case["shots"]
        return s
    if kind == "serve":
        if _server is None:
            _server = Server()
        s["items"] = _uneven(case, seed)
        for it in s["items"]:
            it.spec.op_table()
        return s
    ctx = _lib.Context.default(0)
    s["ctx"] = ctx
    if kind == "batch":
        s["runner"] = BatchRunner(ctx)
        for it in _uneven(case, seed):
            s["runner"].add_spec(it.spec, it.shots, it.seed)
    elif kind == "frames_device":
        spec = _spec(case, seed)
        s["noisy"], s["quiet"] = _device_program(ctx, spec), _device_program(ctx, spec, noise=False)
        s["shots"] = case["shots"]
        s["out"] = torch.empty((case["shots"], s["noisy"].num_records), dtype=torch.uint8, device="cuda")
        return s
    else:
        s["runner"] = BatchRunner(ctx)
        s["runner"].add_program(_device_program(ctx, _spec(case, seed)), case["shots"], s["seed"])
    sizes = [e.shots * e.program.num_records for e in s["runner"].entries]
    s["out"] = torch.empty(sum(sizes), dtype=torch.uint8, device="cuda")
    s["ptrs"] = [s["out"].data_ptr() + sum(sizes[:i]) for i in range(len(sizes))]
    if kind == "graph":
        s["captured"] = s["runner"].capture(s["ptrs"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "sample":
        return s["program"].sample(s["shots"], seed=s["seed"])
    if kind == "frames":
        return s["program"].sample_frames(s["shots"], seed=s["seed"])
    if kind == "frames_device":
        ctx = s["ctx"]
        rc = ctx.lib.sdim_frame_run(ctx.ptr, s["noisy"].ptr, s["quiet"].ptr, C.c_uint64(s["seed"]), s["shots"],
                                    s["out"].data_ptr(), _lib.FLAG_OUT_DEVICE)
        _lib.check(rc, ctx.ptr, "frames")
        return s["out"]
    if kind == "serve":
        reqs = [_server.submit(it.spec.table, it.spec.num_qudits, it.spec.dimension, it.shots, it.seed)
                for it in s["items"]]
        return np.concatenate([r.wait(60.0).reshape(-1) for r in reqs])
    if kind == "graph":
        s["captured"].launch(seeds=[s["seed"]])
        s["captured"].sync()
        return s["out"]
    s["runner"].run_device(s["ptrs"])
    return s["out"]


# --------------------------------------------------------------------------------------------------------
def _size(case):
    """(qudits, instructions, records, N1 instructions) of a case's circuit."""
    if case["circuit"] == "surface":
        L, r = case["distance"], case["rounds"]
        x, z = workloads.surface_layout(L)
        cnots = sum(c is not None for check in x + z for c in check)
        gates, resets = r * (2 * len(x) + cnots), r * (L * L - 1)
        n1 = r * (2 * len(x) + 2 * cnots) + resets
        return 2 * L * L - 1, gates + resets + L * L + n1, resets + L * L, n1
    resets = (case["gates"] // case["mr"]) * int(round(0.1 * case["n"])) if case["mr"] else 0
    n1 = case["gates"] * 4 // 3 if case["circuit"] == "noisy" else 0
    return case["n"], case["gates"] + resets + case["n"] + n1, resets + case["n"], n1


def _one(d, n, instr, records, n1, shots):
    # read: the program's rows (16 bytes each); written: the records.  Operations: the x / z part once
    # (a rank-1 update of 2n x n residue pairs for half of the records, a column of 2n for the rest), per
    # shot a coin per N1 and a draw per record (a quarter of a Philox block of about 100 operations each)
    # and its share of the records' linear combinations.
    ops = records * (2.0 * n * n) + instr * 4.0 * n + shots * (25.0 * (n1 + records) + records)
    return 16.0 * instr + float(shots) * records, ops


def work(case):
    if case["kind"] in ("batch", "serve"):
        per = 4 if case["kind"] == "batch" else 8
        parts = [_one(d, n, (per + 1) * n, n, 0, shots) for n, d, shots in _mix(case)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    n, instr, records, n1 = _size(case)
    b, f = _one(case["d"], n, instr, records, n1, case["shots"])
    return {"bytes": b, "flops": f}
