"""The work a user of qcb200 has it do, as cases that can be timed.

Every case goes through the public entry points: the Python functions of
`qcb200`, and the C ABI of include/qcb200.h where a program keeps its data on
the device.  Sizes are those of the benchmark's configurations, the test suite
and generic ones between them.  All outputs are whole numbers (bits, phases,
indices), which have to be equal, so there is no `exact` value to compare
against.

Kinds of cases
  call     pftrajectories(circuit; trajectories) and measurements(frame): a
           notebook's call, everything from the compiler to the Bool matrix
  sample   a sampling program that keeps its frame and its compiled circuit:
           a fresh run, then the shot-major syndrome matrix left on the device
           for a decoder
  batch    many such runs of different circuits drained by one launch
  mul      mul_left! on Paulis in the caller's device memory
  canon    canonicalize! of a resident state, read back
  project  project! of a list of Paulis in order on a resident state
  dense    dense apply! of a Clifford operator, some time steps, read back
  gates    symbolic apply! of a gate list, read back
"""
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantumclifford.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import qcb200  # noqa: E402
from qcb200 import circuits, ops  # noqa: E402

DEVICE = "cuda"


def listed():
    return [
        # the repetition-code memory of the benchmark's first configuration: the smallest call,
        # where compiling, allocating and copying count
        {"name": "call_rep7_10k", "kind": "call", "code": "rep", "d": 7, "rounds": 7, "p": 1e-3, "shots": 10_000},
        # the headline configuration, with its syndromes handed over on the device
        {"name": "sample_d11_1e6", "kind": "sample", "d": 11, "rounds": 11, "p": 1e-3, "shots": 1_000_000},
        # a tall circuit, strong noise, a ragged number of shots: the upper end of the serving mix
        {"name": "sample_d21_150k", "kind": "sample", "d": 21, "rounds": 21, "p": 4e-3, "shots": 150_001},
        # the batched workload: uneven circuits, noise strengths and shot counts
        {"name": "batch_24_surface", "kind": "batch", "jobs": 24, "dmax": 13, "smax": 300_000},
        # mul_left! of two Paulis on 1e9 qubits, memory bound
        {"name": "mul_1e9", "kind": "mul", "n": 1_000_000_000, "count": 1, "phases": True},
        # canonicalize! at a code's size, at the sizes of the benchmark and its largest
        {"name": "canon_100", "kind": "canon", "n": 100, "phases": True},
        {"name": "canon_1000", "kind": "canon", "n": 1000, "phases": True},
        {"name": "canon_4000", "kind": "canon", "n": 4000, "phases": True},
        # 1000 Paulis measured in order: a simulation's state with its destabilizers, and a tall stabilizer state
        {"name": "project_destab_1000", "kind": "project", "state": "Destabilizer", "n": 1000, "k": 1000},
        {"name": "project_stab_4000", "kind": "project", "state": "Stabilizer", "n": 4000, "k": 1000},
        # four time steps of tensor_pow(tCNOT, 500) on a random 1000-qubit stabilizer state
        {"name": "dense_1000x4", "kind": "dense", "n": 1000, "op": "tCNOT", "steps": 4},
        # a random circuit of H, S and CNOT layers on a 500-qubit state with its destabilizers
        {"name": "gates_500", "kind": "gates", "n": 500, "depth": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["call", "sample", "sample", "batch", "mul", "canon", "canon", "project", "project", "dense", "gates"])
    if kind == "call":
        d = rng.randrange(3, 16)
        return {"kind": kind, "code": "rep", "d": d, "rounds": rng.randrange(1, 16), "p": 10 ** rng.uniform(-4, -2),
                "shots": _log(rng, 100, 100_000)}
    if kind == "sample":
        d = rng.randrange(3, 23, 2)
        return {"kind": kind, "d": d, "rounds": d, "p": 10 ** rng.uniform(-4, -2),
                "shots": _log(rng, 1000, 1_000_000 if d <= 11 else 150_000)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randrange(4, 25), "dmax": rng.choice([7, 11, 13]), "smax": _log(rng, 2000, 300_000)}
    if kind == "mul":
        n = _log(rng, 500, 1_000_000_000)
        return {"kind": kind, "n": n, "count": min(4096, _log(rng, 1, max(1, 1_000_000_000 // n))), "phases": rng.random() < 0.75}
    if kind == "canon":
        return {"kind": kind, "n": _log(rng, 16, 4000), "phases": rng.random() < 0.75}
    if kind == "project":
        state = rng.choice(["Stabilizer", "MixedStabilizer", "Destabilizer", "MixedDestabilizer"])
        n = _log(rng, 100, 4000 if state in ("Stabilizer", "MixedStabilizer") else 1500)
        return {"kind": kind, "state": state, "n": n, "k": _log(rng, 50, 1000)}
    if kind == "dense":
        n = _log(rng, 40, 1500)
        op = rng.choice(["tCNOT", "random"])
        return {"kind": kind, "n": n - n % 2 if op == "tCNOT" else n, "op": op, "steps": rng.randrange(1, 5)}
    return {"kind": "gates", "n": _log(rng, 30, 1000), "depth": rng.randrange(1, 6)}


def _circuit(case):
    if case.get("code") == "rep":
        return ops.to_array(circuits.repetition_code_memory(case["d"], case["rounds"], case["p"]))
    return ops.to_array(circuits.rotated_surface_code_memory(case["d"], case["rounds"], case["p"]))


def _sampler(arr, shots, seed):
    """What a sampling program keeps: the compiled circuit, a frame, the bits a decoder asks for and their place."""
    qmax, bmax = ops.affected_counts(arr)
    bits = np.arange(1, bmax + 1, dtype=np.uint32)
    return {"program": qcb200.Program(arr), "frame": qcb200.PauliFrame(shots, qmax, bmax, init=False), "bits": bits,
            "seed": seed, "out": torch.empty((shots, (bmax + 63) // 64), dtype=torch.int64, device=DEVICE)}


def _syndromes(s):
    qcb200.check(qcb200.lib().qcb_frame_syndrome_rows(s["frame"].handle, s["bits"].ctypes.data, len(s["bits"]),
                                                      s["out"].data_ptr(), 1, None))
    return s["out"]


def _batch_jobs(case, seed):
    # the circuits of the batch are part of the case, their seeds are the inputs
    rng = np.random.default_rng(case["jobs"] * 1_000_003 + case["dmax"])
    for j in range(case["jobs"]):
        d = int(rng.choice(np.arange(3, case["dmax"] + 1, 2)))
        p = float(10 ** rng.uniform(-4, -2))
        shots = int(round(10 ** rng.uniform(3, np.log10(case["smax"]))))
        yield d, p, shots, seed * 1000 + j


def _resident(state):
    """The state on the device, and a copy to work on."""
    base = state.to_gpu()
    return base, base.copy().to_gpu()


def prepare(case, seed):
    qcb200.ensure_init(0)
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "call":
        return {"case": case, "circuit": _circuit(case), "seed": seed}
    if kind == "sample":
        return {"case": case, **_sampler(_circuit(case), case["shots"], seed)}
    if kind == "batch":
        jobs = [_sampler(ops.to_array(circuits.rotated_surface_code_memory(d, d, p)), shots, s)
                for d, p, shots, s in _batch_jobs(case, seed)]
        return {"case": case, "jobs": jobs,
                "batch": qcb200.Batch([(s["frame"], s["program"], s["seed"]) for s in jobs])}
    if kind == "mul":
        n, count = case["n"], case["count"]
        words = 2 * ((n + 63) // 64)
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        bits = [torch.randint(-2**63, 2**63 - 1, (count, words), dtype=torch.int64, device=DEVICE, generator=g) for _ in range(2)]
        if n % 64:  # no qubits past the last one
            for b in bits:
                b[:, words // 2 - 1] &= (1 << (n % 64)) - 1
                b[:, words - 1] &= (1 << (n % 64)) - 1
        ph = [torch.randint(0, 4, (count,), dtype=torch.uint8, device=DEVICE, generator=g) for _ in range(2)]
        return {"case": case, "r": bits[0], "l": bits[1], "rph": ph[0], "lph": ph[1]}
    n = case["n"]
    if kind == "canon":
        base, work = _resident(qcb200.random_stabilizer(n, rng))
        return {"case": case, "base": base, "work": work}
    if kind == "project":
        if case["state"] == "Stabilizer":
            state = qcb200.random_stabilizer(n, rng)
        elif case["state"] == "MixedStabilizer":
            state = qcb200.MixedStabilizer(qcb200.random_stabilizer(n, rng).tab, n)
        elif case["state"] == "Destabilizer":
            state = qcb200.random_destabilizer(n, rng)
        else:  # a state of rank below n, with logical operators
            state = qcb200.MixedDestabilizer(qcb200.random_destabilizer(n, rng).tab, n - n // 4)
        base, work = _resident(state)
        return {"case": case, "base": base, "work": work, "paulis": qcb200.random_paulis(case["k"], n, rng).to_gpu()}
    if kind == "dense":
        if case["op"] == "tCNOT":
            op = qcb200.tensor_pow(qcb200.tCNOT(), n // 2)
        else:
            op = qcb200.random_clifford(n, rng)
        return {"case": case, "work": qcb200.random_stabilizer(n, rng).to_gpu(), "op": op.to_gpu()}
    if kind == "gates":
        circuit = ops.to_array(qcb200.random_clifford_ops(n, case["depth"], rng))
        return {"case": case, "work": qcb200.random_destabilizer(n, rng).to_gpu(), "circuit": circuit}
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        frame = qcb200.pftrajectories(state["circuit"], trajectories=case["shots"], seed=state["seed"])
        return qcb200.measurements(frame)
    if kind == "sample":
        qcb200.check(qcb200.lib().qcb_pftrajectories_fresh(state["frame"].handle, state["program"].handle, state["seed"], 0, None))
        return _syndromes(state)
    if kind == "batch":
        state["batch"].run()
        return [_syndromes(s) for s in state["jobs"]]
    if kind == "mul":
        qcb200.check(qcb200.lib().qcb_mul_left_pauli_batch_noalloc(
            state["r"].data_ptr(), state["rph"].data_ptr(), state["l"].data_ptr(), state["lph"].data_ptr(), case["n"],
            case["count"], int(case["phases"]), None))
        return state["r"], state["rph"]
    work = state["work"]
    if "base" in state:  # the elimination and the projections start from the resident state
        qcb200.check(qcb200.lib().qcb_tableau_copy(work.tab.dev.handle, state["base"].tab.dev.handle, None))
        work.rank = state["base"].rank
    extra = []
    if kind == "canon":
        _, rx, rz = qcb200.canonicalize_(work, phases=case["phases"], ranks=True)
        extra = [rx, rz]
    elif kind == "project":
        _, anticom, result = qcb200.project_(work, state["paulis"])
        extra = [np.array(anticom), np.array([-1 if v is None else v for v in result]), -1 if work.rank is None else work.rank]
    elif kind == "dense":
        for _ in range(case["steps"]):
            qcb200.apply_(work, state["op"])
    else:
        qcb200.apply_(work, state["circuit"])
    work.to_cpu()
    return [work.tab.phases, work.tab.xzs] + extra


def work(case):
    kind = case["kind"]
    if kind == "call":  # the Bool matrix
        return {"bytes": case["shots"] * (case["rounds"] * (case["d"] - 1) + case["d"]), "flops": 0}
    if kind in ("sample", "batch"):  # the record, and its shot-major copy
        total = 0
        jobs = [(case["d"], 0.0, case["shots"], 0)] if kind == "sample" else _batch_jobs(case, 0)
        for d, _, shots, _ in jobs:
            nbits = d * (d * d - 1) + d * d
            total += shots * (2 * nbits / 8 + 8 * ((nbits + 63) // 64))
        return {"bytes": total, "flops": 0}
    n = case["n"]
    row = 16 * ((n + 63) // 64) + 1
    if kind == "mul":  # both read, one written
        return {"bytes": 3 * case["count"] * row, "flops": 0}
    if kind == "canon":  # the tableau in and out
        return {"bytes": 2 * n * row, "flops": 0}
    if kind == "project":
        rows = n if case["state"] in ("Stabilizer", "MixedStabilizer") else 2 * n
        return {"bytes": 2 * rows * row + case["k"] * row, "flops": 0}
    if kind == "dense":  # per step the state in and out and the operator; the product of its bits with the operator's
        return {"bytes": case["steps"] * (2 * n * row + 2 * n * row), "flops": case["steps"] * 2 * n * (2 * n) * (2 * n)}
    return {"bytes": 2 * 2 * n * row, "flops": 0}


def exact(case, seed):
    """Every output is whole numbers, compared for equality: there is nothing to measure a rounding error against."""
    return None
