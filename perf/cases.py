"""The workloads whose speed this repository cares about, through its public entry points.

Programs are the compiled benchmark programs of tests/golden/programs (near-Clifford circuits
after the reference's bytecode passes, peak rank 4 to 24), and circuits of clifft_b200.workloads
lowered here: noisy memory grids, random near-Clifford circuits and rotation circuits with
Pauli probes. A case names its program, the call that a user makes on it, the number of shots
(records, phase vectors) and the precision of the statevector.
"""

from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

import clifft_b200 as cb
from clifft_b200 import grad, workloads
from clifft_b200.program import ACTIVE_MEAS, EXPANDS, OP, OPCODES, Program

PROGRAMS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(cb.__file__))), "tests", "golden", "programs")


def listed():
    return [
        # Trying a program out, a few shots at a time: launches, copies and latency are everything.
        {"name": "few_shots_k7", "call": "sample", "program": "cfg0", "shots": 16, "precision": "fp64"},
        # Logical error rate of a post-selected noisy memory experiment: counters only, most shots die early.
        {"name": "memory_survivors", "call": "survivors", "program": "cfg1", "shots": 1_000_000, "precision": "fp32"},
        # Training or evaluation data for a decoder: every measurement and detector bit of every shot.
        {"name": "memory_records", "call": "sample", "program": "grid", "rows": 7, "cols": 7, "rounds": 10, "t": 12,
         "p": 1e-3, "circuit_seed": 7, "shots": 100_003, "precision": "fp32"},
        # Small circuits in the reference's own precision.
        {"name": "circuit_k7_fp64", "call": "sample", "program": "cfg0", "shots": 50_000, "precision": "fp64"},
        # The everyday sizes of the multi-program set (10^4 shots each): states in shared memory, in L2, in HBM.
        {"name": "circuit_k10", "call": "sample", "program": "cfg2_12", "shots": 10_000, "precision": "fp32"},
        {"name": "circuit_k16", "call": "sample", "program": "cfg2_36", "shots": 10_000, "precision": "fp32"},
        {"name": "circuit_k18_fp64", "call": "sample", "program": "cfg2_01", "shots": 1_000, "precision": "fp64"},
        # Circuits full of fused one- and two-axis unitaries (U2 / U4), a ragged number of shots.
        {"name": "dense_k20", "call": "sample", "program": "dense_k20", "shots": 150, "precision": "fp32"},
        # One trajectory of a large program (the reference quotes compile + one shot), and a full set of them.
        {"name": "one_shot_k24", "call": "sample", "program": "cfg3", "shots": 1, "precision": "fp32"},
        {"name": "shots_k24", "call": "sample", "program": "cfg3", "shots": 148, "precision": "fp32"},
        # Log-probabilities of given records (forced replay).
        {"name": "record_probabilities", "call": "replay", "program": "circuit", "n": 16, "layers": 100, "t": 8,
         "circuit_seed": 42, "shots": 2_000, "precision": "fp64"},
        # One optimiser step of a variational circuit: 16 observables, gradients of 32 angles, forward and backward.
        {"name": "gradients_k13", "call": "gradient", "program": "rotations", "n": 40, "layers": 120, "t": 32,
         "observables": 16, "rot_layers": 10, "circuit_seed": 3, "shots": 256, "precision": "fp64"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))

    kind = rng.choice(["grid", "grid", "set", "set", "set", "circuit", "large", "replay", "gradient"])
    precision = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "grid":
        call = rng.choice(["survivors", "sample", "k_faults"])
        while True:
            c = {"call": call, "program": "grid", "rows": rng.randint(3, 7), "cols": rng.randint(3, 7),
                 "rounds": rng.randint(2, 10), "t": rng.randint(1, 12), "p": round(math.exp(rng.uniform(-8.1, -5.5)), 7),
                 "circuit_seed": rng.randrange(1 << 20)}
            if _program(c).peak_rank <= 7:
                break
        c["shots"] = log_int(10_000, 1_000_000) if call == "survivors" else log_int(256, 100_000)
        if call == "k_faults":
            c["k"] = rng.randint(1, 5)
    elif kind == "set":
        c = {"call": "sample", "program": "cfg2_%02d" % rng.randrange(64)}
        c["shots"] = log_int(1, min(20_000, (3 << 27) >> _program(c).peak_rank))
    elif kind == "circuit":
        while True:
            c = {"call": "sample", "program": "circuit", "n": rng.randint(5, 70), "layers": rng.randint(20, 120),
                 "t": rng.randint(2, 20), "circuit_seed": rng.randrange(1 << 20)}
            if _program(c).peak_rank <= 19:
                break
        c["shots"] = log_int(1, min(20_000, (3 << 27) >> _program(c).peak_rank))
    elif kind == "large":
        c = {"call": "sample", "program": rng.choice(["cfg3", "dense_k20"])}
        c["shots"] = log_int(1, 70)
    elif kind == "replay":
        c = {"call": "replay", "program": "circuit", "n": rng.randint(6, 16), "layers": rng.randint(20, 120),
             "t": rng.randint(2, 12), "circuit_seed": rng.randrange(1 << 20), "shots": log_int(16, 2_000)}
        precision = "fp64"
    else:
        while True:
            c = {"call": "gradient", "program": "rotations", "n": rng.randint(10, 40), "layers": rng.randint(20, 120),
                 "t": rng.randint(5, 32), "observables": rng.randint(1, 16), "rot_layers": rng.randint(4, 12),
                 "circuit_seed": rng.randrange(1 << 20)}
            if 3 <= _program(c).peak_rank <= 13:
                break
        c["shots"] = log_int(1, 256)
        precision = "fp64"
    c["precision"] = precision
    return c


# ------------------------------------------------------------------ programs
def _circuit(case):
    return workloads.random_near_clifford(case["n"], case["layers"], case["t"], case["circuit_seed"])


@functools.lru_cache(maxsize=64)
def _arrays(key):
    """The compiled program of a case as a dict of arrays; compiled once per process."""
    case = dict(key)
    name = case["program"]
    if name == "grid":
        circ = workloads.memory_grid(case["rows"], case["cols"], case["rounds"], case["t"], case["p"],
                                     case["circuit_seed"])
        p = workloads.lower(circ, case["call"] == "survivors")
    elif name == "circuit":
        p = workloads.lower(_circuit(case))
    elif name == "rotations":
        circ, _ = workloads.config4(case["circuit_seed"], case["n"], case["layers"], case["t"], case["observables"],
                                    case["rot_layers"])
        p = workloads.active_probes(workloads.lower(circ), case["circuit_seed"])
    else:
        p = Program.load(os.path.join(PROGRAMS, name + ".npz"))
    return p.to_npz_dict()


def _program(case):
    keys = ("call", "program", "rows", "cols", "rounds", "t", "p", "circuit_seed", "n", "layers", "observables",
            "rot_layers")
    return Program.from_npz_dict(_arrays(tuple((k, case[k]) for k in keys if k in case)))


# ------------------------------------------------------------------- the case
def _records(case, program, seed):
    """Records that the program emits, the ones a user would ask probabilities for."""
    return cb.sample(program, case["shots"], seed, precision="fp64").measurements


def _phases(case, program, seed):
    g = torch.Generator().manual_seed(seed)
    n = grad.rot_phases(program).size
    return (torch.rand((case["shots"], n), dtype=torch.float64, generator=g) * 2 * math.pi,
            torch.randn((case["shots"], program.num_exp_vals), dtype=torch.float64, generator=g))


def prepare(case, seed):
    program = _program(case)
    cb.load(program)
    state = {"call": case["call"], "program": program, "shots": case["shots"], "seed": seed,
             "precision": case["precision"], "k": case.get("k", 0)}
    if case["call"] == "replay":
        state["records"] = _records(case, program, seed)
    elif case["call"] == "gradient":
        phases, weights = _phases(case, program, seed)
        state["phases"], state["weights"] = phases.cuda().requires_grad_(), weights.cuda()
    return state


def run(state):
    call, program, precision = state["call"], state["program"], state["precision"]
    if call == "sample":
        r = cb.sample(program, state["shots"], state["seed"], precision=precision)
        return {"measurements": r.measurements, "detectors": r.detectors, "observables": r.observables}
    if call == "survivors":
        r = cb.sample_survivors(program, state["shots"], state["seed"], precision=precision)
        return {"passed": r.passed_shots, "logical_errors": r.logical_errors, "ones": r.observable_ones}
    if call == "k_faults":
        r = cb.sample_k(program, state["shots"], state["k"], state["seed"], precision=precision)
        return {"measurements": r.measurements, "detectors": r.detectors, "observables": r.observables}
    if call == "replay":
        return {"log_prob": cb.record_probabilities(program, state["records"], precision=precision)}
    phases = state["phases"]
    phases.grad = None
    values = grad.ExpVal.apply(phases, program, precision)
    (values * state["weights"]).sum().backward()
    return {"exp_vals": values.detach(), "grad": phases.grad}


def work(case):
    """Bytes: the program and the inputs read once, the outputs written once. Flops: the arithmetic on the 2^k
    active amplitudes of every shot, opcode by opcode (permutations are free)."""
    program = _program(case)
    shots = case["shots"]
    flops = 0.0
    for op, k in zip(program.opcodes.tolist(), program.active_k_history().tolist()):
        name, amps = OPCODES[op], float(1 << k)
        if op in EXPANDS:
            flops += 0.0 if name == "EXPAND" else 6 * amps
        elif op in ACTIVE_MEAS:
            flops += 4 * amps if "DIAGONAL" in name else 12 * amps
        elif name.startswith("ARRAY_"):
            flops += {"CZ": 0.5, "MULTI_CZ": 1, "H": 4, "S": 1, "S_DAG": 1, "T": 3, "T_DAG": 3, "ROT": 3, "U2": 14,
                      "U4": 30}.get(name[6:], 0) * amps
        elif name == "EXP_VAL":
            flops += 12 * amps
    image = float(sum(np.asarray(v).nbytes for v in program.to_npz_dict().values() if np.asarray(v).dtype.kind != "U"))
    per_shot = {"survivors": 0, "replay": program.num_measurements + 8}.get(
        case["call"], program.num_measurements + program.num_detectors + program.num_observables)
    if case["call"] == "gradient":
        p, e = grad.rot_phases(program).size, program.num_exp_vals
        flops *= 2 + e  # forward once, the state undone once, one adjoint vector per observable
        per_shot = 8 * (2 * p + 2 * e)
    return {"bytes": image + float(shots) * per_shot, "flops": shots * flops}


# ---------------------------------------------------------------- exact values
def exact(case, seed):
    if case["call"] in ("sample", "survivors", "k_faults"):
        return None  # bits and counts
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    program = _program(case)
    if case["call"] == "replay":
        records = torch.from_numpy(_records(case, program, seed).astype(np.int64)).to(dev)
        return {"log_prob": _circuit_log_prob(_circuit(case), records).cpu()}
    phases, weights = (t.to(dev) for t in _phases(case, program, seed))
    phases.requires_grad_()
    values = _exp_vals(program, phases)
    (values * weights).sum().backward()
    return {"exp_vals": values.detach(), "grad": phases.grad}


def _circuit_log_prob(circuit, records):
    """log P(record) of every row by projecting the 2^n physical statevector onto each outcome in turn."""
    rows, n = records.shape[0], circuit.num_qubits
    v = torch.zeros((rows, 1 << n), dtype=torch.complex128, device=records.device)
    v[:, 0] = 1.0
    log_prob = torch.zeros(rows, dtype=torch.float64, device=records.device)
    at = 0
    for g in circuit.gates:
        q = g.qubits[0]
        w = v.view(rows, -1, 2, 1 << q)
        if g.kind == "H":
            a, b = w[:, :, 0].clone(), w[:, :, 1].clone()
            w[:, :, 0], w[:, :, 1] = (a + b) * math.sqrt(0.5), (a - b) * math.sqrt(0.5)
        elif g.kind in ("S", "S_DAG", "T", "T_DAG"):
            angle = math.pi / (2 if g.kind[0] == "S" else 4) * (-1 if g.kind.endswith("DAG") else 1)
            w[:, :, 1] *= complex(math.cos(angle), math.sin(angle))
        elif g.kind == "CX":
            i = torch.arange(1 << n, device=v.device)
            v = v[:, i ^ (((i >> q) & 1) << g.qubits[1])]
        elif g.kind == "M":
            other = (records[:, at] ^ 1).view(-1, 1, 1)
            gone = torch.arange(2, device=v.device).view(1, 2, 1) == other  # rows, bit, 1
            w.masked_fill_(gone.unsqueeze(1), 0.0)
            prob = torch.view_as_real(v).square().sum(dim=(1, 2))
            log_prob += torch.log(prob)
            v /= prob.sqrt().unsqueeze(1)
            at += 1
        else:
            raise ValueError(g.kind)
    return log_prob


def _exp_vals(program, phases):
    """<P_e> for every row of phases, differentiable: the array opcodes of a measurement- and noise-free program on
    its 2^k active amplitudes (the Pauli frame of such a program stays the identity)."""
    rows, dev = phases.shape[0], phases.device
    v = torch.ones((rows, 1), dtype=torch.complex128, device=dev)
    k, param, values = 0, 0, [None] * program.num_exp_vals
    a1, a2 = program.axis_1.tolist(), program.axis_2.tolist()
    words = program.instructions[:, 8:16].copy().view(np.uint64).reshape(-1).tolist()
    half = torch.tensor(math.pi / 4, dtype=torch.float64, device=dev).expand(rows, 1)

    def parity(x):
        for s in (32, 16, 8, 4, 2, 1):
            x = x ^ (x >> s)
        return x & 1

    def angle_of(name):
        nonlocal param
        if name.endswith("ROT"):
            param += 1
            return phases[:, param - 1:param]
        return half * {"T": 1, "T_DAG": -1, "S": 2, "S_DAG": -2}[name.split("_", 1)[1]]

    for pc, op in enumerate(program.opcodes.tolist()):
        name, a, b = OPCODES[op], a1[pc], a2[pc]
        i = torch.arange(1 << k, device=dev)
        if name.startswith("FRAME_"):
            continue
        if name.startswith("EXPAND"):
            angle = torch.zeros_like(half) if name == "EXPAND" else angle_of(name)
            v = torch.cat([v, v * torch.exp(1j * angle)], dim=1) * math.sqrt(0.5)
            k += 1
        elif name in ("ARRAY_T", "ARRAY_T_DAG", "ARRAY_S", "ARRAY_S_DAG", "ARRAY_ROT"):
            angle = angle_of(name)
            if a < k:
                v = v * torch.exp(1j * angle * ((i >> a) & 1))
        elif name == "ARRAY_H":
            w = v.view(rows, -1, 2, 1 << a)
            v = torch.stack([w[:, :, 0] + w[:, :, 1], w[:, :, 0] - w[:, :, 1]], dim=2).view(rows, -1) * math.sqrt(0.5)
        elif name == "ARRAY_CNOT":
            v = v[:, i ^ (((i >> a) & 1) << b)]
        elif name == "ARRAY_MULTI_CNOT":
            v = v[:, i ^ (parity(i & words[pc]) << a)]
        elif name == "ARRAY_SWAP":
            d = ((i >> a) ^ (i >> b)) & 1
            v = v[:, i ^ (d << a) ^ (d << b)]
        elif name in ("ARRAY_CZ", "ARRAY_MULTI_CZ"):
            v = v * (1.0 - 2.0 * (((i >> a) & 1) * parity(i & (1 << b if name == "ARRAY_CZ" else words[pc]))))
        elif name == "EXP_VAL":
            mask, row = words[pc] & 0xFFFFFFFF, words[pc] >> 32
            xs, zs = ([int(x) for x in m[mask]] for m in (program.exp_val_x, program.exp_val_z))
            if xs[0] >> k or any(xs[1:]):
                values[row] = torch.zeros(rows, dtype=torch.float64, device=dev)
                continue
            x, z = xs[0], zs[0] & ((1 << k) - 1)
            sign = (1.0 - 2.0 * parity(i & z)) * (1j ** (bin(x & z).count("1") & 3))
            if program.exp_val_sign[mask]:
                sign = -sign
            values[row] = (v[:, i ^ x].conj() * v * sign).real.sum(dim=1)
        else:
            raise ValueError(name)
    return torch.stack(values, dim=1)
