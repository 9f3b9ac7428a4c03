"""Condensed frame runs (stars of FRAME_CNOT / FRAME_CZ on a shared axis) against the oracle, which
runs the program gate by gate: one-word and four-word frames, stars of every role and length, repeated
axes, gates whose two axes coincide, and stars inside fused blocks of a tiled statevector."""

import numpy as np
import pytest

import clifft_b200 as cb
from clifft_b200.program import OP, Program, instr
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def star_program(seed, n, k=0):
    rng = np.random.default_rng(seed)
    code, slots = [], 0

    def stars(lo, count):
        for _ in range(count):
            axis = int(rng.integers(lo, n))
            role = int(rng.integers(0, 3))
            for _ in range(int(rng.integers(1, 9))):
                other = int(rng.integers(lo, n))
                if role == 0:
                    code.append(instr(OP["FRAME_CNOT"], axis, other))
                elif role == 1:
                    code.append(instr(OP["FRAME_CNOT"], other, axis))
                else:
                    a, b = (axis, other) if rng.random() < 0.5 else (other, axis)
                    code.append(instr(OP["FRAME_CZ"], a, b))
            kind = ["FRAME_H", "FRAME_S", "FRAME_S_DAG", "FRAME_SWAP"][int(rng.integers(0, 4))]
            code.append(instr(OP[kind], int(rng.integers(lo, n)),
                              int(rng.integers(lo, n)) if kind == "FRAME_SWAP" else 0))

    for q in range(n):  # random X bits, spread over both frame halves
        code.append(instr(OP["MEAS_DORMANT_RANDOM"], q, payload=int(slots).to_bytes(4, "little")))
        slots += 1
        if rng.random() < 0.5:
            code.append(instr(OP["FRAME_H"], q))
    stars(0, 40)
    for a in range(k):
        code.append(instr(OP["EXPAND_T"], a))
        code.append(instr(OP["ARRAY_H"], a))
    if k:
        for _ in range(12):
            a, b = (int(x) for x in rng.choice(k, 2, replace=False))
            code.append(instr(OP["ARRAY_CNOT"], a, b))
            code.append(instr(OP["ARRAY_T"], b))
            stars(k, 2)
    for q in range(k, n):
        code.append(instr(OP["MEAS_DORMANT_STATIC"], q, payload=int(slots).to_bytes(4, "little")))
        slots += 1
    return Program(num_qubits=n, peak_rank=k, num_measurements=slots, total_meas_slots=slots,
                   instructions=np.frombuffer(b"".join(code), np.uint8).reshape(-1, 32).copy())


@pytest.mark.parametrize("n,k,groups", [(2, 0, (0, 1)), (7, 0, (1, 32)), (64, 0, (0, 2, 64)), (65, 0, (0, 4)),
                                        (130, 0, (1, 32)), (256, 0, (0,)), (40, 13, (32, 128, 288)),
                                        (100, 13, (32, 256))])
def test_condensed_frame_runs(n, k, groups):
    prog = star_program(10 * n + k, n, k)
    shots = 70 if k == 0 else 3
    o = O.run(prog, shots, seed=11, rng=O.RNG_PHILOX)
    fm = np.ascontiguousarray(o["meas"], np.uint8)
    ref = O.run(prog, shots, forced_meas=fm)
    for group in groups:
        free = cb.run(prog, shots, 11, precision="fp64", group_threads=group)
        assert np.array_equal(cb.api._unpack(free["meas_words"], prog.num_measurements), o["meas"])
        g = cb.run(prog, shots, 0, precision="fp64", forced_meas=fm, trace=True, group_threads=group)
        assert g["survived"].all()
        assert np.array_equal(g["final_px"], ref["final_px"]) and np.array_equal(g["final_pz"], ref["final_pz"])
        # gamma only changes by exact signs and powers of i here, and by the oracle's own products
        np.testing.assert_allclose(g["final_gamma"], ref["final_gamma"], rtol=0, atol=1e-13)
