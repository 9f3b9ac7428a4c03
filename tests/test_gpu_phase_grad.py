"""Gradients of programs without ARRAY_H (one transform per observable) against the general reverse walk,
which the same program takes when a pair ARRAY_H, ARRAY_H (the identity) is appended to its state: ranks
below, at and above one value per thread, permutations, CZ stars, EXP_VALs at several points, parameters that
do not reach an observable, masks with X on dormant axes, and rank 14, where both take the general kernel."""

import math

import numpy as np
import pytest

import clifft_b200 as cb
from clifft_b200 import grad as GR
from clifft_b200.program import OP, Program, instr, p_f64x2, p_u32x2, p_u64

pytestmark = pytest.mark.gpu


def program(seed, n, top, pair, dense):
    """dense: many entangling opcodes and Z masks (most observables then read 0); else few of both."""
    rng = np.random.default_rng(seed)
    code, ex, ez, es, k = [], [], [], [], 0
    W = (n + 63) // 64

    def axes(count):
        return [int(a) for a in rng.choice(k, count, replace=False)]

    def rot():
        phi = rng.uniform(0, 2 * math.pi)
        return p_f64x2(math.cos(phi), math.sin(phi))

    def observe():
        x = sum(1 << a for a in axes(min(k, int(rng.integers(1, 3)))))
        if rng.random() < 0.15 and n > k:
            x |= 1 << (n - 1)
        z = sum(1 << a for a in range(n) if rng.random() < 0.3) if dense else x & int(rng.integers(0, 1 << k))
        for words, v in ((ex, x), (ez, z)):
            words.append([(v >> (64 * w)) & 0xFFFFFFFFFFFFFFFF for w in range(W)])
        es.append(int(rng.integers(0, 2)))
        code.append(instr(OP["EXP_VAL"], payload=p_u32x2(len(es) - 1, len(es) - 1)))

    while True:
        if k < top and (k == 0 or rng.random() < 0.4):
            kind = ["EXPAND", "EXPAND_T", "EXPAND_T_DAG", "EXPAND_ROT"][int(rng.integers(0, 4))]
            code.append(instr(OP[kind], k, payload=rot() if kind == "EXPAND_ROT" else b""))
            k += 1
            continue
        if k == top and rng.random() < 0.03:
            break
        c = int(rng.integers(0, 9))
        if not dense and c in (4, 5) and rng.random() < 0.8:
            c = 1
        a = axes(1)[0]
        if c <= 2:
            code.append(instr(OP["ARRAY_ROT"], a if c else n - 1, payload=rot()))
        elif c == 3:
            code.append(instr(OP[["ARRAY_T", "ARRAY_T_DAG", "ARRAY_S", "ARRAY_S_DAG"][int(rng.integers(0, 4))]], a))
        elif c == 4 and k >= 2:
            code.append(instr(OP[["ARRAY_CNOT", "ARRAY_CZ", "ARRAY_SWAP"][int(rng.integers(0, 3))]], *axes(2)))
        elif c == 5 and k >= 2:
            mask = sum(1 << b for b in range(k) if b != a and rng.random() < 0.5)
            code.append(instr(OP[["ARRAY_MULTI_CNOT", "ARRAY_MULTI_CZ"][int(rng.integers(0, 2))]], a,
                              payload=p_u64(mask)))
        elif c == 6:
            code.append(instr(OP["FRAME_S"], int(rng.integers(0, n))))
        elif c == 7 and rng.random() < 0.3:
            if pair:
                code.extend([instr(OP["ARRAY_H"], a)] * 2)
            observe()
            observe()
    if pair:
        code.extend([instr(OP["ARRAY_H"], 0)] * 2)
    for _ in range(3):
        observe()
    code.append(instr(OP["ARRAY_ROT"], 0, payload=rot()))  # after every observable
    return Program(num_qubits=n, peak_rank=top, num_measurements=0, total_meas_slots=0, num_exp_vals=len(es),
                   instructions=np.frombuffer(b"".join(code), np.uint8).reshape(-1, 32).copy(),
                   exp_val_x=np.array(ex, np.uint64).reshape(-1, W), exp_val_z=np.array(ez, np.uint64).reshape(-1, W),
                   exp_val_sign=np.array(es, np.uint8))


@pytest.mark.parametrize("n,top,batch", [(3, 1, 1), (4, 2, 300), (8, 5, 7), (9, 6, 2), (10, 8, 3), (12, 9, 5),
                                          (70, 10, 150), (15, 12, 2), (20, 13, 5), (20, 13, 160), (20, 14, 2)])
@pytest.mark.parametrize("dense", [True, False])
def test_phase_polynomial_gradients_match_the_general_kernel(n, top, batch, dense):
    one, general = (program(100 * top + n, n, top, pair, dense) for pair in (False, True))
    assert OP["ARRAY_H"] not in one.opcodes and OP["ARRAY_H"] in general.opcodes
    assert GR.num_rot_params(one) == GR.num_rot_params(general)
    phases = np.random.default_rng(top).uniform(0, 2 * math.pi, (batch, GR.num_rot_params(one)))
    # both kernels round ~100 FP64 products per amplitude and sum 2^k terms of weight 2^-k: errors near 1e-15
    for ph in (phases, None):
        ev, g = GR.expval_grad(one, ph)
        ev2, g2 = GR.expval_grad(general, ph)
        np.testing.assert_allclose(ev, ev2, rtol=0, atol=1e-13)
        np.testing.assert_allclose(g, g2, rtol=0, atol=1e-12)
    assert np.all(g[:, :, -1] == 0.0)
    assert dense or np.abs(g).max() > 1e-3
    np.testing.assert_allclose(ev[0], cb.run(one, 1, 0, precision="fp64")["exp_vals"][0], atol=1e-13)
