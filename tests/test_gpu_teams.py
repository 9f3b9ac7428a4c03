"""Teams of CTAs per shot (few shots of a large statevector) against the oracle: team sizes from one
shot over half the GPU down to one CTA each, ranks that cross the tile size in both directions, expectation
values and renormalisation on the split state, survivors, and FP32 against the one-CTA shape bit by bit."""

import math
import os

import numpy as np
import pytest

import clifft_b200 as cb
from _programs import random_program
from clifft_b200.program import OP, Program, instr, p_f64x2, p_u32x2
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def is_team(r):
    # the automatic shape for a few hundred shots at most and states larger than a tile
    return r["group_threads"] == 288 and not r["state_in_smem"]


@pytest.mark.parametrize("precision,seed,max_k", [("fp64", 3, 17), ("fp64", 7, 18), ("fp32", 5, 18), ("fp32", 7, 19)])
@pytest.mark.parametrize("shots", [1, 5])
def test_teams_match_oracle(precision, seed, max_k, shots):
    prog = random_program(seed, n=22, length=260, max_k=max_k, noise=True, classical=True, expand_bias=0.4)
    assert prog.peak_rank >= 17
    o = O.run(prog, shots, seed=3, rng=O.RNG_PHILOX)
    fm = np.zeros((shots, prog.total_meas_slots), np.uint8)
    fm[:, :prog.num_measurements] = o["meas"]
    ref = O.run(prog, shots, forced_meas=fm, faults=[[]] * shots, readout_faults=[[]] * shots, want_state=True)
    g = cb.run(prog, shots, 0, precision=precision, forced_meas=fm, faults=[[]] * shots,
               readout_faults=[[]] * shots, trace=True, dump_shots=shots)
    assert is_team(g)
    assert np.array_equal(g["survived"].astype(bool), ref["reachable"].astype(bool))
    ok = ref["reachable"].astype(bool)
    assert np.array_equal(g["final_k"][ok], ref["final_k"][ok])
    assert np.array_equal(g["final_px"][ok], ref["final_px"][ok])
    tol = 1e-10 if precision == "fp64" else 1e-5
    np.testing.assert_allclose(np.nan_to_num(g["meas_prob"][ok]), np.nan_to_num(ref["meas_prob"][ok]), atol=tol)
    np.testing.assert_allclose(g["exp_vals"][ok], ref["exp_vals"][ok], atol=1e-10 if precision == "fp64" else 1e-4)
    ga = (g["final_gamma"][:, 0] + 1j * g["final_gamma"][:, 1])[:, None] * g["final_v"]
    ra = (ref["final_gamma"][:, 0] + 1j * ref["final_gamma"][:, 1])[:, None] * ref["final_v"]
    n = np.linalg.norm(ra[ok], axis=1, keepdims=True)
    np.testing.assert_allclose(ga[ok] / n, ra[ok] / n, atol=1e-10 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("name", ["cfg2_01", "cfg2_02", "cfg2_36", "cfg2_55"])
def test_ranks_that_rise_and_fall_through_the_tile_size(precision, name):
    prog = Program.load(os.path.join(os.path.dirname(__file__), "golden", "programs", name + ".npz"))
    shots = 4
    o = O.run(prog, shots, seed=8, rng=O.RNG_PHILOX)
    ref = O.run(prog, shots, forced_meas=o["meas"])
    if precision == "fp64":
        free = cb.run(prog, shots, 8, precision=precision)
        assert np.array_equal(cb.api._unpack(free["meas_words"], prog.num_measurements), o["meas"])
    g = cb.run(prog, shots, 0, precision=precision, forced_meas=o["meas"], trace=True)
    assert g["survived"].all() and is_team(g)
    np.testing.assert_allclose(g["meas_prob"], ref["meas_prob"], atol=1e-10 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shots", [1, 2, 37, 149, 300])
def test_team_sizes_give_the_records_of_one_cta(precision, shots):
    prog = random_program(11, n=21, length=200, max_k=18, noise=True, classical=True, expand_bias=0.4)
    assert prog.peak_rank >= 17
    g = cb.run(prog, shots, 5, precision=precision)
    assert is_team(g)
    one = cb.run(prog, shots, 5, precision=precision, group_threads=288)
    assert np.array_equal(g["meas_words"], one["meas_words"])
    assert np.array_equal(g["det_words"], one["det_words"]) and np.array_equal(g["obs_words"], one["obs_words"])
    np.testing.assert_allclose(g["exp_vals"], one["exp_vals"], atol=1e-12 if precision == "fp64" else 1e-6)
    capped = cb.run(prog, shots, 5, precision=precision, max_resident=2)
    assert np.array_equal(g["meas_words"], capped["meas_words"])


def renormalising_program(k, rounds):
    """Rank k by EXPAND_T, then rounds of an X rotation by 2e-3 on the top axis whose outcome 1 (probability
    1e-6) is forced: gamma grows 1e3-fold each round and leaves the FP32 window (1e20) and the FP64 one
    (1e100), so the split state is rescaled."""
    code, slots = [], 0
    for a in range(k - 1):
        code.append(instr(OP["EXPAND_T"], a))
    for _ in range(rounds):
        code.append(instr(OP["EXPAND"], k - 1))
        code.append(instr(OP["ARRAY_ROT"], k - 1, payload=p_f64x2(math.cos(2e-3), math.sin(2e-3))))
        code.append(instr(OP["ARRAY_H"], k - 1))
        code.append(instr(OP["ARRAY_CNOT"], 0, 1))
        code.append(instr(OP["MEAS_ACTIVE_DIAGONAL"], k - 1, payload=p_u32x2(slots, 0)))
        slots += 1
    return Program(num_qubits=k + 1, peak_rank=k, num_measurements=slots, total_meas_slots=slots,
                   instructions=np.frombuffer(b"".join(code), np.uint8).reshape(-1, 32).copy())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_teams_renormalise_like_one_cta(precision):
    prog = renormalising_program(18, 40)
    shots = 3
    fm = np.zeros((shots, prog.total_meas_slots), np.uint8)
    fm[1] = 1
    ref = O.run(prog, shots, forced_meas=fm, dust_eps=1e-9)
    g = cb.run(prog, shots, 0, precision=precision, forced_meas=fm, trace=True)
    one = cb.run(prog, shots, 0, precision=precision, forced_meas=fm, trace=True, group_threads=288)
    assert is_team(g)
    np.testing.assert_allclose(g["meas_prob"], one["meas_prob"], rtol=1e-12)
    np.testing.assert_allclose(g["final_gamma"], one["final_gamma"], rtol=1e-10)
    np.testing.assert_allclose(g["log_prob"], one["log_prob"], rtol=1e-12)
    assert g["log_prob"][1] < -500
    np.testing.assert_allclose(g["log_prob"], ref["log_prob"], rtol=1e-10 if precision == "fp64" else 1e-4)
