"""Fused blocks on relabelled states (CNOT, multi-CNOT and SWAP move no amplitude) against the execution of one
opcode at a time and against the oracle: every shape that tiles the statevector, ranks that cross the tile size
in both directions, expectation values in the middle of a relabelling, forced outcomes on both sides."""

import numpy as np
import pytest

import clifft_b200 as cb
from _programs import random_program
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

SHOTS = 3
# Each of at most ~200 opcodes rounds an amplitude (|a| <= 1) by a few units in the last place: 200 * 4 * 2^-24 =
# 5e-5 as a bound for FP32 against the oracle, which random signs keep far below; probabilities are sums of
# squares with the same relative error. Both ways of execution round alike but for the order of the FP64 norm
# sums (2^16 terms: 1e-11 relative), which scale the state.
TOL_ORACLE = {"fp64": 1e-10, "fp32": 5e-5}
TOL_PLAIN = {"fp64": 1e-10, "fp32": 5e-6}


def state(g, ok):
    v = (g["final_gamma"][:, 0] + 1j * g["final_gamma"][:, 1])[:, None] * g["final_v"]
    return v[ok] / np.linalg.norm(v[ok], axis=1, keepdims=True)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("group,max_k", [(32, 13), (32, 14), (256, 16), (288, 16), (0, 17)])
@pytest.mark.parametrize("seed", range(6))
def test_blocks_match_single_opcodes_and_oracle(precision, group, max_k, seed):
    prog = random_program(100 + seed, n=20, length=190, max_k=max_k, noise=True, classical=True, expand_bias=0.42,
                          active_expvals=seed % 2 == 0)
    o = O.run(prog, SHOTS, seed=seed, rng=O.RNG_PHILOX)
    fm = np.zeros((SHOTS, prog.total_meas_slots), np.uint8)
    fm[:, :prog.num_measurements] = o["meas"]
    kw = dict(forced_meas=fm, faults=[[]] * SHOTS, readout_faults=[[]] * SHOTS)
    ref = O.run(prog, SHOTS, want_state=True, **kw)
    ok = ref["reachable"].astype(bool)
    run = {f: cb.run(prog, SHOTS, 0, precision=precision, trace=True, dump_shots=SHOTS, group_threads=group,
                     fusion=f, **kw) for f in (True, False)}
    for g in run.values():
        assert np.array_equal(g["survived"].astype(bool), ok)
        assert np.array_equal(g["final_k"][ok], ref["final_k"][ok])
        assert np.array_equal(g["final_px"][ok], ref["final_px"][ok])
        assert np.array_equal(g["final_pz"][ok], ref["final_pz"][ok])
    if not ok.any():
        return
    for other, tol in ((ref, TOL_ORACLE[precision]), (run[False], TOL_PLAIN[precision])):
        g = run[True]
        np.testing.assert_allclose(np.nan_to_num(g["meas_prob"][ok]), np.nan_to_num(other["meas_prob"][ok]), atol=tol)
        np.testing.assert_allclose(g["exp_vals"][ok], other["exp_vals"][ok], atol=10 * tol)
        np.testing.assert_allclose(state(g, ok), state(other, ok), atol=tol)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("group", [32, 256, 288, 0])
def test_free_outcomes_are_those_of_single_opcodes(precision, group):
    prog = random_program(131, n=20, length=190, max_k=15, noise=True, classical=True, expand_bias=0.42)
    a = cb.run(prog, 64, 9, precision=precision, group_threads=group, fusion=True)
    b = cb.run(prog, 64, 9, precision=precision, group_threads=group, fusion=False)
    for key in ("meas_words", "det_words", "obs_words", "survived"):
        if a.get(key) is not None:
            assert np.array_equal(a[key], b[key]), key
