"""Record lists and Pauli masks that travel in their instruction, against the oracle: list lengths on both sides of
what fits (3), empty lists and lists with repeated records, frames of one and of two words, every group width."""

import numpy as np
import pytest

import clifft_b200 as cb
from _programs import random_program
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def relist(prog, rng):
    for kind in ("detector", "observable"):
        count = len(getattr(prog, kind + "_offsets")) - 1
        if count < 1:
            continue
        lens = rng.permutation(np.arange(count) % 6)
        setattr(prog, kind + "_offsets", np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32))
        setattr(prog, kind + "_targets", rng.integers(0, prog.num_measurements, int(lens.sum())).astype(np.uint32))


@pytest.mark.parametrize("n", [9, 64, 70])
@pytest.mark.parametrize("group", [1, 4, 32, 256])
@pytest.mark.parametrize("seed", range(3))
def test_lists_and_masks_match_oracle(n, group, seed):
    prog = random_program(300 + seed, n=n, length=700, max_k=5, noise=True, classical=True)
    relist(prog, np.random.default_rng(seed))
    lens = np.concatenate([np.diff(prog.detector_offsets), np.diff(prog.observable_offsets)])
    assert (lens >= 3).any()
    shots = 50
    o = O.run(prog, shots, seed=seed, rng=O.RNG_PHILOX)
    g = cb.run(prog, shots, seed, precision="fp64", group_threads=group)
    for name, bits in (("meas", prog.num_measurements), ("det", prog.num_detectors), ("obs", prog.num_observables)):
        assert np.array_equal(cb.api._unpack(g[name + "_words"], bits), o[name]), name
