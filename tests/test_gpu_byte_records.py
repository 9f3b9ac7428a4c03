"""CLIFFT_GPU_BYTE_RECORDS and the staged result copies: byte records equal the unpacked words at record
counts around the byte and word edges, for results that one thread delivers, that several do, and that exceed
the staging buffer; callers in several threads; outputs asked for by name."""

import threading

import numpy as np
import pytest

import clifft_b200 as cb
from clifft_b200 import _native as N
from clifft_b200.program import OP, Program, instr, p_u32x2

pytestmark = pytest.mark.gpu


def coin_program(meas, det):
    code = [instr(OP["MEAS_DORMANT_RANDOM"], i % 60, payload=p_u32x2(i, 0)) for i in range(meas)]
    code += [instr(OP["DETECTOR"], payload=p_u32x2(d, d)) for d in range(det)]
    return Program(num_qubits=60, peak_rank=0, num_measurements=meas, total_meas_slots=meas, num_detectors=det,
                   detector_offsets=np.arange(det + 1, dtype=np.uint32),
                   detector_targets=np.arange(det, dtype=np.uint32) % max(meas, 1),
                   instructions=np.frombuffer(b"".join(code), np.uint8).reshape(-1, 32).copy())


@pytest.mark.parametrize("meas,det", [(1, 0), (7, 1), (8, 9), (9, 8), (63, 65), (64, 64), (65, 63), (130, 3)])
@pytest.mark.parametrize("shots", [1, 1023, 30_011])
def test_byte_records_equal_unpacked_words(meas, det, shots):
    prog = coin_program(meas, det)
    words = cb.run(prog, shots, 5, autotune=False)
    r = cb.sample(prog, shots, 5)
    assert np.array_equal(r.measurements, cb.api._unpack(words["meas_words"], meas))
    assert np.array_equal(r.detectors, cb.api._unpack(words["det_words"], det))
    assert r.observables.shape == (shots, 0) and r.measurements.flags.c_contiguous


def test_results_larger_than_the_staging_buffer():
    prog = coin_program(250, 0)
    shots = 2_200_000  # 70 MB of packed words
    r = cb.sample(prog, shots, 2)
    words = cb.run(prog, shots, 2, outputs=("meas_words",))
    assert set(words).isdisjoint({"survived", "exp_vals", "det_words"})
    for part in (slice(0, 1000), slice(shots // 2, shots // 2 + 1000), slice(shots - 1000, shots)):
        assert np.array_equal(r.measurements[part], cb.api._unpack(words["meas_words"][part], 250))


def test_concurrent_callers_get_their_own_records():
    progs = [coin_program(20 + i, 0) for i in range(4)]
    alone = [cb.sample(p, 50_000, i).measurements for i, p in enumerate(progs)]
    got = [None] * 4

    def work(i):
        for _ in range(5):
            got[i] = cb.sample(progs[i], 50_000, i).measurements

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got):
        assert np.array_equal(a, b)
    cb.trim()  # the staging buffer goes back and comes again
    assert np.array_equal(cb.sample(progs[0], 50_000, 0).measurements, alone[0])


def test_byte_records_need_host_buffers():
    prog = coin_program(3, 0)
    import ctypes
    a = N.SampleArgs(shots=1, flags=N.CLIFFT_GPU_BYTE_RECORDS | N.CLIFFT_GPU_DEVICE_PTRS)
    o = N.Outputs()
    assert N.lib().clifft_gpu_sample(cb.load(prog).handle, ctypes.byref(a), ctypes.byref(o)) == -1
