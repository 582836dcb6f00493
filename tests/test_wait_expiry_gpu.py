"""Expiry of a bounded wait in every kernel that has one: an error status, then
the same results as before once the limit is restored (the contract of
apsm_set_wait_limit_ns; the reference exits the process on a CUDA error,
cpp/lib/cuda/cuda_errorhandling.cuh:98-108).

A limit of 0 makes a wait that is not already complete give up at once.  The
operand and column copies that the kernels wait for first take microseconds, so
such a wait expires in every call below."""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import _native, synth

pytestmark = pytest.mark.gpu

CFG = {"otype": "APSM", "windowSize": 20, "gaussianKernelVariance": 0.5, "eB": 0.01, "dictionarySize": 300}


@pytest.fixture
def expire():
    """expire(call): the call's error under a limit of 0."""
    lib = _native.load()
    saved = lib.apsm_wait_limit_ns()

    def run(call):
        lib.apsm_set_wait_limit_ns(0)
        try:
            with pytest.raises(L.ApsmError) as ei:
                call()
        finally:
            lib.apsm_set_wait_limit_ns(saved)
        assert ei.value.status == _native.APSM_ERR_CUDA
        return str(ei.value)

    yield run
    lib.apsm_set_wait_limit_ns(saved)


@pytest.mark.parametrize("form,users", [("gram_bf16", 1), ("gram_bf16x3", 4), ("gram_tf32", 4)])
def test_gram_detection(expire, form, users):
    f = synth.generate_frame(70, K=4, N=16, P=300, S=2048, modulation="QAM16", snr_db=20)
    det = L.NomaDetectorFactory.build(dict(CFG, detectVersion=form), 16, num_users=users)
    det.train(f.rx_train, f.tx_train[:users])
    good, _ = det.detect(f.rx_data)
    assert "bounded wait" in expire(lambda: det.detect(f.rx_data))
    again, _ = det.detect(f.rx_data)
    np.testing.assert_array_equal(again, good)


def test_pool_tensor_core_columns(expire):
    f = synth.generate_frame(71, K=2, N=16, P=200, S=500, modulation="QAM16")
    pool = L.DetectorPool(CFG)
    d = pool.add(16)
    jobs = [L.PoolJob(d, f.rx_train, f.tx_train[0], fresh=True), L.PoolJob(d, f.rx_data)]
    good = pool.run(jobs)[1].copy()
    expire(lambda: pool.run(jobs))
    np.testing.assert_array_equal(pool.run(jobs)[1], good)


@pytest.mark.parametrize("window,pilots,users", [(20, 200, 1), (40, 200, 3), (80, 300, 2), (20, 2800, 2)],
                         ids=["shape32", "shape64", "shape84", "blocks"])
def test_training(expire, window, pilots, users):
    f = synth.generate_frame(72, K=3, N=6, P=pilots, S=100, modulation="QAM16", snr_db=20)
    det = L.NomaDetectorFactory.build(dict(CFG, windowSize=window, dictionarySize=pilots), 6, num_users=users)
    det.train(f.rx_train, f.tx_train[:users])
    good = det.get_state()
    det.reset_state()
    assert "training sweep" in expire(lambda: det.train(f.rx_train, f.tx_train[:users]))
    det.reset_state()
    det.train(f.rx_train, f.tx_train[:users])
    again = det.get_state()
    for k in good:
        np.testing.assert_array_equal(again[k], good[k])


@pytest.mark.parametrize("antennas,fresh", [(4, True), (16, False)])
def test_pool_training(expire, antennas, fresh):
    """FP32 detection beside it: no other kernel of the batch waits."""
    f = synth.generate_frame(73, K=2, N=antennas, P=150, S=200, modulation="QAM16")
    g = synth.generate_frame(74, K=2, N=antennas, P=40, S=8, modulation="QAM16")
    pool = L.DetectorPool(CFG)
    d = pool.add(antennas)
    first = L.PoolJob(d, f.rx_train, f.tx_train[0], fresh=True)
    job = first if fresh else L.PoolJob(d, g.rx_train, g.tx_train[0])
    detect = L.PoolJob(d, f.rx_data)

    def run():
        pool.run([first])
        return pool.run([job, detect])[1].copy()

    good = run()
    pool.run([first])
    expire(lambda: pool.run([job, detect]))
    np.testing.assert_array_equal(run(), good)


def test_pool_training_on_device_buffers_reported_after_later_batches(expire):
    import torch

    f = synth.generate_frame(75, K=2, N=4, P=150, S=200, modulation="QAM16")
    pool = L.DetectorPool(CFG)
    d = pool.add(4)
    rx, tx, data = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (f.rx_train, f.tx_train[0], f.rx_data))
    est = torch.zeros(f.rx_data.shape[1], dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    train, detect = [L.PoolJob(d, rx, tx, fresh=True)], [L.PoolJob(d, data, est=est)]

    def run():
        pool.run_device(train)
        pool.run_device(detect)
        pool.wait()
        return est.cpu().numpy().copy()

    good = run()
    expire(run)
    pool.wait()  # reported once
    np.testing.assert_array_equal(run(), good)
