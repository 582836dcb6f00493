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
