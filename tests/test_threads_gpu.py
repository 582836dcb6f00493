"""Distinct handles used from distinct host threads (the threading contract of
include/apsm_b200.h; the reference's detector has no such use): handles whose
launches of one kernel want different amounts of shared memory must not refuse
each other's launches, and get the same bits as alone."""
import threading

import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

CFG = {"otype": "APSM", "windowSize": 20, "gaussianKernelVariance": 0.5, "eB": 0.01}


def detector(form, antennas, dictionary, train):
    f = synth.generate_frame(90 + antennas, K=2, N=antennas, P=40, S=48, modulation="QPSK", snr_db=20)
    det = L.NomaDetectorFactory.build(dict(CFG, detectVersion=form, dictionarySize=dictionary), antennas)

    def call():
        if train:
            det.reset_state()
            det.train(f.rx_train, f.tx_train[0])
        return det.detect(f.rx_data)[0]

    det.train(f.rx_train, f.tx_train[0])
    return call


def pool(form, antennas, dictionary, train):
    f = synth.generate_frame(90 + antennas, K=2, N=antennas, P=40, S=48, modulation="QPSK", snr_db=20)
    p = L.DetectorPool(dict(CFG, detectVersion=form, dictionarySize=dictionary))
    d = p.add(antennas)
    fresh = [L.PoolJob(d, f.rx_train, f.tx_train[0], fresh=True)]
    p.run(fresh)

    def call():
        return p.run((fresh if train else []) + [L.PoolJob(d, f.rx_data)])[-1]

    return call


@pytest.mark.parametrize("make,form,train,sizes", [
    (detector, "balanced", False, [(12, 100), (16, 100)]),
    (detector, "balanced", True, [(17, 100), (64, 2000)]),
    (detector, "gram_tf32x3", False, [(4, 100), (64, 100)]),
    (detector, "gram_tf32", False, [(4, 100), (64, 100)]),
    (pool, "balanced", False, [(16, 100), (64, 100)]),
    (pool, "balanced", True, [(4, 100), (4, 2000)]),
    (pool, "gram_bf16x3", False, [(4, 100), (32, 100)]),
], ids=["exact", "train", "gram-tmem", "gram", "pool-fp32", "pool-train", "pool-gram"])
def test_two_threads(make, form, train, sizes):
    calls = [make(form, n, m, train) for n, m in sizes]
    alone = [c().copy() for c in calls]
    failures = []
    start = threading.Barrier(len(calls))

    def work(k):
        try:
            start.wait()
            for i in range(600 if train else 1500):
                if not np.array_equal(calls[k](), alone[k]):
                    failures.append(f"thread {k}, call {i}: other bits")
                    return
        except Exception as e:
            failures.append(f"thread {k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
