"""FP32 pair-form detection of the pool at the edges of its layout: antenna
counts around the copies of 4, 8 and 16, dictionaries around the chunk of 128
pairs, samples around a warp's 8 and a block's 32, requests alone (chunks
spread over blocks) and in a batch (one block per tile).

Bound: the FP32 oracle at 1e-4 of the largest soft output, the bar of the
pool's FP32 form; alone and in the batch the estimates are the same bits."""
import numpy as np
import pytest

from libapsm_b200 import DetectorPool, PoolJob, synth

pytestmark = pytest.mark.gpu

CFG = {"otype": "APSM", "windowSize": 20, "gaussianKernelVariance": 0.5, "eB": 0.01, "dictionarySize": 400}
SIZES = [(1, 1, 1), (2, 127, 7), (3, 128, 8), (4, 129, 31), (5, 260, 32), (8, 128, 33), (9, 385, 40), (16, 127, 64),
         (17, 129, 65), (31, 256, 9), (32, 128, 95), (33, 129, 33), (50, 60, 31), (64, 257, 97)]


def test_layout_edges(oracle_mod):
    pool = DetectorPool(CFG)
    frames = [synth.generate_frame(300 + n, K=2, N=n, P=p, S=s, modulation="QPSK", snr_db=20) for n, p, s in SIZES]
    ids = [pool.add(n) for n, _, _ in SIZES]
    pool.run([PoolJob(i, f.rx_train, f.tx_train[0]) for i, f in zip(ids, frames)])
    jobs = [PoolJob(i, f.rx_data) for i, f in zip(ids, frames)]
    # enough tiles of every antenna class that no dictionary is split
    many = pool.run(jobs + [PoolJob(i, np.tile(f.rx_data, (1, 60000 // f.rx_data.shape[1]))) for i, f in
                            zip(ids, frames)])
    for k, ((n, p, s), f) in enumerate(zip(SIZES, frames)):
        alone = pool.run([jobs[k]])[0]
        o = oracle_mod.OracleDetector(CFG, n, oracle_mod.F32)
        o.train(f.rx_train, f.tx_train[0])
        ref = o.detect(f.rx_data)
        assert np.max(np.abs(alone - ref)) <= 1e-4 * np.max(np.abs(ref)), (n, p, s)
        np.testing.assert_array_equal(alone, many[k])
        np.testing.assert_array_equal(alone, many[len(jobs) + k][-s:])
