"""The training sweep with the window matrix in registers, at the sizes where
its layout changes: windows at the edges of each register shape (29, 61 and 81
pairs, one beside them on either side; above 81 the other sweep runs),
dictionaries that just hold the window's fetch distance and evict from then
on, fewer pilots than a copy group, calls in blocks (more than 2729 visible
pairs, with and without eviction), several passes, appending calls and users.

Bound: the FP32 oracle at 1e-5 of the largest soft output, the bound of the
exact sweep's own parity tests (both sum some 2000 terms in FP32; measured
agreement of either is below 1e-6)."""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

BASE = {"otype": "APSM", "gaussianKernelVariance": 0.5, "eB": 0.01}
RTOL = 1e-5


def close(est, ref):
    scale = float(np.max(np.abs(ref)))
    err = float(np.max(np.abs(np.asarray(est) - ref)))
    assert err <= RTOL * scale, f"{err:.3e} > {RTOL:.0e} * {scale:.3e}"


@pytest.mark.parametrize("window", [1, 2, 28, 29, 30, 60, 61, 62, 80, 81, 82])
@pytest.mark.parametrize("pilots,dictionary", [(3, 400), (9, 400), (171, 400), (260, 172)])
def test_windows_and_dictionaries(oracle_mod, window, pilots, dictionary):
    f = synth.generate_frame(40 + window, K=3, N=5, P=pilots, S=64, modulation="QAM16", snr_db=20)
    cfg = dict(BASE, windowSize=window, dictionarySize=dictionary)
    det = L.NomaDetectorFactory.build(cfg, 5, num_users=2)
    det.train(f.rx_train, f.tx_train[:2])
    est, _ = det.detect(f.rx_data)
    for u in range(2):
        o = oracle_mod.OracleDetector(cfg, 5, oracle_mod.F32)
        o.train(f.rx_train, f.tx_train[u])
        close(est[u], o.detect(f.rx_data))


@pytest.mark.parametrize("window,dictionary", [(20, 48), (20, 47), (29, 66), (61, 130), (81, 170)])
def test_smallest_evicting_dictionary_appends(oracle_mod, window, dictionary):
    f = synth.generate_frame(61, K=2, N=33, P=150, S=64, modulation="QPSK", snr_db=20)
    g = synth.generate_frame(62, K=2, N=33, P=201, S=8, modulation="QPSK", snr_db=20)
    cfg = dict(BASE, windowSize=window, dictionarySize=dictionary, trainPasses=2)
    det = L.NomaDetectorFactory.build(cfg, 33)
    o = oracle_mod.OracleDetector(cfg, 33, oracle_mod.F32)
    for x in (f, g):
        det.train(x.rx_train, x.tx_train[0])
        o.train(x.rx_train, x.tx_train[0])
    est, _ = det.detect(f.rx_data)
    close(est, o.detect(f.rx_data))


@pytest.mark.parametrize("pilots,dictionary,append", [(2731, 2731, 0), (3001, 2800, 0), (2600, 2900, 700)])
def test_call_in_blocks(oracle_mod, pilots, dictionary, append):
    f = synth.generate_frame(71, K=3, N=4, P=pilots, S=200, modulation="QAM16", snr_db=20)
    g = synth.generate_frame(72, K=3, N=4, P=max(append, 1), S=8, modulation="QAM16", snr_db=20)
    cfg = dict(BASE, windowSize=20, dictionarySize=dictionary)
    det = L.NomaDetectorFactory.build(cfg, 4, num_users=2)
    det.train(f.rx_train, f.tx_train[:2])
    if append:
        det.train(g.rx_train, g.tx_train[:2])
    est, _ = det.detect(f.rx_data)
    for u in range(2):
        o = oracle_mod.OracleDetector(cfg, 4, oracle_mod.F32)
        o.train(f.rx_train, f.tx_train[u])
        if append:
            o.train(g.rx_train, g.tx_train[u])
        assert det.rows() == o.rows()
        close(est[u], o.detect(f.rx_data))
