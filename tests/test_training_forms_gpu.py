"""Training calls beside the ones of test_window_sweep_gpu.py where another
form, or another part of a form, does the work:

* dictionaries whose coefficients do not fit the cluster sweep's shared memory,
  with settings that the window sweep does not take (a sample step other than
  2, windows above 81 pairs, a bound on the norm): the shape search itself
  falls back to coefficient rings in global memory;
* calls in blocks with more users than one tile of the old-pair sums holds (8)
  and more antennas than a warp has lanes;
* the pool's inputs at the edges of the window sweep's register shapes (29, 61
  and 81 pairs), appending to dictionaries that just hold the window's fetch
  distance, so that every appended pilot evicts one.

Bound: the FP32 oracle at 1e-5 of the largest soft output for a single
detector, 1e-4 for the pool (the bounds of their own parity tests)."""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

BASE = {"otype": "APSM", "windowSize": 80, "gaussianKernelVariance": 0.5, "eB": 0.01}


def close(est, ref, rtol):
    scale = float(np.max(np.abs(ref)))
    err = float(np.max(np.abs(np.asarray(est) - ref)))
    assert err <= rtol * scale, f"{err:.3e} > {rtol:.0e} * {scale:.3e}"


def train_and_compare(oracle_mod, cfg, frames, users, checked):
    n = frames[0].rx_train.shape[0]
    det = L.NomaDetectorFactory.build(cfg, n, num_users=users)
    for f in frames:
        det.train(f.rx_train, f.tx_train[:users])
    est, _ = det.detect(frames[0].rx_data)
    for u in checked:
        o = oracle_mod.OracleDetector(cfg, n, oracle_mod.F32)
        for f in frames:
            o.train(f.rx_train, f.tx_train[u])
        close(est[u], o.detect(frames[0].rx_data), 1e-5)


@pytest.mark.parametrize("settings", [{"sampleStep": 4}, {"windowSize": 82}, {"normConstraint": 0.005}],
                         ids=["step4", "window82", "norm"])
def test_large_dictionary_outside_the_window_sweep(oracle_mod, settings):
    f = synth.generate_frame(31, K=4, N=64, P=240, S=200, modulation="QAM16", snr_db=15)
    train_and_compare(oracle_mod, dict(BASE, dictionarySize=8192, **settings), [f], 4, (0, 3))


def test_blocks_with_many_users_and_antennas(oracle_mod):
    f = synth.generate_frame(81, K=17, N=33, P=2750, S=100, modulation="QPSK", snr_db=20)
    g = synth.generate_frame(82, K=17, N=33, P=300, S=8, modulation="QPSK", snr_db=20)
    train_and_compare(oracle_mod, dict(BASE, windowSize=20, dictionarySize=2800), [f, g], 17, (0, 8, 16))


@pytest.mark.parametrize("window", [29, 30, 61, 62, 81, 82])
def test_pool_windows_append_and_evict(oracle_mod, window):
    cfg = dict(BASE, windowSize=window, dictionarySize=2 * window + 8)
    sizes = [(3, 2 * window + 8), (8, 2 * window + 40), (33, 2 * window + 9)]  # antennas, first pilots
    frames = [[synth.generate_frame(1000 * k + n, K=2, N=n, P=p, S=60, modulation="QPSK", snr_db=20)
               for k, p in enumerate((first, window + 3, 5))] for n, first in sizes]
    pool = L.DetectorPool(cfg)
    ids = [pool.add(n) for n, _ in sizes]
    for k in range(3):
        pool.run([L.PoolJob(d, fs[k].rx_train, fs[k].tx_train[0]) for d, fs in zip(ids, frames)])
    ests = pool.run([L.PoolJob(d, fs[0].rx_data) for d, fs in zip(ids, frames)])
    for est, (n, _), fs in zip(ests, sizes, frames):
        o = oracle_mod.OracleDetector(cfg, n, oracle_mod.F32)
        for f in fs:
            o.train(f.rx_train, f.tx_train[0])
        close(est, o.detect(fs[0].rx_data), 1e-4)
