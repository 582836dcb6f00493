"""Exact FP32 detection at the edges of its layout: feature counts around the
chunks of 8, 16, 32 and 64, dictionaries around the 128-row tile, samples
around a warp's eight and both block sizes, user counts on either side of a
pass.

Bound: the rounding of the evaluation order, from the model's own state in
64 bits.  With u = 2^-24 and t_b = |ew| ||d_b - x||^2, the differences (2), the
chain over D features, ew and the scaling put a relative (D + 4) u t_b into a
Gaussian value, expf's 2 ulp 4 u, the products with the coefficient 2 u, the
lane's chain of at most M / 32 + 1 rows and the tree of 32 lanes as many u and
5 u; the linear part has at most D / 32 + 1 terms of two products a lane, then
the same sums.  (First order in u, hence the factor 1.01.)"""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
CASES = [
    # antennas, users, pilots (two rows each), symbols (two samples each)
    (1, 1, 1, 1),
    (4, 1, 63, 3),
    (4, 5, 64, 4),
    (5, 2, 65, 5),
    (8, 1, 129, 2368),
    (8, 9, 30, 2369),
    (9, 4, 64, 15),
    (16, 8, 127, 2400),
    (17, 1, 70, 17),
    (17, 16, 130, 2500),
    (32, 3, 64, 31),
    (33, 17, 66, 33),
    (50, 6, 40, 2371),
    (64, 1, 128, 16),
    (64, 33, 65, 2369),
]


@pytest.mark.parametrize("antennas,users,pilots,symbols", CASES)
def test_layout_edges(antennas, users, pilots, symbols):
    K = min(users, 4)
    f = synth.generate_frame(antennas + users, K=K, N=antennas, P=pilots, S=symbols, modulation="QAM16", snr_db=20)
    tx = np.stack([f.tx_train[u % K] * (1.0 + 0.1 * (u // K)) for u in range(users)])
    cfg = {"otype": "APSM", "gaussianKernelVariance": 0.5, "eB": 0.01, "windowSize": 20}
    det = L.NomaDetectorFactory.build(cfg, antennas, num_users=users)
    det.train(f.rx_train, tx)
    est = np.atleast_2d(det.detect(f.rx_data)[0])
    st = {k: v.astype(np.float64) for k, v in det.get_state().items()}
    rx = np.asarray(f.rx_data, dtype=np.complex64).astype(np.complex128).T
    x = np.stack([np.concatenate([rx.real, rx.imag], 1), np.concatenate([rx.imag, -rx.real], 1)], 1)
    x = x.reshape(-1, 2 * antennas)
    wG = float(np.float32(0.5))
    wL = 1.0 - wG
    t = 0.5 / (0.5 * antennas**2) * np.stack([((st["dictionary"] - r) ** 2).sum(1) for r in x])  # (samples, rows)
    D, M = 2 * antennas, t.shape[1]
    ref = wL * st["w"] @ x.T + wG * st["a"] @ np.exp(-t).T
    tol = np.abs(st["w"]) @ np.abs(x).T * wL * (D / 32 + 1 + M / 32 + 1 + 5 + 2)
    tol += wG * np.abs(st["a"]) @ (np.exp(-t) * ((D + 4) * t + 4 + 2 + M / 32 + 1 + 5)).T
    got = np.stack([est.real, est.imag], -1).reshape(users, -1)
    err = np.abs(got - ref)
    assert (err <= 1.01 * U * tol + 1e-37).all(), f"worst {np.max(err / (U * tol + 1e-37)):.2f} of the bound"
