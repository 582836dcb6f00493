"""Least-squares training and detection on the GPU at the edges of the solver
and of the linear kernel: features around a warp's 32 lanes, odd right-hand
sides, more users than one pass of the linear kernel, pilot rows around the
blocks of 64.

Reference: numpy's float64 least squares.  Bound: the weights round to FP32 and
D products are summed in FP32, (D + 2) 2^-24 sum |w| |x|, plus the solve in
FP64 through the normal equations, far below that (condition numbers here are
under 1e3, so 1e6 * 2^-53)."""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("antennas,users,pilots,symbols", [
    (1, 1, 2, 1), (2, 3, 31, 63), (15, 2, 32, 64), (16, 8, 33, 65), (17, 17, 100, 130), (31, 5, 64, 40),
    (32, 16, 65, 33), (33, 33, 129, 64), (64, 7, 300, 129)])
def test_matches_float64_least_squares(antennas, users, pilots, symbols):
    K = min(users, 4)
    f = synth.generate_frame(7 * antennas + users, K=K, N=antennas, P=pilots, S=symbols, modulation="QAM16", snr_db=10)
    tx = np.stack([f.tx_train[u % K] * (1.0 + 0.1 * (u // K)) for u in range(users)]).astype(np.complex64)
    det = L.NomaDetectorFactory.build({"otype": "LLS"}, antennas, num_users=users)
    det.train(f.rx_train, tx)
    est = np.atleast_2d(det.detect(f.rx_data)[0])

    def rows(rx):
        y = np.asarray(rx, dtype=np.complex64).astype(np.complex128).T
        return np.stack([np.concatenate([y.real, y.imag], 1), np.concatenate([y.imag, -y.real], 1)], 1).reshape(
            -1, 2 * antennas)

    a, x = rows(f.rx_train), rows(f.rx_data)
    targets = np.stack([tx.real, tx.imag], -1).reshape(users, -1).astype(np.float64)
    w = np.linalg.lstsq(a, targets.T, rcond=None)[0]
    ref = (x @ w).T
    tol = ((2 * antennas + 2) * 2.0**-24 * (np.abs(x) @ np.abs(w))).T + 1e-9 * np.max(np.abs(ref))
    got = np.stack([est.real, est.imag], -1).reshape(users, -1)
    assert (np.abs(got - ref) <= tol).all(), np.max(np.abs(got - ref) / tol)
