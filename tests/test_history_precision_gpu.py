"""Training history of long calls against the model in 64 bits.

Every step's EVM (noma_train_history.cu:65-128) comes from that step's
coefficients and linear weights.  Calls of thousands of steps, with eviction
and in blocks (more than 2729 visible pairs), show a drift of either: the
weights are a running sum over all steps.

Bound: 6e-7 relative.  The sweep's coefficients and weights are within 2e-7 of 64
bits whatever the number of steps (its compensated sums), each moves an EVM by no
more than that, and three roundings (2e-7) are left for the sums of the EVM; a
weight that drifts over the steps is 1e-6 away at these sizes."""
import numpy as np
import pytest
import torch

import libapsm_b200 as L

pytestmark = pytest.mark.gpu

RTOL = 6e-7


def frame(seed, antennas, n):
    r = np.random.default_rng(seed)
    tx = ((r.integers(0, 2, (3, n)) * 2 - 1) + 1j * (r.integers(0, 2, (3, n)) * 2 - 1)) / np.sqrt(2)
    h = (r.standard_normal((antennas, 3)) + 1j * r.standard_normal((antennas, 3))) / np.sqrt(2)
    noise = r.standard_normal((antennas, n)) + 1j * r.standard_normal((antennas, n))
    return (h @ tx + 0.3 * noise).astype(np.complex64), tx[0].astype(np.complex64)


def dedup(rx):
    y = torch.tensor(rx.T.astype(np.complex128), device="cuda")
    return torch.stack([torch.cat([y.real, y.imag], -1), torch.cat([y.imag, -y.real], -1)], -2).flatten(0, 1)


def evm64(rx, tx, P, window, capacity, variance, eb, marks):
    """(training EVM, validation EVM) after the steps `marks`, the whole sweep in 64 bits."""
    N = rx.shape[0]
    X = dedup(rx)
    x = X[: 2 * P]
    target = torch.view_as_real(torch.tensor(tx, device="cuda").to(torch.complex128)).flatten()
    ew = -0.5 / (float(np.float32(variance)) * N * N)
    eb = float(np.float32(eb))
    d2 = X.square().sum(1)[:, None] + x.square().sum(1)[None] - 2 * X @ x.T
    k = d2.clamp_(min=0).mul_(ew).exp_().mul_(0.5)
    norms = 0.5 * x.square().sum(1) + 0.5
    a = torch.zeros(2 * P, dtype=torch.float64, device="cuda")
    w = torch.zeros(2 * N, dtype=torch.float64, device="cuda")
    out = {}
    for t in range(P):
        hi = 2 * t + 2
        lo, w0 = max(0, hi - 2 * capacity), max(0, hi - 2 * min(window, capacity))
        e = target[w0:hi] - 0.5 * x[w0:hi] @ w - k[w0:hi, lo:hi] @ a[lo:hi]
        c = e.sign() * (e.abs() - eb).clamp(min=0) / (hi - w0) / norms[w0:hi]
        a[w0:hi] += c
        w += c @ x[w0:hi]
        if t in marks:
            err = (0.5 * X @ w + k[:, lo:hi] @ a[lo:hi] - target).square().view(-1, 2).sum(1)
            out[t] = float(err[:P].mean().sqrt()), float(err[P:].mean().sqrt())
    return out


@pytest.mark.parametrize("N,P,window,dictionary", [(16, 2500, 20, 2500), (8, 4000, 20, 4000), (8, 4000, 80, 3000)])
def test_evm_of_long_calls(N, P, window, dictionary):
    rx, tx = frame(P + N, N, P + 400)
    det = L.NomaDetectorFactory.build({"otype": "APSM", "windowSize": window, "gaussianKernelVariance": 0.5, "eB": 0.01,
                                       "dictionarySize": dictionary}, N)
    mod = L.Modulation("QPSK")
    hist = L.NomaTrainHistory(mod.bps, mod.scale)
    det.train(rx[:, :P].copy(), tx[:P].copy(), val_set=(hist, rx[:, P:].copy(), tx[P:].copy()))
    steps = np.asarray(hist.steps, np.float64)
    marks = sorted({0, 1, window, P // 2, P - 2, P - 1} | set(range(0, P, P // 16)))
    for t, ref in evm64(rx, tx, P, window, dictionary, 0.5, 0.01, set(marks)).items():
        np.testing.assert_allclose(steps[t, [0, 3]], ref, rtol=RTOL, err_msg=f"step {t}")
