"""apsm_last_kernel_ms is the time of the training sweep alone (the denominator of
roofline figures; the reference returns one event time per call,
apsm_train.cu:163-165): forming the kernel columns is no part of it.

The columns take at least 6 FP32 instructions per antenna for every two pairs
that meet (three differences, three fma, packed by twos), so a call's own event
time exceeds its sweep's by that at the chip's full rate."""
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

FP32_PER_S = 148 * 128 * 1.965e9


@pytest.mark.parametrize("pilots,dictionary", [(8000, 2700), (6000, 6000)], ids=["one launch", "blocks"])
def test_columns_are_not_counted(pilots, dictionary):
    f = synth.generate_frame(77, K=2, N=64, P=pilots, S=16, modulation="QPSK", snr_db=20)
    det = L.NomaDetectorFactory.build({"otype": "APSM", "windowSize": 20, "gaussianKernelVariance": 0.5, "eB": 0.01,
                                       "dictionarySize": dictionary}, 64)
    for _ in range(2):  # (the first call allocates)
        det.reset_state()
        ms = det.train(f.rx_train, f.tx_train[0])
    sweep, detect = det.last_kernel_ms()
    met = sum(min(t + 1, dictionary) for t in range(pilots))
    assert detect == -1 and 0.0 < sweep < ms - 1e3 * 6 * 64 * met / FP32_PER_S
