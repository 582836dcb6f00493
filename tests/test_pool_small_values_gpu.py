"""FP32 detection of the pool where every kernel value lies below the smallest
normal FP32 number: a model without a linear part (gaussianKernelWeight 1) and
samples far from its dictionary.  The reference's expf
(apsm_detect.cu:131-152) keeps such values, and with them the sign that a hard
decision takes.

Bound: 1e-4 of the largest soft output, the bar of the pool's FP32 form, and 4
roundings to FP32's smallest step (2^-149) for each of the sum's terms."""
import numpy as np
import pytest

from libapsm_b200 import DetectorPool, PoolJob

pytestmark = pytest.mark.gpu

CFG = {"otype": "APSM", "windowSize": 4, "gaussianKernelVariance": 0.05, "gaussianKernelWeight": 1.0, "eB": 0.01,
       "dictionarySize": 40}


@pytest.mark.parametrize("antennas,pilots,symbols", [(1, 12, 9), (4, 12, 40), (32, 12, 33)])
def test_kernel_values_below_the_normal_range(oracle_mod, antennas, pilots, symbols):
    r = np.random.default_rng(antennas)

    def complex_normal(*shape):
        return r.standard_normal(shape) + 1j * r.standard_normal(shape)

    rx = (0.01 * complex_normal(antennas, pilots)).astype(np.complex64)
    tx = (r.choice([-1.0, 1.0], pilots) + 1j * r.choice([-1.0, 1.0], pilots)).astype(np.complex64)
    data = complex_normal(antennas, symbols)
    # squared distances of 90 to 100 times 2 variance N^2: exponentials of 3e-44 to 8e-40
    data *= np.sqrt(r.uniform(90, 100, symbols) * 2 * 0.05 * antennas**2 / np.sum(np.abs(data) ** 2, axis=0))
    data = data.astype(np.complex64)
    pool = DetectorPool(CFG)
    d = pool.add(antennas)
    pool.run([PoolJob(d, rx, tx)])
    est = pool.run([PoolJob(d, data)])[0]
    o = oracle_mod.OracleDetector(CFG, antennas, oracle_mod.F64)
    o.train(rx, tx)
    ref = o.detect(data)
    largest = float(np.max(np.abs(ref)))
    assert 0.0 < largest < 2.0**-126
    bound = 1e-4 * largest + 4 * 2 * pilots * 2.0**-149
    assert np.max(np.abs(est.real.astype(np.float64) - ref.real)) <= bound
    assert np.max(np.abs(est.imag.astype(np.float64) - ref.imag)) <= bound
