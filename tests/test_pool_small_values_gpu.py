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


@pytest.mark.parametrize("symbols", [70, 40000], ids=["split", "unsplit"])
def test_far_samples_beside_near_ones(oracle_mod, symbols):
    """Several chunks of the dictionary, spread over blocks or not.  Samples near the dictionary get the bits that
    they get without the far ones; these are within the 1e-4 of the FP32 form and one step of FP32 of 64 bits, for
    every coefficient."""
    antennas, pilots = 4, 300
    cfg = dict(CFG, dictionarySize=pilots)
    r = np.random.default_rng(symbols)

    def complex_normal(*shape):
        return r.standard_normal(shape) + 1j * r.standard_normal(shape)

    rx = (0.01 * complex_normal(antennas, pilots)).astype(np.complex64)
    tx = (r.choice([-1.0, 1.0], pilots) + 1j * r.choice([-1.0, 1.0], pilots)).astype(np.complex64)
    data = complex_normal(antennas, symbols)
    size = 2 * 0.05 * antennas**2
    data *= np.sqrt(r.uniform(90, 100, symbols) * size / np.sum(np.abs(data) ** 2, axis=0))
    near = np.arange(symbols) % 3 != 1
    data[:, near] *= 0.01
    data = data.astype(np.complex64)
    pool = DetectorPool(cfg)
    d = pool.add(antennas)
    pool.run([PoolJob(d, rx, tx)])
    est = pool.run([PoolJob(d, data)])[0].copy()
    alone = pool.run([PoolJob(d, np.ascontiguousarray(data[:, near]))])[0]
    np.testing.assert_array_equal(est[near], alone)
    o = oracle_mod.OracleDetector(cfg, antennas, oracle_mod.F64)
    o.train(rx, tx)
    far = np.flatnonzero(~near)[:500]
    ref = o.detect(np.ascontiguousarray(data[:, far]))
    assert 0.0 < np.max(np.abs(ref)) < 2.0**-126
    rows = np.concatenate([rx.T, -1j * rx.T]).astype(np.complex128)
    x = data[:, far].T.astype(np.complex128)
    total = float(np.sum(np.abs(o.get_state()["a"])))
    for got, part, rotated in ((est[far].real, ref.real, x), (est[far].imag, ref.imag, -1j * x)):
        largest = np.exp(-np.min(np.sum(np.abs(rotated[:, None] - rows[None]) ** 2, -1), axis=1) / size)
        assert np.all(np.abs(got.astype(np.float64) - part) <= total * (1e-4 * largest + 2.0**-149))
