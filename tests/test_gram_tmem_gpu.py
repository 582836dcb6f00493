"""The Gram forms with the data tile in tensor memory (gram_tf32x3; gram_bf16
with four users or more) at the edges of their layout: feature counts around
the ring slice of 32 and the K steps of 8 and 16, dictionaries around the chunk
of 128 rows, of one to seven chunks and split over blocks, data rows around the
tile of 128, every class of user counts.  Reference and bounds as for the other
sizes of these forms: the float64 model of the same state, 2e-5 and 2e-3 of the
largest soft output (operands carry 2^-21 and 2^-8 of |x||d|)."""
import numpy as np
import pytest

import libapsm_b200 as L
from libapsm_b200 import synth

pytestmark = pytest.mark.gpu

CASES = [  # antennas, users, pilots (two rows each), symbols (two rows each)
    (1, 1, 1, 1),
    (3, 2, 64, 63),
    (4, 3, 63, 64),
    (12, 1, 65, 65),
    (15, 4, 129, 130),
    (16, 5, 200, 2),
    (17, 8, 127, 9472),
    (20, 9, 40, 90),
    (32, 16, 66, 129),
    (33, 1, 130, 33),
    (48, 12, 70, 70),
    (63, 7, 64, 127),
    (64, 2, 200, 64),
    (24, 4, 321, 9472),
    (8, 16, 400, 9473),
]
FORMS = {"gram_tf32x3": 2e-5, "gram_bf16": 2e-3}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("antennas,users,pilots,symbols", CASES)
def test_layout_edges(oracle_mod, form, antennas, users, pilots, symbols):
    K = min(users, 4)
    f = synth.generate_frame(antennas + users, K=K, N=antennas, P=pilots, S=symbols, modulation="QAM16", snr_db=20)
    tx = np.stack([f.tx_train[u % K] * (1.0 + 0.1 * (u // K)) for u in range(users)])
    cfg = {"otype": "APSM", "windowSize": 20, "gaussianKernelVariance": 0.5, "eB": 0.01,
           "detectVersion": form}
    det = L.NomaDetectorFactory.build(cfg, antennas, num_users=users)
    det.train(f.rx_train, tx)
    est = np.atleast_2d(det.detect(f.rx_data)[0])
    st = det.get_state()
    refs = []
    for u in range(users):
        o = oracle_mod.OracleDetector(cfg, antennas, oracle_mod.F64)
        o.set_state(st["dictionary"], st["a"][u], st["w"][u])
        refs.append(o.detect(f.rx_data))
    refs = np.stack(refs)
    assert np.max(np.abs(est - refs)) <= FORMS[form] * np.max(np.abs(refs))
