"""Inference past one batch (262,144 rows) and an ensemble's prediction against the
CPU restatement of the network: rows on both sides of a batch's end come out as
they do alone, and the ensemble's mean and spread are those of the restated
members on the host's features."""
import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim
from geliosphere_gb300 import surrogate as sg
from test_surrogate_oracle import data, init_params

pytestmark = pytest.mark.gpu

BATCH = 262_144


@pytest.mark.parametrize("rows", [BATCH, BATCH + 1, 2 * BATCH + 1037])
def test_forward_past_a_batch(engine, oracle, rows):
    s = sg.Surrogate(engine, members=2, batch_rows=256, seed=3)
    p = init_params(seed=31)
    s.set_params(1, p)
    x, _ = data(rows, seed=8)
    y = s.forward(1, x)
    for end in (BATCH, 2 * BATCH, rows):
        a, b = max(0, min(end, rows) - 700), min(rows, end + 700)
        np.testing.assert_array_equal(y[a:b], s.forward(1, x[a:b]))
    # the bounds of the smaller calls' test: BF16 activations, the two sides round the same values
    pick = np.unique(np.r_[0:300, max(0, BATCH - 300):min(rows, BATCH + 300), rows - 300:rows])
    ref = oracle.mlp_forward(p, x[pick])
    err = np.abs(y[pick] - ref)
    assert np.median(err) < 2e-3 * np.abs(ref).max() and err.max() < 3e-2 * np.abs(ref).max()
    s.close()


@pytest.mark.parametrize("members,points", [(1, 1), (5, 100), (16, 37)])
def test_ensemble_matches_the_restated_members(engine, oracle, members, points):
    s = sg.Surrogate(engine, members=members, batch_rows=256, seed=3)
    params = [init_params(seed=40 + m) for m in range(members)]
    for m, p in enumerate(params):
        s.set_params(m, p)
    sims = [make_sim(abi.GELIO_MODEL_2D_GELIOSPHERE, 1, tilt_deg=5.0 + 7 * i, r_injection=1.0 + 9 * i,
                     polarity=1 if i % 2 else -1, injection=abi.GELIO_INJ_LOG_GRID, inj_points=points) for i in range(8)]
    mean, sd = (np.concatenate(v) for v in s.predict(sims))
    x = np.stack([s.features(q, T) for q in sims for T in sg.grid_energies(q)])
    y = np.stack([oracle.mlp_forward(p, x).astype(np.float64) for p in params])
    scale = np.abs(y).max()
    err = np.abs(mean - y.mean(axis=0))
    assert np.median(err) < 2e-3 * scale and err.max() < 3e-2 * scale
    if members > 1:
        err = np.abs(sd - y.std(axis=0, ddof=1))
        assert np.median(err) < 2e-3 * scale and err.max() < 3e-2 * scale
    else:
        assert np.all(sd == 0.0)
    s.close()
