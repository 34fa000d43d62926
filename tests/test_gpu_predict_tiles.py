"""The fused network kernel at the edges of its tiles and of its work items:
a member's last pair of tiles may have one tile only, and a CTA may meet such
an item before, between or after whole pairs.  The ensemble's mean and spread
equal those of the members run one by one (another division into items), and a
row's output does not depend on the rows around it."""
import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim
from geliosphere_gb300 import surrogate as sg
from test_surrogate_oracle import init_params

pytestmark = pytest.mark.gpu


# rows: below, at and above a tile and a pair; with 5 and 16 members some CTAs
# (152) get two items and more, one of them a lone tile
@pytest.mark.parametrize("members,rows", [(1, 1), (2, 127), (2, 128), (2, 129), (3, 255), (3, 257), (5, 7936 + 64),
                                          (5, 10_000), (16, 2500), (16, 5000), (1, 152 * 256 + 100), (1, 262_144 + 300)])
def test_members_one_by_one(engine, members, rows):
    s = sg.Surrogate(engine, members=members, batch_rows=256, seed=9)
    for m in range(members):
        s.set_params(m, init_params(seed=60 + m))
    sims, left, i = [], rows, 0
    while left:
        pts = min(left, (1, 7, 100, 320)[i % 4] if rows < 20_000 else 320)
        sims.append(make_sim(abi.GELIO_MODEL_2D_GELIOSPHERE, 1, tilt_deg=5.0 + i % 60, r_injection=1.0 + i % 70,
                             injection=abi.GELIO_INJ_LOG_GRID, inj_points=pts))
        left -= pts
        i += 1
    mean, sd = s.predict(sims)
    mean, sd = np.concatenate(mean), np.concatenate(sd)
    pick = np.unique(np.r_[0:min(rows, 300), max(0, rows - 300):rows, np.arange(0, rows, 997)])
    x = [s.features(sim, T) for sim in sims for T in sg.grid_energies(sim)] if rows < 20_000 else None
    if x is None:          # the host's features of the picked rows only
        first = np.cumsum([0] + [q.inj_points for q in sims])
        where = [(int(np.searchsorted(first, r, "right")) - 1, r) for r in pick]
        xs = np.stack([s.features(sims[k], sg.grid_energies(sims[k])[r - first[k]]) for k, r in where])
    else:
        xs = np.stack([x[r] for r in pick])
    y = np.stack([s.forward(m, xs).astype(np.float64) for m in range(members)])
    # FP64 statistics of the same FP32 outputs: some roundings
    np.testing.assert_allclose(mean[pick], y.mean(axis=0), rtol=1e-12, atol=1e-12)
    if members > 1:
        np.testing.assert_allclose(sd[pick], y.std(axis=0, ddof=1), rtol=1e-9, atol=1e-12)
    s.close()
