"""Every particle is run once on both sides of the lines at which a launch's
placement changes, wherever they lie on this device: the lanes of a warp that draw
together (8 in FP32 steps, 16 in FP64), one trajectory on each lane, and two and
six on each lane of four warps an SM."""
import pytest

from geliosphere_gb300 import abi, make_sim
from test_gpu_tickets import same

pytestmark = pytest.mark.gpu


def lines(engine, sim, prec):
    st = engine.run(sim, precision=prec).stats
    warps = st.grid_size * st.block_size // 32
    sms = st.grid_size // st.blocks_per_sm
    if prec:
        return [warps, 16 * warps, 32 * warps]
    return [warps, 8 * warps, 32 * warps] + [k * 4 * 32 * sms * f for k in (1, 2, 3) for f in (2, 6)]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("model", [abi.GELIO_MODEL_2D_GELIOSPHERE, abi.GELIO_MODEL_2D_SOLARPROP, abi.GELIO_MODEL_1D_BP,
                                   abi.GELIO_MODEL_1D_FP])
def test_every_particle_once_at_each_line(engine, model, prec):
    # short trajectories, of like lengths and (grid from 2 GeV) not
    for kw in (dict(inj_min=60.0, inj_max=100.0), dict(inj_min=2.0, inj_max=100.0)):
        def make(n):
            return make_sim(model, n, injection=abi.GELIO_INJ_LOG_GRID, inj_points=7, seed=n, **kw)
        if prec and kw["inj_min"] < 60.0:
            continue
        for line in lines(engine, make(1000), prec):
            for n in (line, line + 1):
                a = engine.run(make(n), precision=prec).spectra[0]
                assert a.n_particles == n
                same(a, engine.run(make(n), precision=prec, plain=True).spectra[0])
