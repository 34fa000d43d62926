"""The kernels of both register budgets integrate the same trajectories: a
SolarProp-like run's exit records do not depend on the budget that an option or the
tuner picks, nor on the kernel (plain, one thread a particle)."""
import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(inj_min=0.05, tilt_deg=20.0), dict(inj_min=0.3, tilt_deg=70.0, polarity=-1, flags=1),
                                dict(inj_min=0.1, r_injection=30.0, theta_deg=150.0, tilt_deg=45.0)])
def test_solarprop_records_do_not_depend_on_the_budget(engine, kw):
    sim = make_sim(abi.GELIO_MODEL_2D_SOLARPROP, 30_000, injection=abi.GELIO_INJ_LOG_GRID, inj_max=150.0, inj_points=29,
                   seed=12, **kw)
    out = []
    for opts in ({"compact": 1}, {"compact": 2}, {"compact": 2, "block_size": 96}, {"plain": True}):
        k = engine.run(sim, record_capacity=40_000, **opts).records
        out.append(k[np.lexsort((k["r"], k["t_exit"], k["particle"]))])
    for k in out[1:]:
        for f in k.dtype.names:
            np.testing.assert_array_equal(k[f], out[0][f], err_msg=f)
