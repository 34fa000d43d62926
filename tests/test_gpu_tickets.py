"""Tickets of the persistent kernels: the segments in which the simulations of
a launch alternate, and the placement of runs smaller than the launch.  Every
particle is run exactly once whatever the counts, so each simulation's
spectrum equals that of the same simulation in the plain kernel (the same
trajectories: counts and steps exactly, sums up to the order of addition)."""
import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim, spectra_dict

pytestmark = pytest.mark.gpu

LOG = abi.GELIO_INJ_LOG_GRID


def same(a, b):
    a, b = spectra_dict(a), spectra_dict(b)
    for k in a:
        if k.endswith("_n") or k.startswith("n_"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
        else:   # FP64 sums of the same terms in another order
            np.testing.assert_allclose(a[k], b[k], rtol=1e-11, err_msg=k)


# counts below, at and above the 16 segments; empty simulations; more particles than grid points
@pytest.mark.parametrize("counts", [[0, 1, 15, 16, 17], [1], [33, 0, 1000, 7], [5] * 40, [4096, 3, 1501]])
@pytest.mark.parametrize("model,prec", [(abi.GELIO_MODEL_2D_GELIOSPHERE, 0), (abi.GELIO_MODEL_2D_SOLARPROP, 0),
                                        (abi.GELIO_MODEL_1D_BP, 0), (abi.GELIO_MODEL_1D_FP, 0),
                                        (abi.GELIO_MODEL_1D_BP, 1), (abi.GELIO_MODEL_2D_GELIOSPHERE, 1)])
def test_every_particle_once(engine, model, prec, counts):
    lo = 20.0 if model == abi.GELIO_MODEL_1D_BP else 1.0
    sims = [make_sim(model, n, injection=LOG, inj_min=lo, inj_max=100.0, inj_points=9, seed=40 + i)
            for i, n in enumerate(counts)]
    one = engine.run(sims, precision=prec)
    plain = engine.run(sims, precision=prec, plain=True)
    for n, a, b in zip(counts, one.spectra, plain.spectra):
        assert a.n_particles == n
        same(a, b)


# around the placement's lines: one, two, sixteen and all lanes of the launch's 2,432 warps
@pytest.mark.parametrize("n", [2431, 2433, 38911, 38913, 77823, 77825])
def test_small_runs_at_the_lines_of_the_placement(engine, n):
    sim = make_sim(abi.GELIO_MODEL_2D_SOLARPROP, n, injection=LOG, inj_min=30.0, inj_max=100.0, inj_points=7, seed=3)
    same(engine.run(sim).spectra[0], engine.run(sim, plain=True).spectra[0])


# around the lines between one, two, three and four warps a scheduler: 6 trajectories a lane of the fewer
@pytest.mark.parametrize("model", [abi.GELIO_MODEL_2D_GELIOSPHERE, abi.GELIO_MODEL_1D_BP, abi.GELIO_MODEL_1D_FP])
@pytest.mark.parametrize("kw", [{}, {"block_size": 96}, {"block_size": 64, "blocks_per_sm": 3}, {"compact": 2}])
def test_every_particle_once_on_fewer_warps(engine, model, kw):
    for n in (19456, 19457, 116736, 116737, 233473, 350209):
        sim = make_sim(model, n, injection=LOG, inj_min=50.0, inj_max=100.0, inj_points=7, seed=n)
        # the 80-register kernels of the 2D models round differently from the plain one: their own on all warps
        ref = {"compact": 2, "block_size": 32, "blocks_per_sm": 4} if "compact" in kw else {"plain": True}
        same(engine.run(sim, **kw).spectra[0], engine.run(sim, **ref).spectra[0])
