"""A run beside another context's run: the other holds part of every SM, so some
of this run's CTAs are not resident until it ends.  Their share of the tickets is
taken by the CTAs that are: the same spectra, in about the time that the same run
takes with a grid that fits."""
import threading
import time

import pytest

from geliosphere_gb300 import Engine, abi, make_sim
from test_gpu_tickets import same

pytestmark = pytest.mark.gpu

GRID = dict(injection=abi.GELIO_INJ_LOG_GRID, inj_min=0.05, inj_max=100.0, inj_points=50)


@pytest.fixture(scope="module")
def other():
    e = Engine(0)
    yield e
    e.close()


def beside(other, fn):
    """fn() while the other context's run has one CTA of eight warps on each SM
    for some 300 ms and more; whether it outlasted fn."""
    sims = [make_sim(abi.GELIO_MODEL_2D_GELIOSPHERE, 3_000_000, seed=70 + i, tilt_deg=20 + i, **GRID) for i in range(4)]
    t = threading.Thread(target=lambda: other.run(sims, block_size=256, blocks_per_sm=1))
    t.start()
    time.sleep(0.05)
    r = fn()
    outlasted = t.is_alive()
    t.join()
    return r, outlasted


# one lane a warp, several, all of them, and more tickets than lanes; lanes refilled in the tail's draws
@pytest.mark.parametrize("model,n,prec", [(abi.GELIO_MODEL_1D_BP, 2000, 0), (abi.GELIO_MODEL_1D_BP, 19_000, 0),
                                          (abi.GELIO_MODEL_1D_BP, 60_000, 0), (abi.GELIO_MODEL_1D_FP, 70_000, 0),
                                          (abi.GELIO_MODEL_1D_FP, 4000, 1), (abi.GELIO_MODEL_2D_GELIOSPHERE, 19_000, 0),
                                          (abi.GELIO_MODEL_2D_SOLARPROP, 150_000, 0)])
def test_same_spectra(engine, other, model, n, prec):
    kw = dict(GRID, inj_min=1.0) if model == abi.GELIO_MODEL_1D_BP or prec else GRID
    sim = make_sim(model, n, seed=5, **kw)
    want = engine.run(sim, precision=prec).spectra[0]
    got, _ = beside(other, lambda: engine.run(sim, precision=prec).spectra[0])
    assert got.n_particles == n
    same(got, want)


@pytest.mark.parametrize("model,n", [(abi.GELIO_MODEL_2D_GELIOSPHERE, 250_000), (abi.GELIO_MODEL_2D_SOLARPROP, 60_000)])
def test_ctas_that_wait_keep_no_tickets(engine, other, model, n):
    sim = make_sim(model, n, seed=1, **GRID)
    engine.run(sim)

    def ms(**kw):
        best, tries = float("inf"), 0
        while tries < 3:
            r, outlasted = beside(other, lambda: engine.run(sim, **kw).stats.kernel_ms)
            if outlasted:
                best, tries = min(best, r), tries + 1
        return best

    # 1.09 to 1.14 times; 1.5 to 1.6 with the first tickets tied to the CTAs
    assert ms() <= 1.3 * ms(block_size=256, blocks_per_sm=1)
