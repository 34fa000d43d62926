"""The 1D kernels integrate four steps as one block where no rare event can
fall into them, and step by step otherwise.  Where events are frequent (starts
beside the inner boundary, beside 1 AU, beside the outer edge, large steps,
caps inside a group) the persistent kernel's records equal those of the plain
kernel, which takes every step by itself, bit for bit."""
import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim

pytestmark = pytest.mark.gpu


def records(engine, sim, **kw):
    r = engine.run(sim, record_capacity=400_000, check=False, **kw)
    assert r.status in (abi.GELIO_OK, abi.GELIO_WARN_STEP_CAP)
    k = r.records
    s = r.spectra[0]
    return (k[np.lexsort((k["r"], k["sumac"], k["t_exit"], k["particle"]))],
            (s.n_particles, s.n_records, s.n_steps, s.n_lost, s.n_step_capped))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("model,kw", [
    (abi.GELIO_MODEL_1D_BP, dict(r_injection=0.3, inj_min=30.0)),                  # undone steps at the inner boundary
    (abi.GELIO_MODEL_1D_BP, dict(r_injection=99.5, inj_min=5.0)),                  # exits in the first steps
    (abi.GELIO_MODEL_1D_BP, dict(r_injection=1.0, inj_min=20.0, dt=5000.0)),       # steps of many AU
    (abi.GELIO_MODEL_1D_BP, dict(r_injection=1.0, inj_min=180.0, inj_max=300.0)),  # energies past the 200 GeV window
    (abi.GELIO_MODEL_1D_FP, dict(inj_min=1.0)),                                    # crossings of 1 AU, outer exits
    (abi.GELIO_MODEL_1D_FP, dict(inj_min=30.0, inj_max=300.0, dt=2000.0)),         # large steps, past the 100 GeV window
])
@pytest.mark.parametrize("max_steps", [0, 5, 402])
def test_records_equal_the_plain_kernels(engine, model, kw, prec, max_steps):
    p = dict(injection=abi.GELIO_INJ_LOG_GRID, inj_points=11, inj_max=100.0, seed=8)
    p.update(kw)
    sim = make_sim(model, 6000 if prec == 0 else 600, **p)
    a, na = records(engine, sim, precision=prec, max_steps=max_steps)
    b, nb = records(engine, sim, precision=prec, max_steps=max_steps, plain=True)
    assert na == nb
    for f in a.dtype.names:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)
