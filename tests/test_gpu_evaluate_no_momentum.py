"""gelio_evaluate of 2D rows whose exit energy has no momentum (0, or negative and
above -2 T0): their bin's three spectra are not numbers, as the reference's square
root of a negative number makes them, and the other rows' bins are what they are
without them."""
import numpy as np
import pytest

from geliosphere_gb300 import abi

pytestmark = pytest.mark.gpu

SP = 0.01 * 1.5 ** np.arange(12)        # centres of twelve windows


@pytest.mark.parametrize("te", [-1.0, -0.5, -1e-6, 0.0])
@pytest.mark.parametrize("n", [12, 1200, 60_000])
def test_weights_are_not_numbers(engine, n, te):
    ti = np.array([float("%g" % t) for t in np.resize(SP, n)])
    rows = np.stack([ti, np.array([float("%g" % t) for t in ti + 0.3])] + [np.ones(n)] * 4, 1)
    good = engine.evaluate(abi.GELIO_MODEL_2D_GELIOSPHERE, rows)
    rows[5, 1] = te                     # a row of the sixth window
    sp = engine.evaluate(abi.GELIO_MODEL_2D_GELIOSPHERE, rows)
    for name in ("sp_weber", "sp_jgr", "sp_burger"):
        a, b = np.array(getattr(sp, name)), np.array(getattr(good, name))
        assert np.isnan(a[6]), name
        a[6] = b[6]
        np.testing.assert_allclose(a, b, rtol=1e-12, err_msg=name)
    np.testing.assert_array_equal(sp.sp_n, good.sp_n)
