"""gelio_evaluate on rows that sit where its paths change: blocks of one energy
and of all-distinct energies, part blocks, the sizes at which the rows go up
in pieces, values on bin edges, zeros, NaN and infinities.  The bins of the
reference's evaluators in NumPy: counts exact, sums to 1e-12 (FP64 weights
from other groupings of the same logarithms: some tens of roundings)."""
import numpy as np
import pytest

from geliosphere_gb300 import abi
from perf import cases

pytestmark = pytest.mark.gpu


def check(engine, model, rows, monkeypatch):
    monkeypatch.setattr(cases, "_log_rows", lambda case, seed: rows)
    want = cases._exact_evaluate({"model": model, "rows": len(rows)}, 0)
    got = engine.evaluate(cases.MODELS[model], rows)
    for name in cases.FIELDS:
        g = getattr(got, name)
        g = g if isinstance(g, float) else np.ctypeslib.as_array(g)
        if name.startswith("n_") or name.endswith("_n"):
            np.testing.assert_array_equal(g, want[name], err_msg=name)
        else:
            np.testing.assert_allclose(g, want[name], rtol=1e-12, err_msg=name)


# around one warp, one block, the line of the slices, two pieces of rows and several
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 32_768, 32_769, 131_071, 131_073, 600_001])
@pytest.mark.parametrize("model", ["2D Geliosphere", "1D Bp", "1D Fp"])
def test_sizes(engine, model, n, monkeypatch):
    rows = cases._log_rows({"model": model, "rows": min(n, 4099)}, n)
    check(engine, model, np.resize(rows, (n, rows.shape[1])), monkeypatch)


@pytest.mark.parametrize("energies", ["one", "distinct", "edges"])
def test_2d_energies(engine, energies, monkeypatch):
    n = 5000
    rng = np.random.default_rng(3)
    if energies == "one":
        ti = np.full(n, 0.57665)
    elif energies == "distinct":
        ti = np.array([float("%g" % v) for v in np.arange(1, n + 1) / 400.0])
    else:
        ti = np.array(cases.SP + cases.AMS + [0.125, 0.25, 2.0] + [float("%g" % (f * e)) for e in cases.SP
                                                                    for f in (0.99, 1.01, 0.995)])
        ti = np.resize(ti, n)
    te = np.array([float("%g" % v) for v in ti + rng.gamma(2.0, 0.3, n)])
    rows = np.stack([ti, te] + [np.ones(n)] * 4, 1)
    check(engine, "2D SolarProp-like", rows, monkeypatch)


def test_2d_unusual_values_do_not_disturb_the_others(engine):
    """Zero, negative, infinite and NaN energies land in no bin (or only
    their own); the other rows' bins are what they are without them."""
    good = cases._log_rows({"model": "2D Geliosphere", "rows": 1500}, 4)
    odd = np.tile(good[:1], (8, 1))
    odd[:, 0] = [0.0, -1.0, np.inf, -np.inf, np.nan, 1e-300, 1e300, 5e-324]
    both = np.concatenate([good[:700], odd, good[700:]])
    a, b = engine.evaluate(3, good), engine.evaluate(3, both)
    for name in cases.FIELDS:
        x, y = getattr(a, name), getattr(b, name)
        if name == "n_records":
            assert y == x + len(odd)
        else:
            x, y = np.asarray(x, dtype=np.float64), np.asarray(y, dtype=np.float64)
            np.testing.assert_allclose(y, x, rtol=1e-12, err_msg=name)
    nan = np.full(1, 0xFFFFFFFFFFFFFFFF, np.uint64).view(np.float64)   # every bit set
    rows = good[:3].copy()
    rows[1, 0] = nan[0]
    assert engine.evaluate(3, rows).n_records == 3.0
