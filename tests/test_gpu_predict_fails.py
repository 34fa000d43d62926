"""A prediction that fails on the device (a wait of its kernels ran out: the error
flag, which the test sets) leaves the caller's arrays as they were, with few rows
and with many, and the next one succeeds."""
import ctypes

import numpy as np
import pytest

from geliosphere_gb300 import abi, make_sim
from geliosphere_gb300 import surrogate as sg
from test_surrogate_oracle import init_params

pytestmark = pytest.mark.gpu


# rows: through the staging (16,384 and fewer) and straight into the arrays
@pytest.mark.parametrize("rows", [100, 8193, 16_384, 16_385, 50_000])
def test_arrays_stay_as_they_were(engine, rows):
    s = sg.Surrogate(engine, members=2, batch_rows=256, seed=3)
    for m in range(2):
        s.set_params(m, init_params(seed=m))
    sims, left = [], rows
    while left:
        sims.append(make_sim(abi.GELIO_MODEL_2D_GELIOSPHERE, 1, tilt_deg=len(sims) % 70, injection=abi.GELIO_INJ_LOG_GRID,
                             inj_points=min(left, 320)))
        left -= sims[-1].inj_points
    arr = (abi.SimParams * len(sims))(*sims)
    want = np.zeros(rows), np.zeros(rows)
    s.predict_into(arr, len(sims), *want)
    r, sd = np.full(rows, -7.0), np.full(rows, -9.0)
    set_error = s.lib.gelio_internal_surrogate_error
    set_error.restype, set_error.argtypes = ctypes.c_int32, [ctypes.c_void_p, ctypes.c_uint32]
    assert set_error(s.h, 12) == abi.GELIO_OK
    with pytest.raises(abi.GelioError) as ei:
        s.predict_into(arr, len(sims), r, sd)
    assert ei.value.status == abi.GELIO_ERR_TIMEOUT
    assert np.all(r == -7.0) and np.all(sd == -9.0)
    s.predict_into(arr, len(sims), r, sd)
    np.testing.assert_array_equal(r, want[0])
    np.testing.assert_array_equal(sd, want[1])
    s.close()
