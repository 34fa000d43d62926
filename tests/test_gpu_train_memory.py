"""A surrogate that could be created can be trained: one member's training memory
is taken at create, and where a group's is refused the members train in smaller
groups, one by one at last, with the same weights."""
import numpy as np
import pytest

from geliosphere_gb300 import abi
from geliosphere_gb300 import surrogate as sg
from test_surrogate_oracle import data

pytestmark = pytest.mark.gpu


# allocations that go through once training starts: the rows (2 x), and then the losses and
# orders of a member, which are smaller than any activation buffer (4096 x 256 x 2 bytes)
@pytest.mark.parametrize("members", [1, 3, 6])
def test_no_activation_buffer_after_create(engine, members):
    x, t = data(6000, seed=9)
    out = []
    for refuse in (False, True):
        s = sg.Surrogate(engine, members=members, batch_rows=4096, seed=4)
        s.add_rows(x, t)
        fn = abi.ALLOC_HOOK(lambda kind, nbytes, user: int(kind == abi.GELIO_ALLOC_DEVICE and nbytes >= 4096 * 256 * 2))
        if refuse:
            assert engine.lib.gelio_set_alloc_hook(fn, None) == abi.GELIO_OK
        try:
            loss = s.train(2)
            g = s.gradient(0, x[:500], t[:500])
        finally:
            engine.lib.gelio_set_alloc_hook(abi.ALLOC_HOOK(), None)
        out.append([loss, g[0], g[1]] + [s.get_params(m) for m in range(members)])
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_create_is_refused_where_training_would_be(engine):
    fn = abi.ALLOC_HOOK(lambda kind, nbytes, user: int(nbytes == 16384 * 256 * 2))      # an activation buffer
    assert engine.lib.gelio_set_alloc_hook(fn, None) == abi.GELIO_OK
    try:
        with pytest.raises(abi.GelioError) as ei:
            sg.Surrogate(engine, members=5, batch_rows=16384)
        assert ei.value.status == abi.GELIO_ERR_OUT_OF_MEMORY
    finally:
        engine.lib.gelio_set_alloc_hook(abi.ALLOC_HOOK(), None)
