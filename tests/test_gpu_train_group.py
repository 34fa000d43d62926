"""Members train in groups: a member's weights and losses do not depend on the
group it trains in.  An ensemble's first member equals the same member trained
alone (same seed, same rows, same shuffles: bit for bit), at batch sizes of one
and of several weight-gradient partials, with a ragged last batch and with
fewer rows than a batch.  A gradient equals the oracle's at the same sizes."""
import numpy as np
import pytest

from geliosphere_gb300 import abi
from geliosphere_gb300 import surrogate as sg
from test_surrogate_oracle import data, init_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,rows", [(256, 256), (256, 1001), (512, 130), (4096, 9000), (16384, 16385)])
def test_member_does_not_depend_on_its_group(engine, batch, rows):
    x, t = data(rows, seed=rows)
    out = []
    for members in (1, 3, 5, 16):
        s = sg.Surrogate(engine, members=members, batch_rows=batch, seed=23)
        s.set_params(0, init_params(seed=1))
        s.add_rows(x, t)
        loss = s.train(3)
        out.append((s.get_params(0), loss[0]))
        s.close()
    for p, loss in out[1:]:
        np.testing.assert_array_equal(p, out[0][0])
        assert loss == out[0][1]


@pytest.mark.parametrize("batch,n", [(256, 1), (256, 256), (512, 257), (1024, 1000)])
def test_gradient_at_small_batches(engine, oracle, batch, n):
    """The bound of the larger batches' test (BF16 activations: 1e-2 of each
    parameter block's norm)."""
    p = init_params(seed=6)
    x, t = data(n, seed=n)
    s = sg.Surrogate(engine, members=1, batch_rows=batch, seed=2)
    s.set_params(0, p)
    loss, g = s.gradient(0, x, t)
    s.close()
    loss_o, g_o = oracle.mlp_grad(p, x, t)
    assert abs(loss - loss_o) <= 1e-2 * loss_o
    for k, (off, shape) in sg.OFFSETS.items():
        m = int(np.prod(shape))
        a, b = g[off:off + m].astype(np.float64), g_o[off:off + m]
        assert np.linalg.norm(a - b) < 1e-2 * max(np.linalg.norm(b), 1e-30), k


@pytest.mark.parametrize("largest", [2 * 4096 * 256 * 2 - 1, 5 * 4096 * 256 * 2 - 1])
def test_training_where_the_whole_group_does_not_fit(engine, largest):
    """Allocations above `largest` (less than two members' activations of a
    4096-row batch, or than five's) and all pinned memory refused: smaller groups
    train, the same bits."""
    x, t = data(9000, seed=9)
    out = []
    for refuse in (False, True):
        s = sg.Surrogate(engine, members=6, batch_rows=4096, seed=4)
        s.add_rows(x, t)
        refused = []

        def hook(kind, nbytes, user):
            no = kind == abi.GELIO_ALLOC_PINNED_HOST or nbytes > largest
            refused.append(no)
            return int(no)

        fn = abi.ALLOC_HOOK(hook)
        if refuse:
            assert engine.lib.gelio_set_alloc_hook(fn, None) == abi.GELIO_OK
        try:
            loss = s.train(2)
        finally:
            engine.lib.gelio_set_alloc_hook(abi.ALLOC_HOOK(), None)
        assert any(refused) == refuse
        out.append([loss] + [s.get_params(m) for m in range(6)])
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
