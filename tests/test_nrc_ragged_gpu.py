"""Cache gradients and loss at batches that do not fill their last tile of 128
samples, against the FP64 oracle layer by layer, with test_nrc_gpu's bounds.  The
oracle's batch is the call's own: a live-row mask, a mean over the wrong count or a
column half of another row shows in every layer."""
import numpy as np
import pytest

from kagayaki_gb300 import Scene, scenes
from kagayaki_gb300._lib import check, lib
from oracle import mlp_oracle as mo
from test_nrc_gpu import GRAD_TOL, _p, init, n_params, rand_raw, rand_weights, set_w, split

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("n", [1, 127, 129, 1000, 4097])
def test_gradients_of_a_ragged_batch(width, n):
    tris, mats, _ = scenes.cornell_box()
    w = rand_weights(4, width)
    raw = rand_raw(n, 5)
    tgt = np.random.default_rng(6).uniform(0, 2, (n, 3)).astype(np.float32)
    g = np.empty(n_params(width), np.float32)
    loss = np.zeros(1, np.float32)
    with Scene(tris, mats) as s:
        init(s, width)
        set_w(s, w)
        # a larger call first: its rows lie in the scratch behind the ragged tile
        big = rand_raw(8192, 7)
        check(lib().kgk_nrc_gradients(s._h, _p(big), _p(np.ones((8192, 3), np.float32)), 8192, _p(g), None))
        check(lib().kgk_nrc_gradients(s._h, _p(raw), _p(tgt), n, _p(g), _p(loss)))
    ref_loss, ref_g, _ = mo.gradients(split(w.astype(np.float64), width), raw.astype(np.float64),
                                      tgt.astype(np.float64))
    assert abs(loss[0] - ref_loss) <= 1e-2 * abs(ref_loss)
    for l, (gg, rg) in enumerate(zip(split(g.astype(np.float64), width), ref_g)):
        assert np.linalg.norm(gg - rg) <= GRAD_TOL * np.linalg.norm(rg), l
