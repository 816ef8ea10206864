"""The network's inputs where the previous increment is not finite."""
import ctypes as C

import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu

CLAMP = 64.0  # bound of the scaled inputs


@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_infinite_increment_is_clamped_with_its_sign(value):
    torch = pytest.importorskip("torch")
    lib = tl.load()
    deck = decks.make_deck(x_cells=40, y_cells=24, end_step=3, tl_preconditioner_type="jac_diag",
                           tl_warm_start="prev", tl_max_iters=50)
    with tl.Chunk(tl.parse_deck(deck)) as ch:
        ch.start()
        e = ch.get_field("energy1")
        bad = e.copy()
        bad[9, 13] = value
        ch.set_field("energy1", bad)
        with pytest.raises(tl.TeaLeafError):  # breakdown: its u^n is the next step's u^(n-1)
            ch.timestep()
        ch.set_field("energy1", e)
        assert ch.timestep()["status"] >= 0
        f = torch.zeros(24, 40, 8, dtype=torch.float32, device="cuda")
        assert lib.tl_warm_start_features(ch._h, C.c_void_p(f.data_ptr())) == 0, tl.last_error()
        f = f.cpu().numpy()
    h = 1
    assert f[9 - h, 13 - h, 6] == -np.sign(value) * CLAMP
    assert np.isfinite(f).all()
