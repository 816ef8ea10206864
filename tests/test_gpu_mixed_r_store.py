"""r_store after a mixed-precision PPCG solve: the r before the last update, bit
for bit.  A solve that tl_max_iters ends one iteration earlier leaves that r.

Loops with odd and even numbers of iterations, fused passes in a graph, one
kernel an inner step, and the last fused pass with the outer sum."""
import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["none", "jac_diag", "jac_block"])
@pytest.mark.parametrize("shape,fusion", [((250, 131), None), ((1030, 411), None), ((1030, 411), (1, 0, False)),
                                          ((517, 403), (5, 0, True)), ((1700, 1602), None)])
def test_r_store_is_the_r_before(precond, shape, fusion):
    got = {}
    for n in (19, 20, 21):
        deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=1, tl_max_iters=n, tl_use_cg=False,
                               tl_use_ppcg=True, tl_ppcg_inner_steps=7, tl_ch_cg_presteps=7, tl_ch_cg_epslim=1.0e10,
                               tl_preconditioner_type=precond, tl_precision="mixed")
        with tl.Chunk(tl.parse_deck(deck)) as ch:
            if fusion:
                ch.set_inner_fusion(*fusion)
            ch.start()
            info = ch.timestep()
            got[n] = info["iterations"], ch.interior("r").copy(), ch.interior("r_store").copy()
    assert got[20][0] == got[19][0] + 1 and got[21][0] == got[20][0] + 1
    assert np.array_equal(got[20][2], got[19][1])
    assert np.array_equal(got[21][2], got[20][1])
