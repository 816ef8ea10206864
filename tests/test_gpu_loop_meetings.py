"""The meetings of the loop kernels' thread blocks (many iterations a launch)."""
import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,precond", [("cg", "none"), ("cg", "jac_diag"), ("ppcg", "jac_block")])
@pytest.mark.parametrize("shape", [(9, 8), (96, 80), (130, 37)])
def test_mixed_cg_loop_completes_its_groups_of_sums(solver, precond, shape):
    """Fifteen warps pass, and the sums of a group are added by fours: the
    sixteenth warp's are zeros that are there before the first sum of a launch.
    Few rows, so that the warps of the last group have none and come to their
    first sum at once; FP64 loops in between leave other values in the shared
    memory.  Every solve gives the same bits."""
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=1, tl_max_iters=4000, tl_eps=1e-9,
                           tl_use_cg=solver == "cg", tl_use_ppcg=solver == "ppcg", tl_ch_cg_presteps=12,
                           tl_preconditioner_type=precond, tl_precision="mixed")
    other = decks.make_deck(x_cells=700, y_cells=333, end_step=1, tl_max_iters=20, tl_preconditioner_type="jac_diag")
    got = []
    with tl.Chunk(tl.parse_deck(deck)) as ch, tl.Chunk(tl.parse_deck(other)) as fp64:
        for _ in range(12):
            fp64.start()
            fp64.timestep()
            ch.start()
            info = ch.timestep()
            got.append((info["status"], info["iterations"], info["error"], ch.interior("u").copy()))
    assert got[0][0] == 0 and got[0][1] > 2
    for g in got[1:]:
        assert g[:3] == got[0][:3]
        assert np.array_equal(g[3], got[0][3])
