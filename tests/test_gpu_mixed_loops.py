"""Mixed-precision PPCG in loops (many outer iterations a launch, the inner steps'
arrays in shared memory) against the same solve launched pass by pass: the same
operations on the same values and sums in the same order, so equal bit for bit.

Sizes: ragged in both directions, one tile group a multiprocessor and several,
runs of one to four strips, with all private arrays in shared memory and with
some of them left in L2."""
import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["none", "jac_diag", "jac_block"])
@pytest.mark.parametrize("shape,inner", [((33, 18), 10), ((64, 5), 1), ((250, 131), 2), ((517, 403), 7),
                                         ((1030, 411), 10), ((1201, 997), 3), ((1400, 1350), 4)])
def test_mixed_loop_equals_single_passes(precond, shape, inner):
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=2, tl_max_iters=25, tl_use_cg=False,
                           tl_use_ppcg=True, tl_ppcg_inner_steps=inner, tl_ch_cg_presteps=7, tl_ch_cg_epslim=1.0e10,
                           tl_preconditioner_type=precond, tl_precision="mixed")
    got = {}
    for loop in (True, False):
        with tl.Chunk(tl.parse_deck(deck)) as ch:
            if not loop:  # one kernel a step: never the loop
                ch.set_inner_fusion(1)
            ch.start()
            infos = [ch.timestep() for _ in range(2)]
            got[loop] = ([(i["iterations"], i["error"]) for i in infos],
                         {n: ch.interior(n).copy() for n in ("u", "p", "r", "z", "w", "energy1")})
    assert got[True][0] == got[False][0]
    for n, a in got[True][1].items():
        assert np.array_equal(a, got[False][1][n]), (n, int((a != got[False][1][n]).sum()))
