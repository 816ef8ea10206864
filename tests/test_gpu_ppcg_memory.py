"""FP64 PPCG on a chunk that filled the memory: the fused passes' second buffer
of sd, allocated by the first solve, is not there, and the solve runs the
single pieces, which need none and give the same bits."""
import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu

FIELDS = ("u", "p", "r", "z", "w", "sd", "rtemp", "utemp", "r_store", "energy1")


@pytest.mark.parametrize("precond", ["none", "jac_block"])
@pytest.mark.parametrize("inner", [4, 5])
def test_no_memory_for_the_second_buffer(precond, inner):
    deck = decks.make_deck(x_cells=130, y_cells=75, end_step=3, tl_max_iters=60, tl_use_cg=False, tl_use_ppcg=True,
                           tl_ppcg_inner_steps=inner, tl_ch_cg_presteps=7, tl_ch_cg_epslim=1.0e10,
                           tl_preconditioner_type=precond)
    lib = tl.load()
    got = []
    for fail in (0, 1):
        with tl.Chunk(tl.parse_deck(deck)) as ch:
            ch.start()
            assert lib.tl_test_fail_alloc(fail) == 0
            try:
                infos = [ch.timestep() for _ in range(3)]
            finally:
                lib.tl_test_fail_alloc(0)
            if fail:
                assert tl.last_error() == ""
            got.append(([(i["status"], i["iterations"], i["error"]) for i in infos],
                        {n: ch.interior(n).copy() for n in FIELDS}))
    assert got[0][0] == got[1][0]
    for n in FIELDS:
        assert np.array_equal(got[0][1][n], got[1][1][n]), n
