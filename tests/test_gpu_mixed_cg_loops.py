"""The FP32 CG iterations of the mixed-precision solves in loops (many iterations a
launch) against the same iterations launched pass by pass, whose sums run in
another order.

Both end with an FP64 residual below eps times the initial one, and the
operator's smallest eigenvalue is 1 (1 plus a sum of non-negative faces), so the
two solutions differ by 2 eps |r0| at most (and FP64 rounding, 1e-13 |u|).

Sizes: one warp's run of rows and many, columns that end within a lane's four,
within a warp and with it, more runs than multiprocessors, and the largest runs
that the loop takes."""
import ctypes as C

import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,precond", [("cg", "none"), ("cg", "jac_diag"), ("ppcg", "none"),
                                            ("ppcg", "jac_diag"), ("ppcg", "jac_block")])
@pytest.mark.parametrize("shape", [(9, 8), (127, 5), (128, 4), (130, 37), (33, 700), (517, 403), (1400, 1201)])
def test_mixed_cg_loop_and_passes_reach_the_same_solution(solver, precond, shape):
    lib = tl.load()
    lib.tl_set_profiling.argtypes = [C.c_void_p, C.c_int]
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=1, tl_max_iters=4000, tl_eps=1e-9,
                           tl_use_cg=solver == "cg", tl_use_ppcg=solver == "ppcg", tl_ch_cg_presteps=12,
                           tl_preconditioner_type=precond, tl_precision="mixed")
    got = []
    for passes in (0, 1):
        with tl.Chunk(tl.parse_deck(deck)) as ch:
            lib.tl_set_profiling(ch._h, passes)  # one kernel at a time
            ch.start()
            before = ch.kernel_launches
            info = ch.timestep()
            got.append((ch.interior("u").copy(), info, ch.kernel_launches - before))
    (u, a, few), (v, b, many) = got
    assert a["status"] == b["status"] == 0 and a["iterations"] > 2
    if solver == "cg" and a["iterations"] > 10:
        assert few < many
    bound = 2e-9 * b["initial_residual"] + 1e-13 * np.linalg.norm(v)
    assert np.linalg.norm(u - v) <= bound
