"""The warm start's projection over one to eight increments against the same
projection in numpy: random energies each step make increments that are
independent of one another, so none is dropped.

The start's residual over the plain start's, which the solve reports, follows from
the coefficients.  Bound: 1e-8, for sums of some 1e3 FP64 values (1e-13) and Gram
matrices of condition numbers up to 1e4, ten times over."""
import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("projection", [tl.WARM_PROJ_ENERGY, tl.WARM_PROJ_RESIDUAL])
@pytest.mark.parametrize("history,shape", [(8, (37, 30)), (3, (64, 9))])
def test_projection_over_every_number_of_increments(projection, history, shape):
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=12, tl_max_iters=3,
                           tl_preconditioner_type="jac_diag").replace("*endtea", "tl_warm_start prev\n*endtea")
    rng = np.random.default_rng(history)
    with tl.Chunk(tl.parse_deck(deck)) as ch:
        ch.set_warm_start_options(history, projection)
        ch.start()
        h = ch.cfg.halo_depth
        rho = ch.interior("density").copy()
        increments, before = [], None
        for step in range(11):
            e = ch.get_field("energy1")
            e[h:-h, h:-h] = rng.uniform(0.1, 10.0, size=rho.shape)
            ch.set_field("energy1", e)
            u = e[h:-h, h:-h] * rho
            info = ch.timestep()
            if before is not None:
                increments = ([u - before] + increments)[:history]
            before = u
            if not increments:
                assert info["warm_used"] == 0
                continue
            kx, ky = ch.get_field("kx"), ch.get_field("ky")
            w, s = kx[h:-h, h:-h], ky[h:-h, h:-h]
            east, north = kx[h:-h, h + 1:kx.shape[1] - h + 1], ky[h + 1:ky.shape[0] - h + 1, h:-h]

            def apply(v):
                p = np.pad(v, 1)
                return ((1 + w + s + east + north) * v - w * p[1:-1, :-2] - east * p[1:-1, 2:] - s * p[:-2, 1:-1]
                        - north * p[2:, 1:-1])

            r0 = u - apply(u)
            D = np.stack([d.ravel() for d in increments], 1)
            AD = np.stack([apply(d).ravel() for d in increments], 1)
            left = D if projection == tl.WARM_PROJ_ENERGY else AD
            c = np.linalg.solve(left.T @ AD, left.T @ r0.ravel())
            want = np.linalg.norm(r0.ravel() - AD @ c) / np.linalg.norm(r0)
            assert info["warm_used"] == 1
            assert info["warm_ratio"] == pytest.approx(want, rel=1e-8), (step, len(increments))
