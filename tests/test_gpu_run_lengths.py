"""Runs of two lengths (fields with more than eight strips a run: as many bands
of strips as the device has warps for): every strip is in one run, and the
fused passes give the bits of the reference-named entry points.

Sizes: bands that differ, also with one longer or shorter band only and with a
cut last strip; few columns and many rows; a field that the loops still take."""
import ctypes as C

import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu

SOLVERS = {
    "cg": ({}, ("u", "p", "r", "z", "w", "energy1")),
    "cheby": ({"tl_use_cg": False, "tl_use_chebyshev": True, "tl_ch_cg_presteps": 4, "tl_ch_cg_epslim": 1.0e10},
              ("u", "p", "r", "w", "energy1")),
    "ppcg": ({"tl_use_cg": False, "tl_use_ppcg": True, "tl_ch_cg_presteps": 4, "tl_ch_cg_epslim": 1.0e10,
              "tl_ppcg_inner_steps": 3}, ("u", "p", "r", "z", "w", "sd", "rtemp", "utemp", "r_store", "energy1")),
    "jacobi": ({"tl_use_cg": False, "tl_use_jacobi": True}, ("u", "energy1")),
}


@pytest.mark.parametrize("shape", [(2300, 2101), (2500, 2403), (2500, 2201), (33, 80001), (32, 78000)])
@pytest.mark.parametrize("solver,precond", [("cg", "none"), ("cg", "jac_diag"), ("cg", "jac_block"),
                                            ("cheby", "jac_block"), ("ppcg", "jac_block"), ("jacobi", "none")])
def test_every_strip_is_in_one_run(shape, solver, precond):
    kw, names = SOLVERS[solver]
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=1, tl_max_iters=9,
                           tl_preconditioner_type=precond, **kw)
    lib = tl.load()
    cfg = tl.parse_deck(deck)
    with tl.Chunk(cfg) as ch:
        vol, mass, ie, temp = ch.start()
        assert abs(vol - 100.0) <= 1e-11 * 100.0  # 10 x 10, every cell once
        rho, e = ch.interior("density"), ch.interior("energy0")
        cell = 100.0 / (shape[0] * shape[1])
        assert abs(mass - rho.sum() * cell) <= 1e-11 * mass
        assert abs(ie - (rho * e).sum() * cell) <= 1e-11 * ie
        info = ch.timestep()
        fields = {n: ch.interior(n).copy() for n in names}
    recs, _ = tl.run_deck(deck, legacy_abi=True)
    assert (info["iterations"], info["error"]) == (recs[1]["iterations"], recs[1]["error"])
    a = np.empty((cfg.y_cells + 2, cfg.x_cells + 2))
    for n in names:
        assert lib.tl_get_field(C.c_void_p(lib.tl_default_chunk()), tl.FIELDS[n], a.ctypes.data) == 0
        assert np.array_equal(a[1:-1, 1:-1], fields[n]), n
