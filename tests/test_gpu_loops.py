"""The device-resident FP64 solves (fused passes; many iterations a launch)
against the reference-named entry points, one piece of an iteration a call:
the same operations on the same values in the same order, so every field and
every number of the solve is equal bit for bit.

Sizes: one warp's columns and a strip, ragged in both directions; one tile
group a multiprocessor, several, several rounds of them; runs of more than one
strip; and a size above which the passes are launched one by one."""
import ctypes as C

import numpy as np
import pytest

import tealeaf_cuda_gb300 as tl
from tests import decks

pytestmark = pytest.mark.gpu

SOLVERS = {
    "cg": {"tl_use_cg": True},
    "cheby": {"tl_use_cg": False, "tl_use_chebyshev": True, "tl_ch_cg_presteps": 7, "tl_ch_cg_epslim": 1.0e10},
    "ppcg": {"tl_use_cg": False, "tl_use_ppcg": True, "tl_ch_cg_presteps": 7, "tl_ch_cg_epslim": 1.0e10,
             "tl_ppcg_inner_steps": 5},
    "jacobi": {"tl_use_cg": False, "tl_use_jacobi": True},
}
FIELDS = {"cg": ("u", "p", "r", "z", "w", "energy1"), "cheby": ("u", "p", "r", "w", "energy1"),
          "ppcg": ("u", "p", "r", "z", "w", "sd", "rtemp", "utemp", "r_store", "energy1"),
          "jacobi": ("u", "energy1")}
SHAPES = [(12, 11), (33, 3), (31, 18), (64, 5), (250, 131), (517, 403), (1030, 411), (1201, 997)]


def _field(lib, h, cfg, name):
    a = np.empty((cfg.y_cells + 2 * cfg.halo_depth, cfg.x_cells + 2 * cfg.halo_depth))
    assert lib.tl_get_field(h, tl.FIELDS[name], a.ctypes.data) == 0
    hd = cfg.halo_depth
    return a[hd:-hd, hd:-hd]


def _run(deck, solver, steps, profiling=False):
    lib = tl.load()
    cfg = tl.parse_deck(deck)
    with tl.Chunk(cfg) as ch:
        ch.start()
        if profiling:
            assert lib.tl_set_profiling(ch._h, 1) == 0
        infos = [ch.timestep() for _ in range(steps)]
        return infos, {n: _field(lib, ch._h, cfg, n).copy() for n in FIELDS[solver]}


def _same(a, b, what):
    for n in a:
        bad = np.argwhere(a[n] != b[n])
        assert bad.size == 0, f"{what} {n}: {len(bad)} cells differ, first {bad[0]}"


@pytest.mark.parametrize("precond", ["none", "jac_diag", "jac_block"])
@pytest.mark.parametrize("solver", list(SOLVERS))
@pytest.mark.parametrize("shape", SHAPES)
def test_loops_equal_reference_entry_points(solver, precond, shape):
    steps = 2
    deck = decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=steps, tl_max_iters=41,
                           tl_preconditioner_type=precond, **SOLVERS[solver])
    infos, fields = _run(deck, solver, steps)
    recs, _ = tl.run_deck(deck, legacy_abi=True)
    lib = tl.load()
    cfg = tl.parse_deck(deck)
    slow = {n: _field(lib, C.c_void_p(lib.tl_default_chunk()), cfg, n).copy() for n in FIELDS[solver]}
    assert [i["iterations"] for i in infos] == [r["iterations"] for r in recs[1:]]
    assert [i["error"] for i in infos] == [r["error"] for r in recs[1:]]
    _same(fields, slow, (solver, precond, shape))


@pytest.mark.parametrize("precond", ["none", "jac_diag", "jac_block"])
@pytest.mark.parametrize("solver", list(SOLVERS))
def test_loops_equal_single_passes(solver, precond):
    """a size that takes the loop, against the same passes launched one by one (per-kernel timing)"""
    deck = decks.make_deck(x_cells=700, y_cells=333, end_step=2, tl_max_iters=60, tl_preconditioner_type=precond,
                           **SOLVERS[solver])
    a, fa = _run(deck, solver, 2)
    b, fb = _run(deck, solver, 2, profiling=True)
    assert [(i["iterations"], i["error"]) for i in a] == [(i["iterations"], i["error"]) for i in b]
    _same(fa, fb, (solver, precond))


@pytest.mark.parametrize("solver,precond", [("cg", "jac_block"), ("cheby", "jac_diag"), ("ppcg", "jac_block"),
                                            ("jacobi", "none")])
def test_long_runs_equal_reference_entry_points(solver, precond):
    """runs of more than eight strips: graphs of single passes"""
    deck = decks.make_deck(x_cells=2400, y_cells=2301, end_step=1, tl_max_iters=24, tl_preconditioner_type=precond,
                           **SOLVERS[solver])
    infos, fields = _run(deck, solver, 1)
    recs, _ = tl.run_deck(deck, legacy_abi=True)
    lib = tl.load()
    slow = {n: _field(lib, C.c_void_p(lib.tl_default_chunk()), tl.parse_deck(deck), n).copy() for n in FIELDS[solver]}
    assert infos[0]["error"] == recs[1]["error"]
    _same(fields, slow, (solver, precond))
