"""The meetings of the loop kernels' thread blocks (many iterations a launch)."""
import threading

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


# method -> deck settings, fields that the loops and the passes leave equal bit for bit
PP = {"tl_use_cg": False, "tl_use_ppcg": True, "tl_ch_cg_presteps": 7, "tl_ch_cg_epslim": 1.0e10,
      "tl_ppcg_inner_steps": 5}
METHODS = {
    "cg": ({}, ("u", "p", "r", "z", "w", "energy1")),
    "cheby": ({"tl_use_cg": False, "tl_use_chebyshev": True, "tl_ch_cg_presteps": 7, "tl_ch_cg_epslim": 1.0e10},
              ("u", "p", "r", "w", "energy1")),
    "ppcg": (PP, ("u", "p", "r", "z", "w", "sd", "rtemp", "utemp", "r_store", "energy1")),
    "jacobi": ({"tl_use_cg": False, "tl_use_jacobi": True}, ("u", "energy1")),
    "mixed cg": ({"tl_precision": "mixed", "tl_eps": 1e-9}, ("u", "r", "energy1")),
    "mixed ppcg": (dict(PP, tl_precision="mixed"), ("u", "p", "r", "z", "w", "energy1")),
}
CASES = [(m, p) for m in METHODS for p in ("none", "jac_diag", "jac_block")
         if not (m == "mixed cg" and p == "jac_block") and not (m == "jacobi" and p != "none")]


def _deck(method, precond, shape, max_iters=41):
    return decks.make_deck(x_cells=shape[0], y_cells=shape[1], end_step=2, tl_preconditioner_type=precond,
                           **dict({"tl_max_iters": max_iters}, **METHODS[method][0]))


def _set(ch, start_wait=-1, wait=-1, iters=0):
    assert tl.load().tl_test_loops(ch._h, start_wait, wait, iters) == 0


def _solve(ch, method, steps=2):
    before = ch.kernel_launches
    infos = [ch.timestep() for _ in range(steps)]
    return ([(i["status"], i["iterations"], i["error"]) for i in infos],
            {n: ch.interior(n).copy() for n in METHODS[method][1]}, ch.kernel_launches - before)


def _run(deck, method, **limits):
    with tl.Chunk(tl.parse_deck(deck)) as ch:
        _set(ch, **limits)
        ch.start()
        return _solve(ch, method)


def _same(a, b):
    assert a[0] == b[0]
    for n in a[1]:
        assert np.array_equal(a[1][n], b[1][n]), (n, int((a[1][n] != b[1][n]).sum()))


@pytest.mark.parametrize("method,precond", CASES)
@pytest.mark.parametrize("shape,iters", [((33, 18), 1), ((250, 131), 3), ((700, 333), 16), ((1201, 997), 5)])
def test_launch_boundaries_carry_the_solve_on(method, precond, shape, iters):
    """few and odd numbers of iterations a launch, so that a phase takes many
    launches and either of two buffers holds the iterate where they meet"""
    deck = _deck(method, precond, shape)
    few = _run(deck, method, iters=iters)
    usual = _run(deck, method)
    _same(few, usual)
    if usual[0][0][1] > 2 * iters + 8:
        assert few[2] > usual[2]


@pytest.mark.parametrize("method,precond", CASES)
@pytest.mark.parametrize("start_wait,iters", [(-2, 0), (0, 0), (2000, 3), (4000, 1)])
def test_blocks_that_start_late(method, precond, start_wait, iters):
    """Thread blocks that do not wait for the others' start (or are told that one
    is missing): the launch does nothing and the solve goes on in passes (also in the middle of a phase), to
    the same bits.  The second timestep is the one looked at: the first of mixed
    PPCG begins with FP32 CG iterations, whose loop and passes add in different
    orders.  Mixed CG, for the same reason, against its passes launched one by one."""
    mixed_cg = method == "mixed cg"
    if mixed_cg and start_wait >= 0:
        pytest.skip("some launches in loops and some in passes: no bits to compare with")
    deck = _deck(method, precond, (700, 333))

    def second_step(late):
        with tl.Chunk(tl.parse_deck(deck)) as ch:
            ch.start()
            ch.timestep()
            if late:
                _set(ch, start_wait=start_wait, iters=iters)
            elif mixed_cg:
                assert tl.load().tl_set_profiling(ch._h, 1) == 0
            return _solve(ch, method, steps=1)

    usual, late = second_step(False), second_step(True)
    if start_wait < 0 and not mixed_cg:  # (else all blocks may start within one another's first look)
        assert late[2] > usual[2]  # passes
    _same(late, usual)


@pytest.mark.parametrize("method,precond", CASES)
@pytest.mark.parametrize("wait", [0, 1000, 2500, 4000, 20000])
def test_wait_that_runs_out_is_an_error(method, precond, wait):
    """A meeting's limit that is too short, so that blocks give up at any of the
    kernel's meetings: the solve returns TL_ERR_CUDA (or its usual result, if
    no wait was that long), and the next one is as usual."""
    deck = _deck(method, precond, (250, 131))
    with tl.Chunk(tl.parse_deck(deck)) as ch:
        ch.start()
        usual = _solve(ch, method)
        for _ in range(3):
            _set(ch, wait=wait)
            ch.start()
            try:
                got = _solve(ch, method)
            except tl.TeaLeafError as e:
                assert e.code == tl.TL_ERR_CUDA and "gave up waiting" in str(e)
            else:
                assert wait > 0
                _same(got, usual)
            _set(ch)
            ch.start()
            _same(_solve(ch, method), usual)


@pytest.mark.parametrize("a,b", [(("cg", "jac_diag"), ("mixed ppcg", "jac_block")),
                                 (("cheby", "jac_block"), ("mixed cg", "jac_diag")),
                                 (("ppcg", "jac_block"), ("cg", "none"))])
def test_two_chunks_on_two_threads(a, b):
    """each with its own stream: their loop kernels take turns on the device"""
    jobs = [(m, _deck(m, p, (1030, 411))) for m, p in (a, b)]
    usual = [_run(deck, m) for m, deck in jobs]
    got = [[], []]

    def work(k):
        m, deck = jobs[k]
        for _ in range(4):
            got[k].append(_run(deck, m))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(got[k]) == 4
        for g in got[k]:
            _same(g, usual[k])
