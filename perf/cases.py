"""The workloads that the framework is measured on.

A solve case is a heat-conduction problem on a 10 x 10 domain (dt 0.004) run
through the chunk API, in one of two ways:
  flow "host"  the state lives in the caller: density and energy go in from
               page-locked arrays, one implicit solve, energy comes back (a
               hydrodynamics code that calls the conduction step);
  flow "run"   a fresh run of a deck: start, `steps` timesteps, the field
               summary, and the final energy and temperature fields.
A deck case runs the whole main program on a tea.in text.  A conv case is one
residual layer of the warm-start network, forward and backward.

Two kinds of decks: "standard", the five-state problem of the benchmark decks
with its densities and energies varied by the seed, and "random", 3 to 8
rectangles of density U[0.05, 200] and log-uniform energy over a background
drawn the same way (milder contrasts, so fewer iterations).
"""
import ctypes
import functools
import math
import os
import random

import numpy as np
import torch

import tealeaf_cuda_gb300 as tl
from tealeaf_cuda_gb300 import learned

DT = 0.004
MODEL = os.path.join(os.path.dirname(os.path.abspath(tl.__file__)), "warm_start.tlws")


def solve(nx, ny, solver="cg", precond="none", precision="fp64", warm="none", flow="host", steps=1,
          deck="random", eps=1e-15):
    return {"kind": "solve", "nx": nx, "ny": ny, "solver": solver, "precond": precond, "precision": precision,
            "warm": warm, "flow": flow, "steps": steps, "deck": deck, "eps": eps}


def listed():
    return [
        # the smallest calls: a toy deck, where launches and latency are all there is
        dict(solve(48, 40, deck="standard"), name="cg tiny"),
        # the main program on the smallest of the benchmark decks that people time
        {"kind": "deck", "nx": 250, "ny": 250, "precond": "none", "steps": 5, "deck": "standard", "name": "deck 250"},
        # plain CG on the 512 x 512 deck of the project's first configuration
        dict(solve(512, 512, flow="run", steps=2, deck="standard"), name="cg 512"),
        # block-Jacobi CG on a ragged grid called from a host code
        dict(solve(1277, 963, precond="jac_block"), name="cg block ragged"),
        # the FP64 drop-in at the size the four plain methods are compared at
        dict(solve(4096, 4096, precond="jac_diag"), name="cg diag 4096"),
        # Chebyshev after its CG presteps
        dict(solve(1024, 1024, solver="chebyshev", precond="jac_diag", flow="run", deck="standard", eps=1e-10),
             name="chebyshev 1024"),
        # FP64 PPCG with ten inner steps and block-Jacobi strips
        dict(solve(1500, 1100, solver="ppcg", precond="jac_block", flow="run", steps=2), name="ppcg 1500x1100"),
        # the solver a deck gets when it names none
        dict(solve(130, 96, solver="jacobi"), name="jacobi small"),
        # FP32 inner CG inside FP64 refinement
        dict(solve(3000, 2100, precond="jac_diag", precision="mixed"), name="mixed cg 3000x2100"),
        # the mixed-precision method on an ordinary grid, with the increment history
        dict(solve(1400, 1000, solver="ppcg", precond="jac_block", precision="mixed", warm="prev", flow="run",
                   steps=3, deck="standard"), name="mixed ppcg 1400x1000"),
        # the headline method at the headline size, with the learned warm start
        dict(solve(8192, 8192, solver="ppcg", precond="jac_block", precision="mixed", warm="learned", flow="run",
                   steps=2), name="mixed ppcg 8192"),
        # one residual layer of the network as its trainer runs it, forward and backward
        {"kind": "conv", "batch": 32, "height": 144, "width": 144, "name": "conv layer"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi):  # hi x hi cells at most; sides up to a factor of two apart
        n, a = size(lo, hi), math.exp(rng.uniform(-0.35, 0.35))
        return max(8, min(hi, int(n * a))), max(8, min(hi, int(n / a)))

    family = rng.choice(["cg", "cg", "deck", "chebyshev", "ppcg", "jacobi", "mixed cg", "mixed ppcg", "mixed ppcg",
                         "conv"])
    precond = rng.choice(["none", "jac_diag", "jac_block"])
    flow = rng.choice(["host", "run"])
    if family == "cg":
        nx, ny = grid(16, 3000)
        deck = rng.choice(["standard", "random"]) if nx * ny < 800 * 800 else "random"
        return solve(nx, ny, precond=precond, flow=flow, deck=deck)
    if family == "deck":
        nx, ny = grid(10, 500)
        return {"kind": "deck", "nx": nx, "ny": ny, "precond": precond, "steps": rng.randint(2, 5),
                "deck": rng.choice(["standard", "random"])}
    if family == "chebyshev":
        nx, ny = grid(64, 1200)
        return solve(nx, ny, solver="chebyshev", precond=precond, flow="run", eps=1e-10)
    if family == "ppcg":
        nx, ny = grid(64, 1800)
        return solve(nx, ny, solver="ppcg", precond=precond, flow="run", steps=rng.randint(1, 2))
    if family == "jacobi":
        nx, ny = grid(24, 200)
        return solve(nx, ny, solver="jacobi", flow=flow)
    if family == "mixed cg":
        nx, ny = grid(96, 4000)
        return solve(nx, ny, precond=rng.choice(["none", "jac_diag"]), precision="mixed", flow=flow)
    if family == "mixed ppcg":
        nx, ny = grid(96, 5000)
        return solve(nx, ny, solver="ppcg", precond=precond, precision="mixed",
                     warm=rng.choice(["none", "prev", "learned"]), flow="run", steps=rng.randint(1, 3))
    return {"kind": "conv", "batch": size(1, 48), "height": size(48, 200), "width": 16 * size(3, 12)}


# ------------------------------------------------------------------- decks

def states_of(case, seed):
    """[(density, energy, (xmin, xmax, ymin, ymax) or None), ...]"""
    rng = random.Random(seed)
    if case["deck"] == "standard":
        base = [(100.0, 1e-4, None), (0.1, 25.0, (0.0, 1.0, 1.0, 2.0)), (0.1, 0.1, (1.0, 6.0, 1.0, 2.0)),
                (0.1, 0.1, (5.0, 6.0, 1.0, 8.0)), (0.1, 0.1, (5.0, 10.0, 7.0, 8.0))]
        return [(d * rng.uniform(0.9, 1.1), e * rng.uniform(0.5, 2.0), r) for d, e, r in base]

    def material():
        return rng.uniform(0.05, 200.0), math.exp(rng.uniform(math.log(1e-4), math.log(50.0)))

    out = [material() + (None,)]
    for _ in range(rng.randint(3, 8)):
        d, e = material()
        x0, x1 = sorted((rng.uniform(0.0, 10.0), rng.uniform(0.0, 10.0)))
        y0, y1 = sorted((rng.uniform(0.0, 10.0), rng.uniform(0.0, 10.0)))
        out.append((d, e, (x0, max(x1, x0 + 0.3), y0, max(y1, y0 + 0.3))))
    return out


def deck_text(case, seed):
    lines = ["*tea"]
    for k, (d, e, rect) in enumerate(states_of(case, seed)):
        lines.append("state %d density=%r energy=%r%s" % (k + 1, d, e, " \\" if rect else ""))
        if rect:  # a deck line is read up to its 100th character: go on on the next ones
            lines += ["geometry=rectangle xmin=%r xmax=%r \\" % rect[:2], "ymin=%r ymax=%r" % rect[2:]]
    solver = case.get("solver", "cg")
    lines += ["x_cells=%d" % case["nx"], "y_cells=%d" % case["ny"], "xmin=0.0", "ymin=0.0", "xmax=10.0", "ymax=10.0",
              "initial_timestep=%r" % DT, "end_step=%d" % case["steps"], "end_time=100.0", "summary_frequency=1",
              "tl_max_iters=10000", "tl_use_%s" % solver, "tl_preconditioner_type %s" % case["precond"],
              "tl_eps=%r" % case.get("eps", 1e-15)]
    if solver in ("chebyshev", "ppcg"):
        lines += ["tl_ch_cg_presteps=%d" % (20 if solver == "chebyshev" else 10), "tl_ch_cg_epslim=1.0e10"]
    if solver == "ppcg":
        lines.append("tl_ppcg_inner_steps=10")
    if case.get("precision") == "mixed":
        lines.append("tl_precision mixed")
    if case.get("warm", "none") != "none":
        lines.append("tl_warm_start %s" % case["warm"])
    return "\n".join(lines + ["*endtea"]) + "\n"


# ------------------------------------------------------------ prepare, run

def pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    if case["kind"] == "conv":
        return prepare_conv(case, seed)
    text = deck_text(case, seed)
    if case["kind"] == "deck":
        return {"case": case, "text": text}
    ch = tl.Chunk(tl.parse_deck(text))
    st = {"case": case, "chunk": ch, "energy": pinned(ch.shape)}
    if case["warm"] == "learned":
        p = np.ascontiguousarray(learned.load_model(MODEL), dtype=np.float32)
        if tl.load().tl_set_warm_start_model(ch._h, ctypes.c_void_p(p.ctypes.data), p.size) != 0:
            raise RuntimeError(tl.last_error())
    if case["flow"] == "host":
        ch.start()
        st["density_in"] = ch.get_field("density", out=pinned(ch.shape))
        st["energy_in"] = ch.get_field("energy1", out=pinned(ch.shape))
    else:
        st["u"] = pinned(ch.shape)
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "conv":
        return run_conv(state)
    if case["kind"] == "deck":
        recs, _ = tl.run_deck(state["text"], max_records=16)
        return {"summary": np.array([[r[k] for k in ("vol", "mass", "ie", "temp")] for r in recs[1:]])}
    ch = state["chunk"]
    if case["flow"] == "host":
        ch.set_field("density", state["density_in"])
        ch.set_field("energy1", state["energy_in"])
        ch.timestep()
        return {"energy": inner(ch.get_field("energy1", out=state["energy"]))}
    ch.start()
    for _ in range(case["steps"]):
        ch.timestep()
    summary = np.array(ch.field_summary())
    return {"energy": inner(ch.get_field("energy1", out=state["energy"])),
            "u": inner(ch.get_field("u", out=state["u"])), "summary": summary}


def inner(a):
    return a[1:-1, 1:-1]


# ------------------------------------------------------------------- exact

def exact(case, seed):
    if case["kind"] == "conv":
        return exact_conv(case, seed)
    rho, e, dx, dy = exact_state(case, seed)
    kx, ky, inv = exact_operator(rho, dx, dy)
    sums = []
    for _ in range(case["steps"]):
        u = exact_solve(kx, ky, inv, e * rho)
        e = u / rho
        cell = torch.full_like(rho, dx * dy)
        sums.append([float(v) for v in (cell.sum(), (cell * rho).sum(), (cell * rho * e).sum(), (cell * rho * u).sum())])
    if case["kind"] == "deck":
        return {"summary": np.array(sums)}
    if case["flow"] == "host":
        return {"energy": e}
    return {"energy": e, "u": u, "summary": np.array(sums[-1])}


def exact_state(case, seed):
    """density and energy of the deck's states on the cells that they touch"""
    nx, ny = case["nx"], case["ny"]
    dx, dy = 10.0 / float(np.float32(nx)), 10.0 / float(np.float32(ny))
    at = dict(dtype=torch.float64, device="cuda")
    x0, x1 = dx * torch.arange(nx, **at), dx * torch.arange(1, nx + 1, **at)
    y0, y1 = dy * torch.arange(ny, **at), dy * torch.arange(1, ny + 1, **at)
    rho, e = torch.empty((ny, nx), **at), torch.empty((ny, nx), **at)
    for d, en, rect in states_of(case, seed):
        if rect is None:
            rho.fill_(d)
            e.fill_(en)
            continue
        hit = ((y1 >= rect[2] + dy / 100.0) & (y0 < rect[3] - dy / 100.0))[:, None] & \
            ((x1 >= rect[0] + dx / 100.0) & (x0 < rect[1] - dx / 100.0))[None, :]
        rho[hit] = d
        e[hit] = en
    return rho, e, dx, dy


def exact_operator(rho, dx, dy):
    """conductivities of the inner faces, and 1 / diagonal"""
    kx = DT / (dx * dx) * (rho[:, :-1] + rho[:, 1:]) / (2.0 * rho[:, :-1] * rho[:, 1:])
    ky = DT / (dy * dy) * (rho[:-1] + rho[1:]) / (2.0 * rho[:-1] * rho[1:])
    diag = torch.ones_like(rho)
    diag[:, :-1] += kx
    diag[:, 1:] += kx
    diag[:-1] += ky
    diag[1:] += ky
    return kx, ky, 1.0 / diag


def exact_apply(kx, ky, x):
    y = x.clone()
    f = kx * (x[:, 1:] - x[:, :-1])
    y[:, :-1] -= f
    y[:, 1:] += f
    f = ky * (x[1:] - x[:-1])
    y[:-1] -= f
    y[1:] += f
    return y


def exact_solve(kx, ky, inv, b):
    """conjugate gradients with the diagonal, restarted from the true residual until it no longer falls"""
    x, last = b.clone(), math.inf
    for _ in range(6):
        r = b - exact_apply(kx, ky, x)
        norm = float(r.norm())
        if not norm or norm > 0.25 * last:
            break
        last = norm
        z = r * inv
        p, d, rz = z.clone(), torch.zeros_like(b), (r * z).sum()
        for k in range(20000):
            w = exact_apply(kx, ky, p)
            alpha = rz / (p * w).sum()
            d += alpha * p
            r -= alpha * w
            if k % 16 == 15 and float(r.norm()) < 1e-12 * norm:
                break
            z = r * inv
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        x = x + d
    return x


# -------------------------------------------------------------- conv layer

CH = 32  # channels of the network's residual layers


@functools.lru_cache(maxsize=1)
def conv_inputs(batch, height, width, seed):
    """activations, weights and the gradient of the output: values as the trained network has them"""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def field(scale):
        t = torch.zeros((batch, height + 2, width + 2, CH), dtype=torch.bfloat16, device="cuda")
        t[:, 1:-1, 1:-1] = scale * torch.randn((batch, height, width, CH), generator=g, device="cuda")
        return t

    w = math.sqrt(2.0 / (9 * CH)) * torch.randn((9, CH, CH), generator=g, device="cuda")
    w = w.bfloat16().float()  # exact in the layer's own type
    b = 0.1 * torch.randn(CH, generator=g, device="cuda")
    return field(1.0), w, b, field(0.01)


def prepare_conv(case, seed):
    x, w, b, dout = conv_inputs(case["batch"], case["height"], case["width"], seed)
    lib = tl.load()
    shape = (case["batch"], case["height"], case["width"])
    st = {"case": case, "x": x.clone(), "b": b.clone(), "dout": dout.clone(), "lib": lib}
    for k in ("out", "pre", "dpre", "dx"):
        st[k] = torch.zeros_like(x)
    st["wf"], st["wb"] = (torch.zeros(9 * CH * CH, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    n = lib.tl_nn_wgrad_partial_floats(CH, CH, *shape, 8)
    st["partial"] = torch.zeros(int(n), device="cuda")
    st["dw"], st["db"] = torch.zeros((9, CH, CH), device="cuda"), torch.zeros(CH, device="cuda")
    check(lib, lib.tl_nn_pack(ptr(w), ptr(st["wf"]), ptr(st["wb"]), CH, CH, stream()))
    torch.cuda.synchronize()
    conv_inputs.cache_clear()
    return st


def run_conv(s):
    lib, case = s["lib"], s["case"]
    shape = (case["batch"], case["height"], case["width"])
    q = stream()
    check(lib, lib.tl_nn_conv(1, CH, CH, ptr(s["x"]), ptr(s["wf"]), ptr(s["b"]), ptr(s["x"]), ptr(s["out"]),
                              ptr(s["pre"]), None, *shape, q))
    check(lib, lib.tl_nn_gelu_backward(ptr(s["dout"]), ptr(s["pre"]), ptr(s["dpre"]), CH, *shape, q))
    check(lib, lib.tl_nn_wgrad(ptr(s["dpre"]), ptr(s["x"]), CH, CH, ptr(s["partial"]), ptr(s["dw"]), ptr(s["db"]),
                               *shape, 8, q))
    check(lib, lib.tl_nn_conv(3, CH, CH, ptr(s["dpre"]), ptr(s["wb"]), None, ptr(s["dout"]), ptr(s["dx"]), None, None,
                              *shape, q))
    return {k: s[k] for k in ("out", "pre", "dpre", "dx", "dw", "db")}


def check(lib, rc):
    if rc != 0:
        raise RuntimeError(lib.tl_last_error().decode())


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def exact_conv(case, seed):
    x, w, b, dout = (t.double() for t in conv_inputs(case["batch"], case["height"], case["width"], seed))
    conv_inputs.cache_clear()
    h, v = case["height"], case["width"]

    def taps(t):
        return [t[:, dy:dy + h, dx:dx + v] for dy in range(3) for dx in range(3)]

    def padded(t):
        out = torch.zeros_like(x)
        out[:, 1:-1, 1:-1] = t
        return out

    pre = sum(t @ w[k].T for k, t in enumerate(taps(x))) + b
    c = math.sqrt(2.0 / math.pi)
    th = torch.tanh(c * (pre + 0.044715 * pre ** 3))
    out = x[:, 1:-1, 1:-1] + 0.5 * pre * (1.0 + th)
    grad = 0.5 * (1.0 + th) + 0.5 * pre * (1.0 - th * th) * c * (1.0 + 3 * 0.044715 * pre * pre)
    dpre = dout[:, 1:-1, 1:-1] * grad
    dx = dout[:, 1:-1, 1:-1] + sum(t @ w[8 - k] for k, t in enumerate(taps(padded(dpre))))
    flat = dpre.reshape(-1, CH)
    dw = torch.stack([flat.T @ t.reshape(-1, CH) for t in taps(x)])
    return {"out": padded(out), "pre": padded(pre), "dpre": padded(dpre), "dx": padded(dx), "dw": dw,
            "db": flat.sum(0)}


# -------------------------------------------------------------------- work

def work(case):
    if case["kind"] == "conv":
        cells = case["batch"] * case["height"] * case["width"]
        # forward: x in, out and pre out; backward: x, pre and dout in, dpre and dx out
        return {"bytes": cells * CH * 2 * 8, "flops": cells * 3 * 2 * 9 * CH * CH}
    cells = case["nx"] * case["ny"]
    # Krylov iterations to tl_eps go with the square root of the operator's
    # condition number, 1 + 8 dt / dx^2 / density; 10 and 0.1 are typical
    # 1 / density of the thin materials of the two kinds of decks
    k = 10.0 if case["deck"] == "standard" else 0.1
    cond = 1.0 + 8.0 * DT * cells / 100.0 * k
    its = max(10.0, 12.0 * math.sqrt(cond))
    solver, precond = case.get("solver", "cg"), case["precond"]
    pc = {"none": 0, "jac_diag": 8, "jac_block": 24}[precond]
    if case.get("precision") == "mixed" and solver == "ppcg":
        # outer: u, p, w = A p in one sweep, r, the two dot products; the ten
        # FP32 inner steps in two sweeps of five
        its, per, ops = its / 10, 72 + 24 + 24 + 72, 30 + 10 * 18
    elif case.get("precision") == "mixed":
        # FP32: u, p, w = A p in one sweep, r and z in the other; about twice the iterations
        its, per, ops = its * 2, 52, 22
    elif solver == "cg":
        # two sweeps: z, p, u, Kx, Ky, diagonal in, p, u, w out; w, r, preconditioner in, r, z out
        its, per, ops = its, 72 + 24 + (8 + pc if pc else 0), 22 + pc / 4
    elif solver == "chebyshev":
        # u, u0, p, Kx, Ky, diagonal, preconditioner in; u, p, r out
        its, per, ops = its * 1.5, 72 + pc, 20 + pc / 4
    elif solver == "ppcg":
        # each inner step: sd, rtemp, utemp in and out, operator and preconditioner in
        its, per, ops = its / 10, 10 * (72 + pc) + 72 + 24 + 24, 30 + 10 * (18 + pc / 4)
    else:
        its, per, ops = cond * 4, 40, 12  # Jacobi: u, u0, Kx, Ky in, u out
    return {"bytes": case["steps"] * cells * its * per, "flops": case["steps"] * cells * its * ops}
