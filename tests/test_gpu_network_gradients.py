"""The network's convolution, its weight and bias gradients and the GELU gradient
at the sizes where their kernels' tiles end: one 16-pixel group, segments of 64 pixels and
their remainders, partial buffers with room for one block only, buffers that
are not 16-byte aligned.

Reference: the same contraction of the same BF16 values in FP64.  Bound: FP32
accumulation along chains of at most a few hundred additions at these sizes,
300 * 2^-24 < 2e-5 of the sum of the absolute products."""
import ctypes as C

import pytest

import tealeaf_cuda_gb300 as tl

pytestmark = pytest.mark.gpu


def _field(torch, shape, ch, offset, gen):
    """[B][H+2][W+2][ch] BF16 with a zero halo, `offset` elements into its allocation"""
    B, H, W = shape
    n = B * (H + 2) * (W + 2) * ch
    t = torch.zeros(n + 16, dtype=torch.bfloat16, device="cuda")[offset:offset + n].view(B, H + 2, W + 2, ch)
    t[:, 1:-1, 1:-1] = torch.randn((B, H, W, ch), generator=gen, device="cuda")
    return t


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("shape,gpc,offset", [((1, 1, 16), 8, 0), ((1, 3, 64), 4, 0), ((1, 5, 80), 8, 0),
                                              ((2, 7, 144), 8, 0), ((1, 2, 64), 100, 0), ((3, 200, 48), 8, 0),
                                              ((1, 4, 80), 8, 3)])
def test_weight_and_bias_gradients(cin, cout, shape, gpc, offset):
    torch = pytest.importorskip("torch")
    lib = tl.load()
    B, H, W = shape
    gen = torch.Generator(device="cuda").manual_seed(cin + 7 * cout + W)
    d, x = _field(torch, shape, cout, offset, gen), _field(torch, shape, cin, offset, gen)
    part = torch.full((int(lib.tl_nn_wgrad_partial_floats(cin, cout, B, H, W, gpc)) + 64,), 7.0, device="cuda")
    part[-64:] = -5.0
    dw, db = torch.empty((9, cout, cin), device="cuda"), torch.empty(cout, device="cuda")
    rc = lib.tl_nn_wgrad(_p(d), _p(x), cin, cout, _p(part), _p(dw), _p(db), B, H, W, gpc, None)
    assert rc == 0, tl.last_error()
    torch.cuda.synchronize()
    assert bool((part[-64:] == -5.0).all())  # the partial buffer's end is not written over
    dd = d.double()[:, 1:-1, 1:-1].reshape(-1, cout)
    for tap in range(9):
        dy, dx = divmod(tap, 3)
        xs = x.double()[:, dy:dy + H, dx:dx + W].reshape(-1, cin)
        assert bool(((dw[tap].double() - dd.T @ xs).abs() <= 2e-5 * (dd.abs().T @ xs.abs()) + 1e-30).all()), tap
    assert bool(((db.double() - dd.sum(0)).abs() <= 2e-5 * dd.abs().sum(0)).all())


@pytest.mark.parametrize("ch,shape,offset", [(32, (1, 1, 16), 0), (32, (2, 5, 48), 0), (16, (3, 4, 16), 0),
                                             (12, (1, 3, 16), 0), (32, (1, 3, 16), 5)])
def test_gelu_gradient_wide_and_narrow_loads_agree(ch, shape, offset):
    """the 16-byte form and the one-value form give the same bits; the halo stays zero"""
    torch = pytest.importorskip("torch")
    lib = tl.load()
    gen = torch.Generator(device="cuda").manual_seed(ch)
    dh, pre = _field(torch, shape, ch, 0, gen), _field(torch, shape, ch, 0, gen)
    want = torch.zeros_like(dh)
    B, H, W = shape
    # one channel at a time is never a multiple of eight
    flat = lambda t: t.reshape(1, 1, -1, 1)
    n = dh.numel()
    a, b, o = (torch.zeros((1, 3, n + 2, 1), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    a[0, 1, 1:-1, 0], b[0, 1, 1:-1, 0] = dh.reshape(-1), pre.reshape(-1)
    assert lib.tl_nn_gelu_backward(_p(a), _p(b), _p(o), 1, 1, 1, n, None) == 0
    want = o[0, 1, 1:-1, 0].reshape(dh.shape)
    d2, p2 = _field(torch, shape, ch, offset, gen), _field(torch, shape, ch, offset, gen)
    d2.copy_(dh)
    p2.copy_(pre)
    got = torch.zeros(n + 16, dtype=torch.bfloat16, device="cuda")[offset:offset + n].view(dh.shape)
    assert lib.tl_nn_gelu_backward(_p(d2), _p(p2), _p(got), ch, B, H, W, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(got[:, 1:-1, 1:-1], want[:, 1:-1, 1:-1])
    assert float(got[:, 0].abs().sum() + got[:, :, 0].abs().sum()) == 0.0


@pytest.mark.parametrize("cin,cout,mode", [(16, 32, 0), (32, 32, 1), (32, 16, 2), (16, 32, 3), (32, 32, 3)])
@pytest.mark.parametrize("shape", [(1, 1, 16), (1, 7, 16), (2, 3, 112), (1, 2, 128), (2, 4, 48), (1, 9, 256),
                                   (3, 160, 144)])
@pytest.mark.parametrize("with_pre", [True, False])
def test_tensor_memory_conv_tiles(cin, cout, mode, shape, with_pre):
    """tiles of 128 columns by 4 rows across the rows' ends and the image's, one and several a thread block,
    the input itself added (where it has the channels) and another array, against the warp-level kernel: BF16 outputs within one rounding (2^-7), the FP32 head within its sum's rounding; the
    halo and what lies behind the buffers stay as they are"""
    torch = pytest.importorskip("torch")
    lib = tl.load()
    lib.tl_nn_set_conv_kernel.argtypes = [C.c_int]
    B, H, W = shape
    gen = torch.Generator(device="cuda").manual_seed(3 * cin + cout + mode + W)
    x, res = _field(torch, shape, cin, 0, gen), _field(torch, shape, cout, 0, gen)
    if cin == cout and with_pre:
        res = x
    w = (0.2 * torch.randn((9, cout, cin), generator=gen, device="cuda")).bfloat16()
    bias = 0.1 * torch.randn(cout, generator=gen, device="cuda")
    got = {}
    for tc in (1, 0):
        n = B * (H + 2) * (W + 2) * cout
        out, pre = (torch.full((n + 256,), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        head = torch.full((B * H * W + 64,), 5.0, device="cuda")
        out[:n], pre[:n] = 0, 0
        assert lib.tl_nn_set_conv_kernel(tc) == 0
        rc = lib.tl_nn_conv(mode, cin, cout, _p(x), _p(w), _p(bias), _p(res) if mode in (1, 3) else None, _p(out),
                            _p(pre) if with_pre else None, _p(head), B, H, W, None)
        lib.tl_nn_set_conv_kernel(1)
        assert rc == 0, tl.last_error()
        torch.cuda.synchronize()
        assert lib.tl_nn_conv_status() == 0, tl.last_error()
        assert bool((out[n:] == 3.0).all() and (pre[n:] == 3.0).all() and (head[B * H * W:] == 5.0).all())
        got[tc] = [t[:n].float().view(B, H + 2, W + 2, cout) for t in (out, pre)] + [head[:B * H * W]]
        for t in got[tc][:2]:
            assert float(t[:, 0].abs().sum() + t[:, -1].abs().sum() + t[:, :, 0].abs().sum() + t[:, :, -1].abs().sum()) == 0
    for a, b in zip(got[1], got[0]):
        assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-5).all())


def test_gelu_and_its_gradient_against_fp64():
    """through a convolution with zero weights, whose pre-activations are the bias, over the range where the
    function bends, zeros, infinities and NaN.  Bound: BF16 rounding of the result (8 significant bits: 2^-8) and 1e-6 of FP32
    arithmetic (a dozen roundings of values up to 20)"""
    torch = pytest.importorskip("torch")
    lib = tl.load()
    lib.tl_nn_set_conv_kernel.argtypes = [C.c_int]
    inf, nan = float("inf"), float("nan")
    v = torch.cat([torch.linspace(-20, 20, 4001), torch.linspace(-2, 2, 4001),
                   torch.tensor([0.0, -0.0, 1e-30, -1e-30, 1e18, -1e18, inf, -inf, nan])]).cuda()
    v = torch.cat([v, v.new_zeros(-len(v) % 32)])
    x, w = (torch.zeros(s, dtype=torch.bfloat16, device="cuda") for s in ((1, 3, 18, 32), (9, 32, 32)))
    g = lambda u: u / (1 + torch.exp(-2 * (2 / torch.pi) ** 0.5 * (u + 0.044715 * u ** 3)))
    for tc in (1, 0):
        got = []
        for k in range(0, len(v), 32):
            out = torch.zeros_like(x)
            lib.tl_nn_set_conv_kernel(tc)
            rc = lib.tl_nn_conv(0, 32, 32, _p(x), _p(w), _p(v[k:k + 32]), None, _p(out), None, None, 1, 1, 16, None)
            lib.tl_nn_set_conv_kernel(1)
            assert rc == 0, tl.last_error()
            got.append(out[0, 1, 5])
        got = torch.cat(got).double()
        fin = v.abs() < 1e10
        want = g(v.double()[fin])
        assert bool(((got[fin] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
        big = got[v == 1e18]
        assert float((big - 1e18).abs().max()) <= 2.0 ** -8 * 1e18 and float(got[v == -1e18].abs().max()) == 0.0
        assert float(got[v == inf][0]) == inf and bool(got[v == -inf].isnan().all() and got[v.isnan()].isnan().all())
    pre = v[fin].bfloat16()
    n = len(pre)
    a, b, o = (torch.zeros((1, 3, n + 2, 1), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    a[0, 1, 1:-1, 0], b[0, 1, 1:-1, 0] = 1.0, pre
    assert lib.tl_nn_gelu_backward(_p(a), _p(b), _p(o), 1, 1, 1, n, None) == 0
    u = pre.double().requires_grad_()
    g(u).sum().backward()
    want = torch.where(u.grad.isnan(), torch.zeros_like(u), u.grad)  # exp overflows far below zero: the limit
    assert bool(((o[0, 1, 1:-1, 0].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
