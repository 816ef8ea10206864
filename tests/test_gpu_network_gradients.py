"""The network's weight and bias gradients and the GELU gradient at the sizes
where their kernels' tiles end: one 16-pixel group, segments of 64 pixels and
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
