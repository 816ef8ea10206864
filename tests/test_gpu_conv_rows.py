"""The convolution with tiles of one, two and four rows: the same images in
batches that take each of them, whole and ragged heights, against the warp-level
kernel on all of them at once.

Bound as between those two kernels: FP32 sums of the same BF16 products in
another order, so BF16 outputs within one rounding (2^-7) and the FP32 head
within its sum's rounding; halos and what lies behind the buffers untouched."""
import ctypes as C

import pytest

import tealeaf_cuda_gb300 as tl

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


# (images, batch sizes that they are computed in): one row by few tiles and by tiles that are no
# fewer with more rows, two and four by the number of tiles
@pytest.mark.parametrize("shape,batches", [((14, 99, 96), (1, 8, 14)), ((14, 97, 80), (1, 10, 14)),
                                           ((2, 256, 256), (1, 2)), ((520, 1, 32), (1, 520)), ((480, 2, 16), (480,)),
                                           ((300, 3, 112), (100, 300)), ((5, 130, 240), (2, 5))])
@pytest.mark.parametrize("cin,cout,mode", [(16, 32, 0), (32, 32, 1), (32, 16, 2), (32, 32, 3)])
def test_rows_of_a_tile(shape, batches, cin, cout, mode):
    torch = pytest.importorskip("torch")
    lib = tl.load()
    lib.tl_nn_set_conv_kernel.argtypes = [C.c_int]
    N, H, W = shape
    gen = torch.Generator(device="cuda").manual_seed(cin + cout + mode + W)

    def field(ch):
        t = torch.zeros((N, H + 2, W + 2, ch), dtype=torch.bfloat16, device="cuda")
        t[:, 1:-1, 1:-1] = torch.randn((N, H, W, ch), generator=gen, device="cuda")
        return t

    x = field(cin)
    res = x if mode == 1 else field(cout)
    w = (0.2 * torch.randn((9, cout, cin), generator=gen, device="cuda")).bfloat16()
    bias = 0.1 * torch.randn(cout, generator=gen, device="cuda")

    def run(tc, batch):
        out, pre = (torch.zeros((N + 1, H + 2, W + 2, cout), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        head = torch.zeros((N + 1, H, W), device="cuda")
        out[N], pre[N], head[N] = 3.0, 3.0, 3.0
        lib.tl_nn_set_conv_kernel(tc)
        for k in range(0, N, batch):
            rc = lib.tl_nn_conv(mode, cin, cout, _p(x[k:]), _p(w), _p(bias), _p(res[k:]) if mode in (1, 3) else None,
                                _p(out[k:]), _p(pre[k:]), _p(head[k:]), min(batch, N - k), H, W, None)
            assert rc == 0, tl.last_error()
        lib.tl_nn_set_conv_kernel(1)
        torch.cuda.synchronize()
        assert lib.tl_nn_conv_status() == 0, tl.last_error()
        assert bool((out[N] == 3.0).all() and (pre[N] == 3.0).all() and (head[N] == 3.0).all())
        for t in (out[:N], pre[:N]):
            assert float(t[:, 0].abs().sum() + t[:, -1].abs().sum() + t[:, :, 0].abs().sum() + t[:, :, -1].abs().sum()) == 0
        return out[:N].float(), pre[:N].float(), head[:N]

    want = run(0, N)
    for batch in batches:
        for a, b in zip(run(1, batch), want):
            assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-5).all()), batch
