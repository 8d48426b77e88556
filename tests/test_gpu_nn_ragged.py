"""U-Net kernels at ragged sizes and other channel counts.  Epilogues of the tensor-core GEMM and of the implicit
convolution where some lanes of a warp have nothing to store: rows past M, pixels outside the map (a warp holds 2 rows x 16
columns), with several 16-column tensor-memory loads per warp, against 64-bit products of the same bf16 operands; layers
and heads that the wide kernels cannot take.  Tolerance: K products added in float, each addition off by at most 2^-23 of
the running sum, which never exceeds the sum of the magnitudes; as much again for the bias and the output."""
import pytest

pytestmark = pytest.mark.gpu


def _check(got, ref, mag, K):
    assert bool(((got.double() - ref).abs() <= (K + 2) * 2.0 ** -23 * mag).all())


@pytest.mark.parametrize("M,N,K", [(1, 48, 64), (33, 96, 72), (77, 288, 128), (129, 64, 64), (255, 256, 136)])
def test_gemm_rows_past_the_last(M, N, K):
    import torch

    from dsh import nn as dnn

    g = torch.Generator(device="cuda").manual_seed(M)
    A, B = (torch.randn(n, K, device="cuda", generator=g).bfloat16() for n in (M, N))
    bias = torch.randn(N, device="cuda", generator=g)
    c32 = torch.full((M + 3, N), 7.0, device="cuda")
    ctx = dnn.Ctx(torch)
    ctx.gemm(M, N, K, A, K, B, K, c32=c32, bias=bias)
    ctx.check()
    _check(c32[:M], A.double() @ B.double().t() + bias.double(),
           A.double().abs() @ B.double().abs().t() + bias.double().abs(), K)
    assert bool((c32[M:] == 7).all())


@pytest.mark.parametrize("B,H,W,C,N", [(1, 1, 1, 32, 48), (1, 3, 5, 64, 96), (2, 9, 15, 32, 256), (1, 7, 17, 128, 64),
                                       (1, 25, 31, 96, 288)])
def test_convolution_pixels_outside_the_map(B, H, W, C, N):
    import torch

    from dsh import nn as dnn

    g = torch.Generator(device="cuda").manual_seed(H * W)
    P, K = B * H * W, 9 * C
    x = torch.randn(P, C, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, 9, C, device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    c32 = torch.full((P + 3, N), 7.0, device="cuda")
    ctx = dnn.Ctx(torch)
    ctx.conv3x3(x, B, H, W, C, w, K, N, c32=c32, bias=bias)
    ctx.check()

    def conv(xd, wd, bd):
        pad = torch.nn.functional.pad(xd.view(B, H, W, C), (0, 0, 1, 1, 1, 1))
        out = bd.expand(P, N).clone()
        for t in range(9):
            out += pad[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(P, C) @ wd[:, t].t()
        return out

    xd, wd, bd = x.double(), w.double(), bias.double()
    _check(c32[:P], conv(xd, wd, bd), conv(xd.abs(), wd.abs(), bd.abs()), K)
    assert bool((c32[P:] == 7).all())


@pytest.mark.parametrize("cin,cout,off", [(32, 12, 0), (12, 32, 0), (32, 5, 0), (64, 32, 0), (32, 32, 1), (40, 64, 1)])
def test_conv_layer_of_any_channel_counts(cin, cout, off):
    """A layer's forward and backward pass where the implicit convolution does not apply (output channels no multiple of 8,
    tensors off a 16-byte boundary) and where it does."""
    import numpy as np
    import torch

    from dsh import nn as dnn

    B, H, W = 2, 5, 9
    P, K = B * H * W, 9 * cin
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    ctx = dnn.Ctx(torch)
    layer = dnn.Conv3x3(ctx, cin, cout, np.random.default_rng(cout))
    layer.b.copy_(torch.randn(cout, device="cuda", generator=g))
    x = torch.empty(P * cin + off, dtype=torch.bfloat16, device="cuda")[off:]
    y = torch.empty(P * cout + off, dtype=torch.bfloat16, device="cuda")[off:]
    dy, dx = (torch.empty(P * c + off, device="cuda")[off:] for c in (cout, cin))
    x.copy_(torch.randn(P * cin, device="cuda", generator=g))
    dy.copy_(torch.randn(P * cout, device="cuda", generator=g))
    dy0 = dy.double()
    layer.zero_grad()
    layer.forward(x, B, H, W, y)
    layer.backward(x, y, dy, B, H, W, dx=dx)
    ctx.check()
    w = layer.w.bfloat16().double().view(cout, 3, 3, cin).permute(0, 3, 1, 2)
    conv = torch.nn.functional.conv2d
    maps = lambda t, c: t.view(B, H, W, c).permute(0, 3, 1, 2)
    flat = lambda t, c: t.permute(0, 2, 3, 1).reshape(P, c)
    xd = maps(x.double(), cin)
    z, mag = flat(conv(xd, w, layer.b.double(), padding=1), cout), flat(conv(xd.abs(), w.abs(), layer.b.double().abs(), padding=1), cout)
    got = y.view(P, cout).double()
    assert bool(((got - z.clamp(min=0)).abs() <= 2.0 ** -8 * z.abs() + 2 * (K + 2) * 2.0 ** -23 * mag).all())
    dz32 = torch.where(y.double() > 0, dy0, torch.zeros_like(dy0))
    dz = maps(dz32.bfloat16().double(), cout)
    wt = w.flip(2, 3).transpose(0, 1)
    _check(dx.view(P, cin), flat(conv(dz, wt, padding=1), cin), flat(conv(dz.abs(), wt.abs(), padding=1), cin), 9 * cout)
    xp = torch.nn.functional.pad(x.double().view(B, H, W, cin), (0, 0, 1, 1, 1, 1))
    col = torch.cat([xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(P, cin) for t in range(9)], 1)
    dzf = flat(dz, cout)
    _check(layer.gwt.view(K, cout), col.t() @ dzf, col.abs().t() @ dzf.abs(), P)
    _check(layer.gb, dz32.view(P, cout).sum(0), dz32.view(P, cout).abs().sum(0), P)


@pytest.mark.parametrize("P,C,off", [(1, 8, 0), (297, 32, 0), (1001, 36, 0), (640, 5, 0), (300, 16, 1), (2000, 248, 0)])
def test_head_of_any_channel_count(P, C, off):
    """The 1x1 head and its gradients: 8 channels a load (a multiple of 8), 4 (of 4), else one."""
    import torch

    from dsh import nn as dnn

    L = dnn.nnlib()
    g = torch.Generator(device="cuda").manual_seed(P + C)
    x = torch.empty(P * C + off, dtype=torch.bfloat16, device="cuda")[off:]
    x.copy_(torch.randn(P * C, device="cuda", generator=g))
    w, b, dout = (torch.randn(n, device="cuda", generator=g) for n in (C, 1, P))
    out = torch.full((P + 3,), 7.0, device="cuda")
    dx = torch.full((P * C + off + 3,), 7.0, device="cuda")[off:]
    gw, gb, part = torch.zeros(C, device="cuda"), torch.zeros(1, device="cuda"), torch.empty(dnn.RED_BLOCKS * (C + 1), device="cuda")
    assert L.dsh_nn_head_fwd(x.data_ptr(), P, C, w.data_ptr(), b.data_ptr(), out.data_ptr(), None) == 0
    assert L.dsh_nn_head_bwd(dout.data_ptr(), x.data_ptr(), P, C, w.data_ptr(), dx.data_ptr(), gw.data_ptr(), gb.data_ptr(),
                             part.data_ptr(), None) == 0
    torch.cuda.synchronize()
    xd, wd, dd = x.double().view(P, C), w.double(), dout.double()
    _check(out[:P], xd @ wd + b.double(), xd.abs() @ wd.abs() + b.double().abs(), C)
    assert torch.equal(dx[:P * C].view(P, C), dout[:, None] * w) and bool((dx[P * C:] == 7).all()) and bool((out[P:] == 7).all())
    _check(gw, dd @ xd, dd.abs() @ xd.abs(), P + dnn.RED_BLOCKS)
    _check(gb[0], dd.sum(), dd.abs().sum(), P + dnn.RED_BLOCKS)
