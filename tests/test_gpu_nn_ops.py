"""Layout, pooling and reduction kernels of the U-Net against plain PyTorch on the same values: the 16-byte vector
kernels (channels a multiple of 8), at sizes with tile remainders, and the scalar kernels that serve other channel
counts and unaligned bases.  Copies and selections are exact, and so are the column sums: 296 chunks of rows, each added
in row order, then added in chunk order."""
import pytest

pytestmark = pytest.mark.gpu


def _env():
    import torch

    from dsh import nn as dnn

    return torch, dnn.nnlib()


def _buf(torch, n, dtype, off=0):
    """Device buffer of n elements starting off elements past an aligned base, filled with a pattern that must vanish."""
    return torch.full((n + off,), -7.0 if dtype != torch.uint8 else 77, dtype=dtype, device="cuda")[off:]


def _shift(x, tap, torch):
    """x [B, H, W, C] moved by tap (dy, dx) = (tap / 3 - 1, tap % 3 - 1), zero outside."""
    B, H, W, C = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    return p[:, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W]


@pytest.mark.parametrize("B,H,W,C,off", [(1, 1, 1, 8, 0), (2, 5, 7, 8, 0), (1, 9, 31, 40, 0), (2, 8, 16, 64, 0),
                                         (1, 3, 65, 256, 0), (1, 6, 5, 3, 0), (1, 4, 9, 16, 1)])
def test_columns_and_transposes(B, H, W, C, off):
    torch, L = _env()
    P, K = B * H * W, 9 * C
    ldk, ldp = (K + 7) // 8 * 8, (P + 7) // 8 * 8
    x = torch.randn(P * C, device="cuda").bfloat16()
    xb = _buf(torch, P * C, torch.bfloat16, off)
    xb.copy_(x)
    want = torch.stack([_shift(x.view(B, H, W, C), t, torch).reshape(P, C) for t in range(9)], 1).reshape(P, K)
    col, colT, yT = (_buf(torch, n, torch.bfloat16) for n in (P * ldk, K * ldp, C * ldp))
    assert L.dsh_nn_im2col(xb.data_ptr(), B, H, W, C, col.data_ptr(), ldk, None) == 0
    assert L.dsh_nn_im2col_t(xb.data_ptr(), B, H, W, C, colT.data_ptr(), ldp, None) == 0
    assert L.dsh_nn_transpose(xb.data_ptr(), P, C, yT.data_ptr(), ldp, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(col.view(P, ldk)[:, :K], want)
    assert torch.equal(colT.view(K, ldp)[:, :P], want.t())
    assert torch.equal(yT.view(C, ldp)[:, :P], x.view(P, C).t())
    assert bool((col.view(P, ldk)[:, K:] == -7).all()) and bool((colT.view(K, ldp)[:, P:] == -7).all())


@pytest.mark.parametrize("B,h,w,C,off", [(1, 1, 1, 8, 0), (2, 3, 5, 32, 0), (1, 7, 11, 256, 0), (1, 3, 4, 5, 0),
                                         (1, 2, 3, 8, 1)])
def test_pool_upsample_concat(B, h, w, C, off):
    torch, L = _env()
    H, W, P, p = 2 * h, 2 * w, 4 * B * h * w, B * h * w
    g = lambda n: torch.randn(n, device="cuda")
    x = _buf(torch, P * C, torch.bfloat16, off)
    x.copy_(g(P * C).clamp(min=0))                  # ties, as after a ReLU
    y, arg = _buf(torch, p * C, torch.bfloat16, off), _buf(torch, p * C, torch.uint8, off)
    assert L.dsh_nn_maxpool_fwd(x.data_ptr(), B, H, W, C, y.data_ptr(), arg.data_ptr(), None) == 0
    win = x.view(B, h, 2, w, 2, C).permute(0, 1, 3, 5, 2, 4).reshape(p * C, 4).float()
    first = (win == win.amax(1, keepdim=True)).int().argmax(1)
    torch.cuda.synchronize()
    assert torch.equal(y.float(), win.amax(1)) and torch.equal(arg.long(), first)
    dy, dx = _buf(torch, p * C, torch.float32, off), _buf(torch, P * C, torch.float32, off)
    dy.copy_(g(p * C))
    assert L.dsh_nn_maxpool_bwd(dy.data_ptr(), arg.data_ptr(), B, H, W, C, dx.data_ptr(), None) == 0
    ref = torch.zeros((p * C, 4), device="cuda").scatter_(1, first[:, None], dy[:, None].clone())
    ref = ref.view(B, h, w, C, 2, 2).permute(0, 1, 4, 2, 5, 3).reshape(-1)
    torch.cuda.synchronize()
    assert torch.equal(dx, ref)
    up = _buf(torch, P * C, torch.bfloat16, off)
    assert L.dsh_nn_upsample_fwd(y.data_ptr(), B, h, w, C, up.data_ptr(), None) == 0
    back = _buf(torch, p * C, torch.float32, off)
    assert L.dsh_nn_upsample_bwd(dx.data_ptr(), B, h, w, C, back.data_ptr(), None) == 0
    rep = y.view(B, h, 1, w, 1, C).expand(B, h, 2, w, 2, C).reshape(-1)
    d = dx.view(B, h, 2, w, 2, C)
    torch.cuda.synchronize()
    assert torch.equal(up, rep)
    assert torch.equal(back, (((d[:, :, 0, :, 0] + d[:, :, 0, :, 1]) + d[:, :, 1, :, 0]) + d[:, :, 1, :, 1]).reshape(-1))
    cat = _buf(torch, 2 * P * C, torch.bfloat16, off)
    assert L.dsh_nn_concat(x.data_ptr(), C, up.data_ptr(), C, P, cat.data_ptr(), None) == 0
    dcat, a, b = _buf(torch, 2 * P * C, torch.float32, off), *(_buf(torch, P * C, torch.float32, off) for _ in range(2))
    dcat.copy_(g(2 * P * C))
    assert L.dsh_nn_split(dcat.data_ptr(), C, C, P, a.data_ptr(), b.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(cat.view(P, 2 * C), torch.cat([x.view(P, C), up.view(P, C)], 1))
    assert torch.equal(a.view(P, C), dcat.view(P, 2 * C)[:, :C]) and torch.equal(b.view(P, C), dcat.view(P, 2 * C)[:, C:])


@pytest.mark.parametrize("P,N,off", [(1, 8, 0), (295, 32, 0), (1001, 128, 0), (5000, 256, 0), (777, 24, 0), (513, 64, 1)])
def test_relu_backward_add_and_column_sums(P, N, off):
    torch, L = _env()
    dy, other = (_buf(torch, P * N, torch.float32, off) for _ in range(2))
    dy.copy_(torch.randn(P * N, device="cuda"))
    other.copy_(torch.randn(P * N, device="cuda"))
    y, dz = (_buf(torch, P * N, torch.bfloat16, off) for _ in range(2))
    y.copy_(torch.randn(P * N, device="cuda").clamp(min=0))
    want = torch.where(y.float() > 0, dy, torch.zeros_like(dy))
    assert L.dsh_nn_relu_bwd(dy.data_ptr(), y.data_ptr(), dz.data_ptr(), dy.data_ptr(), P * N, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(dy, want) and torch.equal(dz, want.bfloat16())
    gsum = torch.ones(N, device="cuda")
    part = torch.empty(296 * (N + 1), device="cuda")
    assert L.dsh_nn_colsum(dy.data_ptr(), P, N, gsum.data_ptr(), part.data_ptr(), None) == 0
    torch.cuda.synchronize()
    rows = (P + 295) // 296
    pad = torch.zeros((296 * rows, N), device="cuda")
    pad[:P] = dy.view(P, N)
    acc = torch.zeros((296, N), device="cuda")
    for r in range(rows):                           # + 0.0 for the rows past P: no value changes
        acc = acc + pad.view(296, rows, N)[:, r]
    total = torch.zeros(N, device="cuda")
    for b in range(296):
        total = total + acc[b]
    assert torch.equal(gsum, 1 + total)
    s = dy + other
    assert L.dsh_nn_add(dy.data_ptr(), other.data_ptr(), P * N, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(dy, s)


@pytest.mark.parametrize("B,H,W,C,N", [(1, 1, 1, 32, 32), (2, 9, 17, 32, 64), (1, 8, 16, 64, 8), (1, 25, 75, 96, 32),
                                       (1, 13, 40, 128, 256), (2, 7, 15, 256, 128), (1, 16, 33, 64, 288)])
def test_convolution_equals_columns_and_gemm(B, H, W, C, N):
    """The implicit convolution gives the bits of im2col + GEMM, with and without bias and ReLU, at tiles of 8 x 16 pixels
    with remainders, both K block sizes and every N tile."""
    torch, L = _env()
    from dsh import nn as dnn

    P, K = B * H * W, 9 * C
    ctx = dnn.Ctx(torch)
    x = torch.randn(P * C, device="cuda").bfloat16()
    w = (torch.randn(N * K, device="cuda") / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda")
    col = torch.empty(P * K, dtype=torch.bfloat16, device="cuda")
    assert L.dsh_nn_im2col(x.data_ptr(), B, H, W, C, col.data_ptr(), K, None) == 0
    for b, relu in ((None, False), (bias, True)):
        want16, got16 = torch.empty(P * N, dtype=torch.bfloat16, device="cuda"), _buf(torch, P * N, torch.bfloat16)
        ctx.gemm(P, N, K, col, K, w, K, c16=want16, bias=b, relu=relu)
        ctx.conv3x3(x, B, H, W, C, w, K, N, c16=got16, bias=b, relu=relu)
        want32, got32 = torch.empty(P * N, device="cuda"), _buf(torch, P * N, torch.float32)
        ctx.gemm(P, N, K, col, K, w, K, c32=want32, bias=b, relu=relu)
        ctx.conv3x3(x, B, H, W, C, w, K, N, c32=got32, bias=b, relu=relu)
        ctx.check()
        assert torch.equal(got16, want16) and torch.equal(got32, want32)
