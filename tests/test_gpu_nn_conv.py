"""The tile-halo convolutions and weight gradients (hp2d_nn_conv3x3_any, hp2d_nn_conv3x3_wgrad) and the
16-byte forms of the layers between them, at image sizes off the 8 x 16 tile and at every kernel of the
dispatch.  Forward and backward-data run the K steps of im2col + GEMM in the same order: bit for bit.
Weight gradients and column sums only reorder FP32 sums of n exact products: each output is within
n 2^-24 of the sum of the products' magnitudes (here 2^-20 of it, n <= 2048 per chain with a margin)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 16, 8), (2, 5, 3), (1, 17, 9), (2, 33, 26), (1, 20, 28)]


def _rand(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ci,co", [(4, 32), (2, 32), (1, 100), (32, 2), (32, 32), (32, 64), (64, 32), (64, 64), (64, 128),
                                   (64, 200), (96, 40), (128, 64)])
def test_convolution_equals_im2col_gemm(shape, ci, co):
    from hydropol2d_b200 import nn
    B, H, W = shape
    kp = (9 * ci + 63) // 64 * 64
    x = _rand((B, H, W, ci), 1)
    w = torch.zeros(co, kp, dtype=torch.bfloat16, device="cuda")
    w[:, :9 * ci] = _rand((co, 9 * ci), 2)
    bias = _rand((co,), 3, torch.float32)
    for epi, dt in (("bf16_bias_relu", torch.bfloat16), ("f32_bias", torch.float32)):
        got = torch.full((B * H * W, co), 7.0, dtype=dt, device="cuda")
        want = torch.empty_like(got)
        nn.conv3x3_any(x, w, co, got, epi, bias=bias)
        nn.gemm(nn.im2col3x3(x, kp), w, want, epi, bias=bias)
        nn.check()
        assert torch.equal(got, want), epi


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ci,co", [(4, 32), (2, 64), (1, 96), (32, 2), (64, 3), (32, 32), (32, 64), (64, 32), (128, 64),
                                   (96, 160)])
def test_weight_gradient(shape, ci, co):
    from hydropol2d_b200 import nn
    B, H, W = shape
    kp = (9 * ci + 63) // 64 * 64
    x, dy = _rand((B, H, W, ci), 4), _rand((B, H, W, co), 5)
    g0 = torch.zeros(co, kp, device="cuda")
    g0[:, :9 * ci] = 0.5
    gW = g0.clone()
    nn.conv3x3_wgrad(x, dy, gW)
    nn.check()
    cols = nn.im2col3x3(x, kp).double()
    d = dy.reshape(-1, co).double()
    want = g0.double() + d.T @ cols
    scale = g0.double().abs() + d.abs().T @ cols.abs()
    assert torch.all((gW.double() - want).abs() <= scale * 2.0 ** -20)
    assert torch.all(gW[:, 9 * ci:] == 0)


def test_unsupported_channels_are_refused():
    from hydropol2d_b200 import HP2DError, nn
    x = _rand((1, 8, 8, 16), 6)
    with pytest.raises(HP2DError):
        nn.conv3x3_any(x, _rand((32, 192), 7), 32, torch.empty(64, 32, dtype=torch.bfloat16, device="cuda"), "bf16_bias",
                       bias=torch.zeros(32, device="cuda"))
    with pytest.raises(HP2DError):
        nn.conv3x3_wgrad(x, _rand((1, 8, 8, 32), 8), torch.zeros(32, 192, device="cuda"))


@pytest.mark.parametrize("C", [8, 24, 32, 36, 256])
def test_vector_layers_equal_torch(C):
    from hydropol2d_b200 import nn
    x = _rand((3, 6, 10, C), 9)
    p = nn.maxpool2(x)
    assert torch.equal(p, x.reshape(3, 3, 2, 5, 2, C).amax(dim=(2, 4)))
    up = nn.upsample2(x)
    assert torch.equal(up, x.repeat_interleave(2, 1).repeat_interleave(2, 2))
    f = up.float().reshape(3, 6, 2, 10, 2, C)
    s = (f[:, :, 0, :, 0] + f[:, :, 0, :, 1]) + (f[:, :, 1, :, 0] + f[:, :, 1, :, 1])
    assert torch.equal(nn.upsample2_bwd(up), s.to(torch.bfloat16))
    dy, acc = _rand(p.shape, 10), _rand(x.shape, 11)
    hit = x == p.repeat_interleave(2, 1).repeat_interleave(2, 2)
    blocks = hit.reshape(3, 3, 2, 5, 2, C).permute(0, 1, 3, 5, 2, 4).reshape(-1, 4)
    first = (blocks & (blocks.cumsum(1) == 1)).reshape(3, 3, 5, C, 2, 2).permute(0, 1, 4, 2, 5, 3).reshape(x.shape)
    d = dy.repeat_interleave(2, 1).repeat_interleave(2, 2)
    routed = torch.where(first, d, torch.zeros_like(d))
    assert torch.equal(nn.maxpool2_bwd(x, p, dy), routed)
    want = torch.where(first, (acc.float() + d.float()).to(torch.bfloat16), acc)
    assert torch.equal(nn.maxpool2_bwd(x, p, dy, acc.clone()), want)
    dst = _rand((3, 6, 10, 2 * C), 12)
    want = dst.clone()
    want[..., C:] = x
    nn.copy_channels(x, 0, C, dst, C)
    assert torch.equal(dst, want)
    y, g = _rand((180, C), 13), _rand((180, C), 14)
    out = torch.ones(C, device="cuda")
    masked = torch.where(y.float() > 0, g, torch.zeros_like(g))
    nn.relu_colsum(y, g, out)
    assert torch.equal(g, masked)
    assert torch.all((out.double() - 1 - masked.double().sum(0)).abs() <= (1 + masked.double().abs().sum(0)) * 2.0 ** -20)


@pytest.mark.parametrize("c,ld", [(8, 16), (32, 64), (64, 200)])
def test_relu_mask_from_channels_of_a_wider_tensor(c, ld):
    from hydropol2d_b200 import nn
    wide, g = _rand((777, ld), 11), _rand((777, c), 12)
    y = wide[:, 8:8 + c] if ld > c + 8 else wide[:, :c]
    a, b = g.clone(), g.clone()
    sa, sb = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
    nn.relu_colsum(y, a, sa)
    nn.relu_colsum(y.contiguous(), b, sb)
    assert torch.equal(a, b)
    torch.testing.assert_close(sa, sb, rtol=1e-5, atol=1e-4)   # FP32 sums of 777 terms in another order


def test_adam_in_one_buffer_equals_adam_by_layer():
    from hydropol2d_b200.surrogate import UNet
    nets = [UNet(seed=5, base=16, levels=2) for _ in range(2)]
    for c in nets[1].layers.values():   # tensors of their own: the layers one by one
        c.W, c.b = c.W.clone(), c.b.clone()
    for net in nets:
        gen = torch.Generator().manual_seed(7)
        for _ in range(2):
            net.zero_grad()
            for c in net.layers.values():
                c.gW.add_(torch.randn(c.gW.shape, generator=gen).cuda())
                c.gb.add_(torch.randn(c.gb.shape, generator=gen).cuda())
            net.adam_step(1e-3, 1e-2)
    assert nets[0]._one_buffer("W") and not nets[1]._one_buffer("W")
    for a, b in zip(nets[0].layers.values(), nets[1].layers.values()):
        for name in ("W", "b", "mW", "vW", "mb", "vb", "W16", "gW", "gb"):
            assert torch.equal(getattr(a, name), getattr(b, name)), name
