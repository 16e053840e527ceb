"""The weight gradient's distance from 64 bits against that of the split-K GEMM over pixels, on the
network's layers.  Inputs are positive, so that the tensor core's truncation of its sums does not average
out: an accumulator of n steps is low by about n / 2 units of its last place, the sums are low by the mean
over their parts, and longer chains than the GEMM's show directly.  Both round the parts' additions
differently (their order is the hardware's), hence 5 % and a quarter of a unit in the last place."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,height,width", [(16, 128, 128), (4, 128, 128), (8, 56, 40), (2, 16, 16)])
@pytest.mark.parametrize("ci,co", [(4, 32), (32, 32), (32, 64), (64, 32), (64, 128), (128, 128), (256, 128), (256, 256), (32, 2)])
def test_error_is_no_larger_than_the_gemms(ci, co, batch, height, width):
    from hydropol2d_b200 import nn
    gen = torch.Generator(device="cuda").manual_seed(ci + co)
    x = torch.rand(batch, height, width, ci, generator=gen, device="cuda").to(torch.bfloat16)
    dy = torch.rand(batch, height, width, co, generator=gen, device="cuda").to(torch.bfloat16)
    kp, P = (9 * ci + 63) // 64 * 64, batch * height * width
    d = dy.view(P, co)
    want = torch.zeros(co, 9 * ci, dtype=torch.float64, device="cuda")
    cols = nn.im2col3x3(x, kp)
    for p in range(0, P, 1 << 16):
        want += d[p:p + (1 << 16)].double().T @ cols[p:p + (1 << 16), :9 * ci].double()
    tiles = -(-co // 128) * -(-kp // (256 if kp > 128 else kp))
    gW, gemm = torch.zeros(co, kp, device="cuda"), torch.zeros(co, kp, device="cuda")
    nn.conv3x3_wgrad(x, dy, gW)
    nn.gemm(nn.transpose(d), nn.im2col3x3(x, kp, transpose=True), gemm, "f32_atomic",
            split_k=max(1, min(P // 64, (2 * 148) // max(tiles, 1))))
    nn.check()

    def err(g):
        return ((g[:, :9 * ci].double() - want) / want).pow(2).mean().sqrt().item()

    assert err(gW) <= 1.05 * err(gemm) + 0.25 * 2.0 ** -24
