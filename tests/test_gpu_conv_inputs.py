"""One convolution layer on inputs that do not start on a 16-byte boundary (slices of a batch of odd
images) and on output gradients that are channels of a wider tensor: the results of aligned copies."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(ci, co, relu):
    from hydropol2d_b200.surrogate import Conv3x3
    return Conv3x3("layer", ci, co, relu, torch.Generator().manual_seed(1), "cuda")


def _off(t, n):
    """The values of t in memory that starts n elements after an aligned address."""
    flat = torch.empty(t.numel() + n, dtype=t.dtype, device=t.device)
    flat[n:].copy_(t.reshape(-1))
    return flat[n:].view(t.shape)


@pytest.mark.parametrize("ci,co,relu", [(4, 32, True), (1, 32, True), (32, 2, False), (64, 64, True), (32, 3, False)])
@pytest.mark.parametrize("off", [1, 4])
def test_inputs_off_the_boundary(ci, co, relu, off):
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(3, 5, 7, ci, generator=gen, device="cuda").to(torch.bfloat16)
    dy = torch.randn(3, 5, 7, co, generator=gen, device="cuda").to(torch.bfloat16)
    if ci == 4:
        off = 4   # a slice of images starts at a pixel
    a, b = _layer(ci, co, relu), _layer(ci, co, relu)
    ya, yb = a.forward(x), b.forward(_off(x, off))
    assert torch.equal(ya, yb)
    dyb = _off(dy, off)
    da, db = a.backward(dy.clone()), b.backward(dyb)
    assert torch.equal(da, db)
    # FP32 sums of the 105 pixels in another order
    torch.testing.assert_close(a.gW, b.gW, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(a.gb, b.gb, rtol=1e-5, atol=1e-5)


def test_output_gradient_in_a_wider_tensor():
    a, b = _layer(32, 2, False), _layer(32, 2, False)
    x = torch.randn(2, 8, 8, 32, device="cuda").to(torch.bfloat16)
    wide = torch.randn(2, 8, 8, 6, device="cuda").to(torch.bfloat16)
    for layer in (a, b):
        layer.forward(x)
    a.backward(wide[..., 2:4].contiguous(), need_dx=False)
    b.backward(wide[..., 2:4], need_dx=False)
    torch.testing.assert_close(a.gW, b.gW, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(a.gb, b.gb, rtol=1e-5, atol=1e-5)
