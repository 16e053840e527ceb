"""The loss kernel at pixel counts around its blocks: its clusters' blocks add their sums in shared
memory of the first, also where most of them have no pixel.  Against FP64 on the host: each term is
three rounded FP32 products, the sums run in FP64 up to one FP32 atomic for each of the 16 clusters, so
the loss is within (3 + 17) 2^-24 of itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("P", [1, 3, 511, 512, 513, 4097, 65537, 200000])
def test_loss_of_few_and_many_pixels(P, weighted):
    from hydropol2d_b200 import nn
    gen = torch.Generator().manual_seed(P)
    pred, t, w = (torch.rand(P, 2, generator=gen) for _ in range(3))
    scale = 1.0 / (2 * P)
    d = (pred - t)   # the kernel's FP32 difference
    want = ((w.double() if weighted else 1.0) * d.double() ** 2).sum().item() * scale
    pred, t, w = pred.cuda(), t.cuda(), w.cuda()
    for _ in range(20):
        loss = torch.zeros(1, device="cuda")
        dpred = torch.empty(P, 2, dtype=torch.bfloat16, device="cuda")
        nn.mse(pred, t, w if weighted else None, scale, loss, dpred)
        assert abs(loss.item() - want) <= 20 * 2.0 ** -24 * want
    assert torch.equal(dpred.cpu(), ((2.0 * (w.cpu() if weighted else 1.0) * d) * torch.tensor(scale)).to(torch.bfloat16))
