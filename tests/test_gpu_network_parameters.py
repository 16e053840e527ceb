"""The network's parameters: laid out once, in one buffer each, with the values that its layers made one
by one from the same generator would have; making a network allocates no more tensors than its layers
alone (ten each)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_parameters_of_a_network():
    from hydropol2d_b200.surrogate import Conv3x3, UNet
    torch.zeros(1, device="cuda")
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    net = UNet(seed=9, base=16, levels=3)
    made = torch.cuda.memory_stats()["allocation.all.allocated"] - before
    assert made <= 10 * len(net.spec) + 1   # and the loss
    assert net._one_buffer(*net._flat)
    gen = torch.Generator().manual_seed(9)
    for layer in net.spec:
        one, of_net = Conv3x3(*layer, gen, "cuda"), net.layers[layer[0]]
        for name in ("W", "W16", "b", "gW", "gb", "mW", "vW", "mb", "vb", "zero_ci"):
            a, b = getattr(one, name), getattr(of_net, name)
            assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b), (layer[0], name)
            assert b.is_contiguous() and b.data_ptr() % 16 == 0
