"""The layer calls of the compiled extension: what makes an output require a gradient."""
import pytest
import torch

from mappedconvolutions_b200 import nn as mnn

pytestmark = pytest.mark.gpu


def _cases():
    m = torch.rand(5, 6, 3, 2, device="cuda") * 4
    x = torch.randn(2, 4, 5, 6, device="cuda")
    return [(mnn.MappedConvolution(4, 3, 3).cuda(), (x, m)), (mnn.MappedTransposedConvolution(4, 3, 3).cuda(), (x, 7, 8, m)),
            (mnn.MappedMaxPool(3), (x, m)), (mnn.MappedAvgPool(3), (x, m)), (mnn.MappedAvgUnpool(3), (x, 7, 8, m)),
            (mnn.Resample(), (x, m[:, :, 0].contiguous(), (7, 8))), (mnn.Unresample(), (x, m[:, :, 0].contiguous()))]


@pytest.mark.parametrize("which", range(7))
def test_a_map_that_requires_a_gradient(which):
    """The output requires one too, and the map's own is undefined: a loss over frozen layers can be run backward."""
    layer, args = _cases()[which]
    layer.requires_grad_(False)
    assert not layer(*args).requires_grad
    m = next(a for a in args[1:] if isinstance(a, torch.Tensor)).requires_grad_()
    y = layer(*args)
    assert y.requires_grad
    y.backward(torch.ones_like(y))
    assert m.grad is None and args[0].grad is None
