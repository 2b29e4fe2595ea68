"""CPU: what a layer hands to the op behind it, with the op replaced by torch arithmetic of the same arguments."""
import warnings

import pytest
import torch
import torch.autograd.forward_ad as fwad

from mappedconvolutions_b200 import host
from mappedconvolutions_b200 import nn as mnn
from mappedconvolutions_b200.nn import functions as F


def _written_behind_torch(values):
    y = torch.empty(values.shape)
    y.numpy()[...] = 2 * values.detach().numpy()
    return y


OPS = dict(mapped_conv_forward=lambda x, m, w, b, k, i: _written_behind_torch(x[:, :1].expand(-1, w.shape[0], -1, -1)),
           mapped_avg_pool=lambda x, m, k, i: _written_behind_torch(x[:, :, :m.shape[0], :m.shape[1]]),
           resample_from_map=lambda x, m, i: _written_behind_torch(x[:, :, :m.shape[0], :m.shape[1]]))
NODES = dict(conv_layer=lambda x, w, b, m, k, i, *r: OPS["mapped_conv_forward"](x, m, w, b, k, i),
             avg_pool_layer=lambda x, m, k, i, iw: OPS["mapped_avg_pool"](x, m, k, i),
             unresample_layer=lambda x, m, i, iw: OPS["resample_from_map"](x, m, i))


@pytest.fixture
def calls(monkeypatch):
    """Layer calls on the CPU.  Whether a node takes a call is the extension's answer (a CPU tensor that it would
    have taken is refused as such); the arithmetic is the one above.  Lists the nodes that were taken."""
    if not host.COMPILED:
        pytest.skip("extension not built: only the Functions exist")
    taken = []

    def node(name):
        def call(*a):
            try:
                out = getattr(host.impl, name)(*a)
                assert out is None
                return None
            except RuntimeError as e:
                assert "CUDA only" in str(e)
            taken.append(name)
            return NODES[name](*a)
        return call

    monkeypatch.setattr(F, "ops", type("Ops", (), {n: staticmethod(f) for n, f in OPS.items()}
                                       | {n: staticmethod(node(n)) for n in NODES}))
    for name, function in (("conv", F.MappedConvFn), ("avg_pool", F.MappedAvgPoolFn), ("unresample", F.UnresampleFn)):
        monkeypatch.setattr(F, name, F._layer_call(function, name + "_layer"))
    return taken


LAYERS = [(lambda: mnn.MappedConvolution(3, 3, 5, "nearest"), torch.zeros(4, 6, 5, 2)),
          (lambda: mnn.MappedAvgPool(5, "nearest"), torch.zeros(4, 6, 5, 2)),
          (lambda: mnn.Unresample("nearest"), torch.zeros(4, 6, 2))]


@pytest.mark.parametrize("make,m", LAYERS, ids=["conv", "pool", "unresample"])
def test_plain_calls_take_the_node(calls, make, m):
    x = torch.randn(2, 3, 4, 6)
    make()(x, m)
    assert len(calls) == 1


@pytest.mark.parametrize("make,m", LAYERS, ids=["conv", "pool", "unresample"])
@pytest.mark.parametrize("no_grad", [False, True])
def test_traced_layers_run_again_on_replay(calls, make, m, no_grad):
    layer = make()
    layer.requires_grad_(not no_grad)
    x, z = torch.randn(2, 3, 4, 6), torch.randn(2, 3, 4, 6)
    with warnings.catch_warnings(), torch.set_grad_enabled(not no_grad):
        warnings.simplefilter("ignore")
        model = torch.nn.Module()
        model.layer, model.forward = layer, lambda t: layer(t, m)
        traced = torch.jit.trace(model, (x,), check_trace=False)
        assert not calls
        assert torch.equal(traced(z), layer(z, m))


@pytest.mark.parametrize("make,m", LAYERS, ids=["conv", "pool", "unresample"])
@pytest.mark.parametrize("no_grad", [False, True])
def test_tangents_are_not_dropped(calls, make, m, no_grad):
    layer = make().requires_grad_(False)
    with fwad.dual_level(), torch.set_grad_enabled(not no_grad):
        x = fwad.make_dual(torch.randn(2, 3, 4, 6), torch.randn(2, 3, 4, 6))
        with pytest.raises((NotImplementedError, RuntimeError)):
            layer(x, m)
    assert not calls


def test_tangents_of_a_map_are_not_dropped(calls):
    with fwad.dual_level(), pytest.raises((NotImplementedError, RuntimeError)):
        mnn.Unresample("bilinear")(torch.randn(2, 3, 4, 6), fwad.make_dual(torch.zeros(4, 6, 2), torch.ones(4, 6, 2)))
    assert not calls


@pytest.mark.parametrize("make,m", LAYERS, ids=["conv", "pool", "unresample"])
def test_functorch_transforms_are_refused(calls, make, m):
    layer = make().requires_grad_(False)
    x = torch.randn(2, 3, 4, 6)
    for f in (lambda: torch.func.vmap(lambda t: layer(t[None], m))(x), lambda: torch.func.grad(lambda t: layer(t, m).sum())(x),
              lambda: torch.func.jvp(lambda t: layer(t, m), (x,), (x,))):
        with pytest.raises(RuntimeError, match="functorch transforms"):
            f()
    assert not calls


def _layer_and_args(transposed):
    if transposed:
        return mnn.MappedTransposedConvolution(4, 3, 5), (torch.zeros(1, 4, 6, 7), 8, 9, torch.zeros(6, 7, 5, 2))
    return mnn.MappedConvolution(4, 3, 5), (torch.zeros(1, 4, 6, 7), torch.zeros(6, 7, 5, 2))


def _prune(layer):
    import torch.nn.utils.prune as prune
    prune.random_unstructured(layer, "weight", amount=0.3)


def _shared_memory_copy(layer):
    replica = layer._replicate_for_data_parallel()  # (what nn.DataParallel calls: parameters become plain attributes)
    for name, p in layer.named_parameters():
        setattr(replica, name, p.clone())
    return replica


@pytest.mark.filterwarnings("ignore::FutureWarning")
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("change", [
    lambda l: None, torch.nn.utils.parametrizations.weight_norm, torch.nn.utils.parametrizations.spectral_norm,
    torch.nn.utils.weight_norm, torch.nn.utils.spectral_norm, _prune, _shared_memory_copy,
], ids=["plain", "weight_norm", "spectral_norm", "old weight_norm", "old spectral_norm", "prune", "data parallel"])
def test_parameters_that_are_attributes_only(monkeypatch, transposed, change):
    layer, args = _layer_and_args(transposed)
    layer = change(layer) or layer
    seen = {}

    def op(x, weight, bias, *rest):
        seen.update(weight=weight, bias=bias)
        return (weight.sum() + bias.sum()).reshape(1, 1, 1, 1)

    monkeypatch.setattr(F, "tconv" if transposed else "conv", op)
    layer(*args).sum().backward()
    assert seen["weight"].shape == ((4, 3, 5) if transposed else (3, 4, 5)) and seen["bias"].shape == (3,)
    if "_shared" not in change.__name__:
        assert all(p.grad is not None for p in layer.parameters())


@pytest.mark.parametrize("call", [
    lambda x, m: mnn.Resample()(x, m[:, :, 0], (8.0, 9.0)),              # H / 2, a numpy or tensor size
    lambda x, m: mnn.Resample()(x, m[:, :, 0], (8, 9, 3)),               # an image's shape
    lambda x, m: mnn.Resample()(x, m[:, :, 0], torch.tensor([8.0, 9.0])),
    lambda x, m: mnn.MappedMaxPool(5.0)(x, m), lambda x, m: mnn.MappedAvgPool(5.0)(x, m),
    lambda x, m: mnn.MappedAvgUnpool(5.0)(x, 8, 9, m),
])
def test_sizes_are_converted_to_whole_numbers(call):
    with pytest.raises(RuntimeError, match="CUDA only"):  # (the op took the call; there is no CPU path)
        call(torch.zeros(1, 2, 4, 6), torch.zeros(4, 6, 5, 2))
