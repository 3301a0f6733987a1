"""Native calls that stand in for PyTorch operations: only where nobody looks on who would see the allocations of the call and not
its kernel, and only on tensors with memory of their own."""
import types

import pytest
import torch
import torch.nn.functional as F
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx

from asdl_b200 import ops
from asdl_b200.models import layers, resnet_tiny


class _NoExtension:
    """In the place of the extension: every native call fails, before it can touch an address."""

    def __getattr__(self, name):
        def call(*args):
            raise AssertionError(f'native call {name}')
        return call


def test_casts_of_tensors_without_memory_are_left_to_pytorch(monkeypatch):
    monkeypatch.setattr(ops, 'extension', _NoExtension)
    with FakeTensorMode(), torch.device('cuda'):
        model = resnet_tiny(fused=True).eval()
        x = torch.empty(2, 3, 64, 64, dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last)
        with layers.grouped_bf16_weights(model):
            assert model.conv1.weight.dtype == torch.bfloat16 and model(x).shape == (2, 10)
        # the way back: a gradient of a linear layer (transposed) and one of a convolution
        shapes = [(32, 16), (8, 4, 3, 3)]
        ctx = types.SimpleNamespace(meta=[(torch.Size(s), torch.empty(s).stride()) for s in shapes])
        grads = [torch.empty(16, 32, dtype=torch.bfloat16).t(), torch.empty(8, 4, 3, 3, dtype=torch.bfloat16)]
        back = layers._GroupedCast.backward(ctx, *grads)
        assert all(g.dtype == torch.float32 and g.shape == s for g, s in zip(back, shapes))


@pytest.mark.parametrize('device', ['cpu', pytest.param('cuda', marks=pytest.mark.gpu)])
@pytest.mark.parametrize('backend', ['eager', 'aot_eager'])
def test_grouped_casts_compile(backend, device):
    """In a compiled call the casts are operations that the compiler can follow, with the results of the call itself."""
    torch._dynamo.reset()
    model = torch.nn.Sequential(torch.nn.Conv2d(8, 16, 3, bias=False), torch.nn.Flatten(), torch.nn.Linear(16 * 9, 10, bias=False))
    model = model.to(device).to(memory_format=torch.channels_last)
    x = torch.randn(4, 8, 5, 5, device=device).to(torch.bfloat16)

    def call(inp):
        with layers.grouped_bf16_weights(model):
            return model(inp).float()

    want, got = call(x), torch.compile(call, backend=backend)(x)
    torch.testing.assert_close(got, want, rtol=1e-2, atol=1e-2)
    grads = [torch.autograd.grad(y.square().sum(), list(model.parameters())) for y in (want, got)]
    for a, b in zip(*grads):
        assert a.dtype == b.dtype == torch.float32 and (a - b).norm() <= 2e-2 * a.norm()


def test_tensors_without_memory_do_not_reach_a_kernel(monkeypatch):
    monkeypatch.setattr(ops, 'extension', _NoExtension)
    with FakeTensorMode(), torch.device('cuda'):
        x, square = torch.empty(12, 8), torch.empty(8, 8)
        assert ops.gram(x).shape == (8, 8) and ops.kron_apply(torch.empty(12, 12), x, square).shape == (12, 8)
        assert ops.matmul_tn(x, x).shape == (8, 8) and ops.eigh(square)[0].shape == (8,)
        norm = layers.FusedBatchNorm2d(8, act='relu')
        act = torch.empty(2, 8, 5, 5, dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last)
        assert norm(act, residual=act).shape == act.shape
        assert not ops.layer_norm_supported(torch.empty(4, 256, dtype=torch.bfloat16), torch.empty(256), torch.empty(256))
        assert torch.nn.Parameter(x).is_cuda and not ops.cuda_kernels_enabled(torch.nn.Parameter(x))


def test_calls_that_are_looked_at_are_not_native():
    seen = []

    def look(x):
        seen.append(ops.unobserved(x))
        return x * 2

    x = torch.ones(3)
    assert ops.unobserved(x) and ops.unobserved(torch.nn.Parameter(x))
    for options in ({'tracing_mode': 'real'}, {'tracing_mode': 'fake'}, {'pre_dispatch': True}):
        make_fx(look, **options)(x)
    torch.jit.trace(look, (x,), check_trace=False)
    torch.func.vmap(look)(x)
    torch.func.jvp(look, (x,), (x,))
    with torch.autograd.forward_ad.dual_level():
        look(torch.autograd.forward_ad.make_dual(x, x))
    with FakeTensorMode():
        fake = torch.empty(3)
    look(fake)   # outlives its mode
    assert len(seen) == 8 and not any(seen)


@pytest.mark.gpu
def test_recorded_graphs_hold_the_casts():
    """A graph that is recorded on real tensors computes with the weights of the model."""
    model = torch.nn.Sequential(torch.nn.Linear(32, 64, bias=False), torch.nn.Linear(64, 16, bias=False)).to('cuda')

    def call(inp):
        with layers.grouped_bf16_weights(model):
            return model(inp)

    with torch.no_grad():
        x = [torch.randn(8, 32, device='cuda').to(torch.bfloat16) for _ in range(2)]
        graph = make_fx(call)(x[0])
        assert any('copy' in str(n.target) for n in graph.graph.nodes)
        for inp in x:
            assert torch.equal(graph(inp), call(inp))


@pytest.mark.gpu
def test_casts_of_tensors_that_pytorch_has_to_look_into():
    x = torch.randn(64, device='cuda')
    got = torch.empty(64, device='cuda', dtype=torch.bfloat16)
    ops.extension().cast_many([got], [torch._neg_view(x)])
    assert torch.equal(got, -x.bfloat16())
    with FakeTensorMode():
        fake = [torch.empty(64, device='cuda', dtype=t) for t in (torch.bfloat16, torch.float32)]
        ops.extension().cast_many(fake[:1], fake[1:])


@pytest.mark.gpu
@pytest.mark.parametrize('options', [{'tracing_mode': 'real'}, {'pre_dispatch': True}])
def test_recorded_graphs_hold_the_pooling(options):
    """A graph that is recorded on real tensors pools the activations that it is given."""
    pool = layers.FusedMaxPool2d(3, stride=2, padding=1)
    with torch.no_grad():
        x = [torch.randn(2, 8, 9, 9, device='cuda').to(torch.bfloat16).contiguous(memory_format=torch.channels_last) for _ in range(2)]
        assert pool._native(x[0])
        graph = make_fx(lambda inp: pool(inp), **options)(x[0])
        for inp in x:
            assert torch.equal(graph(inp), F.max_pool2d(inp, 3, 2, 1))


@pytest.mark.gpu
@pytest.mark.parametrize('layer,shape', [(torch.nn.Conv2d(8, 16, 3), (2, 8, 5, 5)), (torch.nn.Linear(32, 16), (4, 32))])
def test_gradients_of_grouped_casts_are_not_differentiated_without_their_share(layer, shape):
    """A second derivative through the casts is refused, as PyTorch refuses one of copies of tensor lists; the bias has one, and the
    sum of both would be the bias's alone."""
    layer = layer.to('cuda')
    x = torch.randn(shape, device='cuda', dtype=torch.bfloat16)
    with layers.grouped_bf16_weights(layer), torch.autocast('cuda', dtype=torch.bfloat16):
        y = layer(x).float()
    grads = torch.autograd.grad(y.square().sum(), (layer.weight, layer.bias), create_graph=True)
    with pytest.raises(RuntimeError, match='_foreach_copy_'):
        torch.autograd.grad(sum(g.sum() for g in grads), layer.weight)
