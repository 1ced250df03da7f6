"""The differentiable calls as the rest of torch sees them: recorded by a trace, transformed, their saved tensors moved."""

import pytest
import torch

import selective_oracle as oracle
from selective_attention_b200 import kernels, mixers

pytestmark = pytest.mark.gpu


def _inputs(seed, heads=4, seq=200, dim=64, dtype=torch.bfloat16):
    g = torch.Generator("cpu").manual_seed(seed)
    return tuple(torch.randn(2, heads, seq, dim, generator=g).to(dtype).cuda() for _ in range(3))


def _plain(q, k, v):
    return kernels.selective_attention(q, k, v, exempt=3)


def _layer(q, k, v):
    return mixers.SelectiveAttentionSlot(n_heads=4, context_length=200).attend(q, k, v)[0].float()


def _packed(q, k, v):
    return kernels.selective_attention_packed(torch.stack([x.transpose(1, 2) for x in (q, k, v)], dim=2)).float()


@pytest.mark.filterwarnings("ignore")              # what tracing says of shapes and of itself
@pytest.mark.parametrize("call,dtype,dim", [(_plain, torch.bfloat16, 64), (_plain, torch.float32, 32), (_layer, torch.bfloat16, 64),
                                            (_packed, torch.bfloat16, 64)])
def test_a_traced_call_follows_its_inputs(call, dtype, dim):
    first, second = (_inputs(seed, dim=dim, dtype=dtype) for seed in (1, 2))
    traced = torch.jit.trace(lambda q, k, v: 2.0 * call(q, k, v), first, check_trace=False)
    x, y = ([t.clone().requires_grad_(True) for t in second] for _ in range(2))
    got, want = traced(*x), 2.0 * call(*y)
    assert torch.equal(got, want)
    for a, b in zip(torch.autograd.grad(got.square().sum(), x), torch.autograd.grad(want.square().sum(), y)):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-3        # the order of the fp32 reductions


def test_the_autograd_function_and_the_call_agree():
    q, k, v = _inputs(3)
    assert issubclass(kernels._SelectiveAttentionFn, torch.autograd.Function)
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    got = kernels._SelectiveAttentionFn.apply(*x, None, None, 32, 4, 32, 4, 1, None, None, None, 1)
    assert torch.equal(got, kernels.selective_attention(q, k, v))
    grads = torch.autograd.grad(got.sum(), x)
    ref = oracle.attention_grads(*(t.float().cpu() for t in (q, k, v)), torch.ones(got.shape))
    for a, b in zip(grads, ref[1:]):
        assert float((a.float().cpu() - b).norm() / b.norm()) < 2e-2


def test_transforms_are_refused():
    q, k, v = _inputs(4)
    with pytest.raises(RuntimeError):
        torch.func.vmap(kernels.selective_attention)(*(x[None] for x in (q, k, v)))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda a: kernels.selective_attention(a, k, v).sum())(q)
    with torch.autograd.forward_ad.dual_level(), pytest.raises(RuntimeError):
        kernels.selective_attention(torch.autograd.forward_ad.make_dual(q, torch.ones_like(q)), k, v)


def test_saved_tensors_may_be_moved():
    x = [t.requires_grad_(True) for t in _inputs(5)]
    want = torch.autograd.grad(kernels.selective_attention(*x).sum(), x)
    with torch.autograd.graph.save_on_cpu():
        out = kernels.selective_attention(*x)
    for a, b in zip(torch.autograd.grad(out.sum(), x), want):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-3


@pytest.mark.parametrize("call,dtype,dim", [(_plain, torch.bfloat16, 64), (_plain, torch.float32, 32), (_packed, torch.bfloat16, 64)])
def test_saved_bytes_may_come_back_at_any_address(call, dtype, dim):
    """A hook that keeps saved bytes one byte into a buffer of its own: the statistics among them are floats."""
    x = [t.requires_grad_(True) for t in _inputs(7, dim=dim, dtype=dtype)]
    want = torch.autograd.grad(call(*x).sum(), x)

    def pack(t):
        if t.dtype != torch.uint8:
            return t
        flat = torch.empty(t.numel() + 1, dtype=torch.uint8, device=t.device)
        flat[1:] = t
        return flat

    def unpack(t):
        return t[1:] if t.dtype == torch.uint8 else t

    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        out = call(*x)
    for a, b in zip(torch.autograd.grad(out.sum(), x), want):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2e-3


@pytest.mark.parametrize("call", [_plain, _layer, _packed])
def test_gradients_kept_for_a_graph_are_constants_where_the_cotangent_is_one(call):
    """create_graph with a cotangent that has no graph: the gradients are plain tensors, and what is built on them can be
    differentiated with respect to everything else."""
    x = [t.requires_grad_(True) for t in _inputs(6)]
    scale = torch.ones((), device="cuda", requires_grad=True)
    out = call(*x)
    for create_graph in (False, True):
        (dq,) = torch.autograd.grad(out, x[:1], torch.ones_like(out), create_graph=create_graph, retain_graph=True)
        assert not dq.requires_grad
    (scale * dq.float()).square().sum().backward()
    assert torch.isfinite(scale.grad) and scale.grad > 0
