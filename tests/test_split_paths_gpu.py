"""The forward variants that only larger grids reach (two heads of a selector, or two rows that each select for
themselves, in one CTA), second differentiation, the newest key of a decode step, the split
walk of a short chunk after a long cache, and
the exact-product engine with one and two teams a CTA."""

import pytest
import torch

import selective_oracle as oracle
from selective_attention_b200 import _lib, kernels, mixers

pytestmark = pytest.mark.gpu


def _inputs(batch, heads, seq, dim, scale, seed):
    g = torch.Generator("cpu").manual_seed(seed)
    qk = (scale * torch.randn(batch, heads, seq, dim, generator=g) for _ in range(2))
    return tuple(x.bfloat16() for x in (*qk, *(torch.randn(batch, heads, seq, dim, generator=g) for _ in range(2))))


def _rel(got, want):
    return float((got.float().cpu() - want).norm() / want.norm().clamp_min(1e-30))


# more than 148 (query tile, head) pairs: below that the forward takes one head a CTA
@pytest.mark.parametrize("batch,heads,seq,exempt,scale", [
    (1, 150, 50, 1, 1.0), (1, 76, 129, 3, 1.0), (2, 38, 257, 1, 0.3), (1, 22, 1000, 140, 0.3),          # two heads of a selector
    (150, 1, 50, 1, 1.0), (76, 1, 129, 3, 1.0), (76, 1, 257, 1, 0.3), (22, 1, 1000, 140, 0.3),          # two rows, each its own
])
def test_two_heads_a_cta(batch, heads, seq, exempt, scale):
    q, k, v, w = _inputs(batch, heads, seq, 64, scale, seq + heads)
    want = oracle.attention_grads(q.float(), k.float(), v.float(), w.float(), exempt)
    qq, kk, vv = (x.cuda().requires_grad_(True) for x in (q, k, v))
    out = kernels.selective_attention(qq, kk, vv, exempt=exempt)
    grads = torch.autograd.grad(out, (qq, kk, vv), w.cuda().float())
    _, aux = kernels.selective_attention_forward(q.cuda(), k.cuda(), v.cuda(), return_aux=True, exempt=exempt)
    for got, ref in zip((out.detach(), *grads), want):
        assert _rel(got, ref) < 1e-2
    _, total = kernels.selective_logits(q.float(), k.float(), exempt)
    torch.testing.assert_close(aux["selected_total"].cpu(), total, atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("per_head", [False, True])
def test_two_heads_a_cta_in_a_continued_prefill_and_in_bf16(per_head):
    heads, first, total = 76, 200, 460
    q, k, v, w = (x.cuda() for x in _inputs(1, heads, total, 64, 0.5, 7))
    slot = mixers.SelectiveAttentionSlot(n_heads=heads, context_length=total, per_head=per_head)
    whole, _ = slot.begin_cache(q, k, v)
    y, cache = slot.begin_cache(*(x[:, :, :first] for x in (q, k, v)))
    rows = slot.extend_cache(q[:, :, first:], k[:, :, first:], v[:, :, first:], cache)
    assert whole.dtype == torch.bfloat16
    torch.testing.assert_close(torch.cat([y, rows], dim=2).float(), whole.float(), atol=2e-2, rtol=2e-2)
    qq, kk, vv = (x.clone().requires_grad_(True) for x in (q, k, v))
    layer, _ = slot.attend(qq, kk, vv)                       # the kernels write bf16 and read a bf16 cotangent
    assert layer.dtype == torch.bfloat16 and torch.equal(layer, whole)
    got = torch.autograd.grad(layer, (qq, kk, vv), w)
    views = [x.reshape(heads, 1, total, 64) if per_head else x for x in (qq, kk, vv)]
    out = kernels.selective_attention(*views).reshape(q.shape)
    want = torch.autograd.grad(out, (qq, kk, vv), w.float())
    for a, b in zip(got, want):
        assert _rel(a, b.float().cpu()) < 2e-3


@pytest.mark.parametrize("skip", [False, True])
def test_two_heads_a_cta_with_an_outside_selector_and_in_place_in_a_projection(skip):
    """More than 148 pairs in every call: two halves of the heads with a replica of the selecting head, and the heads where a
    fused projection left them, against the plain call."""
    heads, seq = 80, 600
    q, k, v, w = (x.cuda() for x in _inputs(1, heads, seq, 64, 1.0, 13))
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    whole = kernels.selective_attention(*x)
    want = torch.autograd.grad(whole, x, w.float())
    q0, k0 = (t[:, 0].clone().requires_grad_(True) for t in (q, k))
    halves = [[t[:, s].clone().requires_grad_(True) for t in (q, k, v)] for s in (slice(0, 40), slice(40, 80))]
    outs = [kernels.selective_attention(*part, selector=(q0, k0), skip_dead_tiles=skip) for part in halves]
    assert torch.equal(torch.cat(outs, dim=1), whole)
    grads = torch.autograd.grad(outs, [*halves[0], *halves[1], q0, k0], [w[:, :40].float(), w[:, 40:].float()])
    for i in range(3):
        got = torch.cat([grads[i], grads[3 + i]], dim=1).float()
        if i < 2:
            got[:, 0] += grads[6 + i].float()
        assert _rel(got, want[i].float().cpu()) < 1e-2
    qkv = torch.stack([t.transpose(1, 2) for t in (q, k, v)], dim=2).requires_grad_(True)
    y = kernels.selective_attention_packed(qkv, skip_dead_tiles=skip)
    assert torch.equal(y, whole.detach().bfloat16().transpose(1, 2).reshape(y.shape))
    (dqkv,) = torch.autograd.grad(y, qkv, w.transpose(1, 2).reshape(y.shape))
    for i in range(3):
        assert _rel(dqkv[:, :, i].transpose(1, 2), want[i].float().cpu()) < 2e-3


def test_a_second_differentiation_raises():
    q, k, v, _ = (x.cuda().requires_grad_(True) for x in _inputs(1, 2, 70, 64, 1.0, 3))
    out = kernels.selective_attention(q, k, v)
    (dq,) = torch.autograd.grad(out.square().sum(), q, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        dq.sum().backward()


@pytest.mark.parametrize("dtype,dim,norms", [(torch.bfloat16, 64, False), (torch.bfloat16, 64, True), (torch.float16, 128, False),
                                             (torch.float32, 16, False)])
@pytest.mark.parametrize("start", [0, 1020])
def test_the_newest_key_at_the_edges_of_a_decode_range(dtype, dim, norms, start):
    """The newest key comes from the call, not from the cache: alone in its stage, alone in its range, after either."""
    b, h, steps = 2, 3, 134
    g = torch.Generator("cpu").manual_seed(start + dim)
    q, k, v = ((s * torch.randn(b, h, start + steps, dim, generator=g)).to(dtype) for s in (0.5, 1.0, 1.0))
    ref = {"k": torch.zeros_like(k), "v": torch.zeros_like(v), "len": start, "selected": torch.zeros(b, 1, start + steps)}
    ref["k"][:, :, :start], ref["v"][:, :, :start] = k[:, :, :start], v[:, :, :start]
    dev = {key: (val.cuda() if torch.is_tensor(val) else val) for key, val in ref.items()}
    if norms:
        dev["key_norms"] = dev["k"].float().norm(dim=-1)
    slot = mixers.SelectiveAttentionSlot(n_heads=h, context_length=start + steps)
    for t in range(start, start + steps):
        step = [x[:, :, t:t + 1] for x in (q, k, v)]
        want = oracle.decode_step(ref, *step, groups=1)
        got = slot.step_cache(*(x.cuda() for x in step), dev)
        tol = 2e-5 if dtype == torch.float32 else 2e-2
        torch.testing.assert_close(got.float().cpu(), want, atol=tol, rtol=tol)
    torch.testing.assert_close(dev["selected"].cpu(), ref["selected"], atol=1e-3, rtol=1e-3)
    assert torch.equal(dev["k"].cpu(), k) and torch.equal(dev["v"].cpu(), v)
    if norms:
        torch.testing.assert_close(dev["key_norms"].cpu(), k.float().norm(dim=-1), rtol=1e-5, atol=1e-5)


# up to 296 (32-token block, head) pairs a CTA has two teams, and the last step of an odd number of blocks only one of them
@pytest.mark.parametrize("dim,dtype", [(16, torch.float32), (32, torch.float16), (64, torch.float32), (128, torch.float32)])
@pytest.mark.parametrize("batch,heads,seq,exempt", [(1, 2, 1, 1), (2, 3, 33, 1), (1, 2, 64, 5), (2, 2, 65, 1), (1, 3, 161, 40),
                                                    (50, 3, 33, 1), (60, 2, 97, 3)])
def test_exact_products_with_one_and_two_teams(dim, dtype, batch, heads, seq, exempt):
    g = torch.Generator("cpu").manual_seed(seq + dim)
    q, k, v, w = ((s * torch.randn(batch, heads, seq, dim, generator=g)).to(dtype) for s in (0.5, 0.5, 1.0, 1.0))
    want = oracle.attention_grads(q.float(), k.float(), v.float(), w.float(), exempt)
    qq, kk, vv = (x.cuda().requires_grad_(True) for x in (q, k, v))
    out = kernels.selective_attention(qq, kk, vv, exempt=exempt, dot_precision="ieee")
    grads = torch.autograd.grad(out, (qq, kk, vv), w.cuda().float())
    tol = 1e-5 if dtype == torch.float32 else 2e-3
    for got, ref in zip((out.detach(), *grads), want):
        torch.testing.assert_close(got.float().cpu(), ref, atol=tol * float(ref.abs().max()) + 1e-6, rtol=tol)


# few new rows: the walk over the cached keys is cut into pieces, of which a short one's last has no keys or no live ones
@pytest.mark.parametrize("heads,dim,first,second,per_head", [(2, 64, 1020, 3, False), (3, 128, 1152, 128, False), (2, 64, 4100, 300, True),
                                                             (1, 128, 2200, 1, False), (12, 64, 3000, 129, False)])
@pytest.mark.parametrize("scale", [1.0, 0.2])
def test_a_short_chunk_after_a_long_cache(heads, dim, first, second, per_head, scale):
    total = first + second
    q, k, v, _ = (x.cuda() for x in _inputs(1, heads, total, dim, scale, total))
    slot = mixers.SelectiveAttentionSlot(n_heads=heads, context_length=total, per_head=per_head)
    whole, sums = slot.attend(q, k, v, want_total=True)
    got = []
    for skip in (False, True):
        _, cache = slot.begin_cache(*(x[:, :, :first] for x in (q, k, v)))
        got.append(slot.extend_cache(*(x[:, :, first:] for x in (q, k, v)), cache, skip_dead_tiles=skip))
        torch.testing.assert_close(cache["selected"], sums, atol=1e-3, rtol=1e-4)
    assert _lib.device_status() == 0
    assert torch.equal(got[0], got[1])
    assert _rel(got[0], whole[:, :, first:].float().cpu()) < 4e-3


@pytest.mark.parametrize("heads,dim,per_head", [(2, 64, False), (2, 64, True), (2, 128, False)])
@pytest.mark.parametrize("gone", [(1, 2000), (0, 3968), (1500, 1501)])
def test_a_split_walk_over_keys_with_an_infinite_history(heads, dim, per_head, gone):
    """A key whose history is infinite has no weight; a piece of the walk may hold nothing else, or begin with it."""
    first, total = 4000, 4008
    q, k, v, _ = (x.cuda() for x in _inputs(1, heads, total, dim, 0.3, dim))
    slot = mixers.SelectiveAttentionSlot(n_heads=heads, context_length=total, per_head=per_head)
    _, cache = slot.begin_cache(*(x[:, :, :first] for x in (q, k, v)))
    cache["selected"][:, :, gone[0]:gone[1]] = float("inf")
    whole = {key: (x.clone() if torch.is_tensor(x) else x) for key, x in cache.items()}
    new = [x[:, :, first:] for x in (q, k, v)]
    got = slot.extend_cache(*new, cache)
    want = kernels.prefill_extend(whole, *new)                   # fp32 rows: one walk over all keys
    assert torch.isfinite(want).all()
    assert _rel(got, want.cpu()) < 4e-3                          # the rounding of the rows to bf16
    assert torch.equal(cache["selected"], whole["selected"])
