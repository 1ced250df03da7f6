"""What callers do with a decode cache besides stepping it: copy and save it, give it other tensors or another stream, capture a
step.  Every form is compared with a cache that holds nothing but the tensors."""

import copy
import io

import pytest
import torch

from selective_attention_b200 import _lib, mixers

pytestmark = pytest.mark.gpu

B, H, D, CAPACITY = 2, 4, 64, 700


def _rows(seed, n=1):
    g = torch.Generator("cpu").manual_seed(seed)
    return tuple(torch.randn(B, H, n, D, generator=g).bfloat16().cuda() for _ in range(3))


def _cache(seed=0, length=600, live_keys=True):
    slot = mixers.SelectiveAttentionSlot(n_heads=H, context_length=CAPACITY)
    return slot, slot.begin_cache(*_rows(seed, length), live_keys=live_keys)[1]


def _bare(cache):
    """The same cache as a caller would write it down: tensors of its own and the length."""
    return {key: cache[key].clone() for key in ("k", "v", "selected", "key_norms") if key in cache} | {"len": cache["len"]}


def _same(slot, cache, bare, seeds):
    for seed in seeds:
        assert torch.equal(slot.step_cache(*_rows(seed), cache), slot.step_cache(*_rows(seed), bare))
    for key in ("k", "v", "selected", "key_norms"):
        assert key not in cache or torch.equal(cache[key], bare[key]), key
    assert cache["len"] == bare["len"] and _lib.device_status() == 0


def _saved(cache):
    file = io.BytesIO()
    torch.save(cache, file)
    file.seek(0)
    return torch.load(file, weights_only=False)


@pytest.mark.parametrize("branch", [copy.deepcopy, copy.copy, _saved])
def test_a_cache_that_was_stepped_can_be_branched(branch):
    slot, cache = _cache()
    slot.step_cache(*_rows(1), cache)
    other = branch(cache)
    if branch is copy.copy:                        # the same tensors until they are replaced
        other.update(_bare(cache))
    bare, bare_other = _bare(cache), _bare(other)
    for seed in range(2, 6):                       # the two by turns, with other tokens
        _same(slot, cache, bare, [seed])
        _same(slot, other, bare_other, [seed + 100])


def test_tensors_that_change_in_place_are_looked_at_again():
    slot, cache = _cache()
    slot.step_cache(*_rows(1), cache)
    for key in ("k", "v", "selected", "key_norms"):          # another storage
        cache[key].data = cache[key].clone()
        _same(slot, cache, _bare(cache), [2, 3])
    for key in ("k", "v"):                                   # another capacity
        cache[key].data = cache[key][:, :, :650].contiguous()
    cache["selected"].data = cache["selected"][:, :, :650].contiguous()
    with pytest.raises(ValueError, match="key_norms"):
        slot.step_cache(*_rows(4), cache)
    cache["key_norms"].data = cache["key_norms"][:, :, :650].contiguous()
    _same(slot, cache, _bare(cache), [4, 5])
    cache["k"].data = cache["k"].transpose(1, 2)
    with pytest.raises(ValueError):
        slot.step_cache(*_rows(6), cache)


def test_selections_swapped_between_steps():
    """One set of keys and values, several selections by turns."""
    slot, cache = _cache(live_keys=False)
    beams = [cache["selected"].clone() * s for s in (0.5, 1.0, 2.0)]
    want = [dict(_bare(cache), selected=x.clone()) for x in beams]
    for seed in range(3):
        for beam, bare in zip(beams, want):
            cache["selected"], cache["len"] = beam, bare["len"]
            assert torch.equal(slot.step_cache(*_rows(seed), cache), slot.step_cache(*_rows(seed), bare))
            assert torch.equal(beam, bare["selected"])


def test_steps_on_one_stream_and_then_on_another():
    slot, cache = _cache()
    bare = _bare(cache)
    side = torch.cuda.Stream()
    for seed in range(4):
        with torch.cuda.stream(side if seed & 1 else torch.cuda.current_stream()):
            got = slot.step_cache(*_rows(seed), cache)
        torch.cuda.synchronize()
        assert torch.equal(got, slot.step_cache(*_rows(seed), bare))


def test_a_step_captured_first_leaves_nothing_behind():
    """The first step of a cache is captured in a pool whose memory holds ones; the eager step after it, and the graph's
    replays, find their scratch as they need it."""
    slot, cache = _cache()
    slot.step_cache(*_rows(0), _bare(cache))                 # the library's set-up on this device
    bare, length = _bare(cache), cache["len"]
    dirty, graph = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(dirty):
        torch.ones(250_000, device="cuda")                   # below 1 MiB: where the allocator puts small requests
    dirty.replay()
    q, k, v = _rows(7)
    with torch.cuda.graph(graph, pool=dirty.pool()):
        y = slot.step_cache(q, k, v, cache)
    cache["len"] = length
    dirty.replay()
    _same(slot, cache, bare, [8])
    again = _bare(cache)
    for key in ("k", "v", "selected", "key_norms"):
        cache[key].copy_(again[key])
    again["len"] = length                                    # where the graph's step stands
    for _ in range(2):
        dirty.replay()
        graph.replay()
        assert torch.equal(y, slot.step_cache(q, k, v, again))
        assert torch.equal(cache["selected"], again["selected"])
        again["len"] = length


def _broadcast(x):
    return x[:, :1].expand(B, H, -1, -1)


def _broadcast_all(x):
    return x[:1, :1].expand(B, H, -1, -1)


def _overlapping(x):                              # every head one token further along the same rows
    n = x.shape[2]
    rows = x.reshape(B, H * n, D).contiguous()
    return rows.as_strided((B, H, n, D), (rows.stride(0), D, D, 1))


def _token_major(x):                              # (B, T, H, D) memory
    return x.transpose(1, 2).contiguous().transpose(1, 2)


def _misaligned(x):
    n = x.numel()
    flat = torch.empty(n + 3, dtype=x.dtype, device=x.device)
    flat[3:] = x.reshape(-1)
    return flat[3:].view(x.shape)


def _odd_pitch(x):                                # rows of D + 2 elements
    wide = torch.zeros(*x.shape[:3], D + 2, dtype=x.dtype, device=x.device)
    wide[..., :D] = x
    return wide[..., :D]


@pytest.mark.parametrize("form", [_broadcast, _broadcast_all, _overlapping, _token_major, _misaligned, _odd_pitch])
@pytest.mark.parametrize("n", [1, 20])
def test_new_rows_of_any_strides(form, n):
    slot, cache = _cache()
    bare, length = _bare(cache), cache["len"]
    q, k, v = _rows(9, n)
    k, v = form(k), form(v)
    got = slot.extend_cache(q, k, v, cache)
    want = slot.extend_cache(q, k.contiguous(), v.contiguous(), bare)
    assert torch.equal(got, want)
    for key in ("k", "v", "selected", "key_norms"):
        assert torch.equal(cache[key], bare[key]), key
    assert torch.equal(cache["k"][:, :, length:length + n], k) and torch.equal(cache["v"][:, :, length:length + n], v)
    assert not cache["k"][:, :, length + n:].any() and not cache["v"][:, :, length + n:].any()
    torch.cuda.synchronize()
    assert torch.ones(3, device="cuda").sum() == 3           # no error of a refused copy left for the next call
    # one sequence: the batch stride says nothing about the heads'
    slot, one = mixers.SelectiveAttentionSlot(n_heads=H, context_length=CAPACITY), {}
    for key in ("k", "v", "selected"):
        one[key] = bare[key][:1].contiguous()
    one["len"] = length
    two = {key: (x.clone() if torch.is_tensor(x) else x) for key, x in one.items()}
    assert torch.equal(slot.extend_cache(q[:1], k[:1], v[:1], one), slot.extend_cache(q[:1], k[:1].contiguous(), v[:1].contiguous(), two))
    assert torch.equal(one["k"], two["k"]) and torch.equal(one["v"], two["v"])


def test_new_rows_that_were_written_into_the_cache():
    slot, cache = _cache()
    bare, length, n = _bare(cache), cache["len"], 17
    q, k, v = _rows(10, n)
    for key, x in (("k", k), ("v", v)):
        cache[key][:, :, length:length + n] = x
    rows = [cache[key][:, :, length:length + n] for key in ("k", "v")]
    assert torch.equal(slot.extend_cache(q, *rows, cache), slot.extend_cache(q, k, v, bare))
    assert torch.equal(cache["k"], bare["k"]) and torch.equal(cache["v"], bare["v"])


@pytest.mark.parametrize("form", [torch.clone, _broadcast, _token_major, _odd_pitch])
def test_a_new_cache_is_zero_behind_its_prompt(form):
    for x in [torch.full((B, H, CAPACITY, D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2)]:
        del x                                     # memory that the cache may be given
    q, k, v = _rows(11, 130)
    slot = mixers.SelectiveAttentionSlot(n_heads=H, context_length=CAPACITY)
    _, cache = slot.begin_cache(q, form(k), form(v))
    for key in ("k", "v", "selected"):
        assert not cache[key][:, :, 130:].any()
    assert torch.equal(cache["k"][:, :, :130], form(k)) and torch.equal(cache["v"][:, :, :130], form(v))
