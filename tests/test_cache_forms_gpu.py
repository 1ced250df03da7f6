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
