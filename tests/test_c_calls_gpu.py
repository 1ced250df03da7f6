"""Calls of the C library in forms that the Python entry points do not produce."""

import ctypes

import pytest
import torch

from selective_attention_b200 import _lib, kernels

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _problem(q, k, v):
    return kernels._problem(q, k, v, _lib.ENGINE_TCGEN05, 1)


@pytest.mark.parametrize("heads,dim", [(1, 64), (3, 64), (1, 128), (3, 128)])
def test_backward_writes_gradients_at_any_element(heads, dim):
    """dq, dk and dv of the plain backward are contiguous; where they begin is the caller's affair."""
    lib = _lib.load()
    g = torch.Generator("cpu").manual_seed(dim + heads)
    b, t = 2, 200
    q, k, v, d_out = (torch.randn(b, heads, t, dim, generator=g).bfloat16().cuda() for _ in range(4))
    out, lse2, carry, *_ = kernels._forward(q, k, v, True, 1, 0, 0)
    p = _problem(q, k, v)
    need = lib.sa_backward_workspace_bytes(ctypes.byref(p))
    workspace = torch.empty(need, dtype=torch.uint8, device="cuda")
    n = q.numel()
    got = []
    for first in (8, 9, 11, 12):                   # elements of 2 bytes: at 16, 2, 6 and 8 bytes of a boundary
        flat = [torch.full((n + 32,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
        ptrs = [x.data_ptr() + 2 * first for x in flat]
        _lib.check("sa_backward", lib.sa_backward(ctypes.byref(p), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                                  lse2.data_ptr(), carry.data_ptr(), d_out.data_ptr(), _lib.DTYPE_BF16, *ptrs,
                                                  workspace.data_ptr(), need, _stream()))
        torch.cuda.synchronize()
        for x in flat:
            assert (x[:first] == 7).all() and (x[first + n:] == 7).all()
        got.append([x[first:first + n].float() for x in flat])
    assert _lib.device_status() == 0
    for other in got[1:]:
        for a, ref in zip(other, got[0]):
            assert float((a - ref).norm() / ref.norm()) < 2e-3         # the order of the fp32 reductions


_REFUSED_LAUNCH = """
#define _GNU_SOURCE
#include <dlfcn.h>
typedef struct { unsigned x, y, z; } dim3_t;
typedef int (*launch_t)(const void*, dim3_t, dim3_t, void**, unsigned long, void*);
static int left = -1, failed = 0;             /* launches until one is refused */
void refuse_launch(int n) { left = n; failed = 0; }
int cudaLaunchKernel(const void* f, dim3_t g, dim3_t b, void** a, unsigned long smem, void* s) {
  if (left >= 0 && left-- == 0) return failed = 2;                       /* cudaErrorMemoryAllocation */
  return ((launch_t)dlsym(RTLD_NEXT, "cudaLaunchKernel"))(f, g, b, a, smem, s);
}
int cudaGetLastError(void) {
  const int e = failed;
  failed = 0;
  return e ? e : ((int (*)(void))dlsym(RTLD_NEXT, "cudaGetLastError"))();
}
"""

_RETRIED_CHUNK = """
import ctypes, sys
import torch
from selective_attention_b200 import _lib, mixers
shim = ctypes.CDLL(sys.argv[1])
heads, dim, per_head, skip = (int(x) for x in sys.argv[2:])
g = torch.Generator("cpu").manual_seed(3)
first, total = 300, 330
q, k, v = (torch.randn(1, heads, total, dim, generator=g).bfloat16().cuda() for _ in range(3))
slot = mixers.SelectiveAttentionSlot(n_heads=heads, context_length=total, per_head=bool(per_head))
_, cache = slot.begin_cache(*(x[:, :, :first] for x in (q, k, v)))
new = [x[:, :, first:] for x in (q, k, v)]
want = {key: (x.clone() if torch.is_tensor(x) else x) for key, x in cache.items()}
before = _lib.launch_count()
rows = slot.extend_cache(*new, want, skip_dead_tiles=bool(skip))
launches = _lib.launch_count() - before
history = cache["selected"].clone()
for n in range(launches):
    shim.refuse_launch(n)
    try:
        slot.extend_cache(*new, cache, skip_dead_tiles=bool(skip))
        sys.exit(f"launch {n} was not refused")
    except _lib.LibraryError as e:
        assert e.status == 5, e
    assert cache["len"] == first and torch.equal(cache["selected"], history), n
shim.refuse_launch(-1)
assert torch.equal(slot.extend_cache(*new, cache, skip_dead_tiles=bool(skip)), rows)
assert torch.equal(cache["selected"], want["selected"]) and cache["len"] == total
print("launches", launches)
"""


@pytest.mark.parametrize("heads,dim,per_head,skip", [(2, 64, 0, 0), (2, 64, 1, 1), (160, 64, 0, 1), (2, 128, 0, 0)])
def test_a_chunk_whose_call_fails_can_be_tried_again(heads, dim, per_head, skip, tmp_path):
    """Whichever of its launches is refused (by a stand-in for the runtime's launch function, in a process of its own), the
    history of the cache is what it was, and the chunk counts once when it goes through."""
    import os
    import subprocess
    import sys

    source, shim = tmp_path / "refuse.c", tmp_path / "refuse.so"
    source.write_text(_REFUSED_LAUNCH)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(source), "-o", str(shim), "-ldl"], check=True)
    package = os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__)))
    res = subprocess.run([sys.executable, "-c", _RETRIED_CHUNK, str(shim), *map(str, (heads, dim, per_head, skip))],
                         env=dict(os.environ, LD_PRELOAD=str(shim), PYTHONPATH=package), capture_output=True, text=True, timeout=240)
    assert res.returncode == 0 and f"launches {5 if skip else 3}" in res.stdout, res.stdout + res.stderr
