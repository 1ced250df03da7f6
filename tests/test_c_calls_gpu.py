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
