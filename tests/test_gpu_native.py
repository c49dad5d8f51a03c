"""The native eager route (csrc/dm_torch.cpp) against the traceable one (autograd function over the custom ops) on the same
inputs: outputs, gradients in each layout and mode, the refusal of a second differentiation."""
import pytest
import torch

import delta_matching_b200 as dm
from delta_matching_b200 import attn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["matched", "stale"])
@pytest.mark.parametrize("head_major", [False, True])
@pytest.mark.parametrize("D,N,H,Hk", [(128, 256, 2, 2), (128, 768, 6, 2), (256, 384, 3, 1)])
def test_native_route_equals_the_traceable_route(mode, head_major, D, N, H, Hk):
    g = torch.Generator("cpu").manual_seed(41)
    dims = (lambda h: (2, h, N, D)) if head_major else (lambda h: (2, N, h, D))
    q, k, v = (torch.randn(*dims(h), generator=g).to("cuda", torch.bfloat16).requires_grad_(True) for h in (H, Hk, Hk))
    do = torch.randn(2, N, H, D, generator=g).to("cuda", torch.bfloat16)
    got = attn.attention(q, k, v, True, None, mode, head_major)
    view = (lambda t: t) if head_major else (lambda t: t.transpose(1, 2))
    ref = attn._DMAttn.apply(view(q), view(k), view(v), True, mode)
    assert torch.equal(got, ref)
    for a, b in zip(torch.autograd.grad(got, (q, k, v), do), torch.autograd.grad(ref, (q, k, v), do)):
        assert a.shape == b.shape and torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(attn.attention(q, k, v, True, None, mode, head_major), got)


def test_a_second_differentiation_is_refused():
    q, k, v = (torch.randn(1, 256, 2, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    o = dm.dm_attn_func(q, k, v, causal=True)
    do = torch.randn_like(o).requires_grad_(True)
    gq, = torch.autograd.grad(o, q, do, create_graph=True)
    with pytest.raises(RuntimeError, match="twice"):
        gq.sum().backward()
