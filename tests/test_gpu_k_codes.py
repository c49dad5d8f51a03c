"""The K quantizer: blocks of special values against the definition, and the composite forward's K codes (several key blocks per thread
block from 4096 keys on) against the separate entry points, bit for bit."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [128, 256])
def test_special_blocks(D):
    rk = O.blocks(D)[1]
    g = torch.Generator().manual_seed(D)
    N = 16 * 128
    x = torch.randn(1, N // rk, rk, D, generator=g).to(torch.bfloat16)
    km = torch.randn(1, D, generator=g) * 0.1
    km[0, ::3] = 0.0
    x[0, 0] = 0.0
    x[0, 1] = -0.0
    x[0, 2, ::2] = -0.0
    x[0, 3, 5, 7] = float("nan")
    x[0, 4, 9, 1], x[0, 4, 3, 3] = float("inf"), float("-inf")
    x[0, 5, 2, 2], x[0, 5, 4, 4] = float("-inf"), float("nan")
    x[0, 6] = float("nan")
    x[0, 7] *= 2.0 ** 70
    x[0, 8] *= 2.0 ** -70
    x[0, 9] = 3.0e38
    xb = (x.float() - km[:, None, None, :]).view(1, N // rk, rk * D)
    amax = torch.where(xb.isnan(), torch.zeros_like(xb), xb.abs()).amax(dim=-1)
    s = torch.maximum(amax, torch.tensor(O.TINY)) / torch.tensor(448.0)
    q = (xb / s[..., None])
    q = torch.where(q.isnan(), torch.full_like(q, -448.0), q.clamp(-448.0, 448.0))
    codes, scales = _lib.quant(1, x.view(1, N, 1, D).cuda(), km.cuda())
    assert torch.equal(scales.cpu(), s)
    assert torch.equal(codes.cpu().view(torch.uint8).view(-1), O.to_e4m3(q).view(torch.uint8).view(-1))


@pytest.mark.parametrize("B,N,Hk", [(5, 4096, 15), (1, 4096, 2), (3, 4352, 8), (2, 8192, 5), (2, 8448, 3), (9, 256, 40), (4, 3840, 9)])
def test_composite_equals_separate(B, N, Hk):
    g = torch.Generator(device="cuda").manual_seed(N)
    k = torch.randn(B, N, Hk, 128, generator=g, device="cuda", dtype=torch.bfloat16) + 0.5
    k[0, N // 2, 0, 3] = float("nan")
    q = v = torch.randn(B, N, Hk, 128, generator=g, device="cuda", dtype=torch.bfloat16)
    _, _, _, _, K8, K8s, _, _ = _lib.attn_forward(q, k, v, True)
    c, s = _lib.quant(1, k, _lib.kmean(k))
    assert torch.equal(K8s, s) or torch.equal(K8s.view(torch.int32), s.view(torch.int32))
    assert torch.equal(K8.view(torch.uint8), c.view(torch.uint8))
