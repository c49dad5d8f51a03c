"""The forward at head_dim 256 over walks of one tile, of one item and of several items per CTA (its roles carry rings of two and three
tiles across items), against the oracle and against the same call made in head ranges of one item per CTA."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,causal,scale", [(1, 128, 1, 1, True, 1), (8, 128, 64, 8, True, 1), (1, 256, 2, 1, False, 1), (1, 640, 3, 1, True, 1),
                                                     (2, 640, 32, 4, False, 1), (2, 1152, 24, 8, True, 1), (1, 384, 2, 2, True, 8)])
def test_forward_d256(B, N, H, Hk, causal, scale):
    q, k, v, _ = O.make_inputs(B, N, H, Hk, 256, 2031)
    if scale > 1:
        q = q * scale                                              # groups more than 12 binades below the row's maximum
        q[:, N // 2:N // 2 + 64] = 0                               # and a block of equal scores
    Q8, Q8s = O.quant_q(q.transpose(1, 2))
    K8, K8s, _ = O.quant_k(k.transpose(1, 2))
    V8, V8s = O.quant_v(v.transpose(1, 2))
    d = [t.cuda() for t in (Q8, K8, V8, Q8s, K8s, V8s)]
    o, lse = _lib.fwd_fp8(*d, B, H, Hk, causal)
    assert _lib.device_status() == 0
    o_ref, lse_ref = O.forward(Q8, Q8s, K8, K8s, V8, V8s, H, Hk, causal, tile_keys=128, pv="group")
    # LSE: a few roundings of exponents of up to |lse| log2 e; O: bf16 (2^-9) and single e4m3 codes that the approximate exponential moves
    assert ((lse.cpu() - lse_ref).abs() <= 2e-4 + 1e-6 * lse_ref.abs()).all()
    head = ((o.cpu().float() - o_ref.float()).norm(dim=(1, 3)) / o_ref.float().norm(dim=(1, 3))).max().item()
    assert head < 4e-3, head
    o2, lse2 = torch.zeros_like(o), torch.zeros_like(lse)
    for h0 in range(H):
        _lib.fwd_fp8(*d, B, H, Hk, causal, h0=h0, hcount=1, out=(o2, lse2))
    assert torch.equal(o, o2) and torch.equal(lse, lse2), "the walk over several items changed the bits"


@pytest.mark.parametrize("off", [1, 2, 3])
def test_scales_at_any_multiple_of_4_bytes(off):
    """Codes are promised to be 16-byte aligned, scales only to be fp32: views into one buffer give the bits of tensors of their own."""
    B, N, H, Hk = 1, 640, 3, 1
    q, k, v, _ = O.make_inputs(B, N, H, Hk, 256, 2032)
    Q8, Q8s = O.quant_q(q.transpose(1, 2))
    K8, K8s, _ = O.quant_k(k.transpose(1, 2))
    V8, V8s = O.quant_v(v.transpose(1, 2))
    codes, scales = [t.cuda() for t in (Q8, K8, V8)], [t.float().cuda() for t in (Q8s, K8s, V8s)]
    views = []
    for t in scales:
        buf = torch.full((t.numel() + 8,), float("nan"), device="cuda")
        assert buf.data_ptr() % 16 == 0
        views.append(buf[off:off + t.numel()].view(t.shape))
        views[-1].copy_(t)
    o, lse = _lib.fwd_fp8(*codes, *scales, B, H, Hk, True)
    o2, lse2 = _lib.fwd_fp8(*codes, *views, B, H, Hk, True)
    assert _lib.device_status() == 0
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
