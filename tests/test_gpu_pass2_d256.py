"""Pass 2 at head_dim 256 over walks of one tile, of one item and of several items per CTA: dQ against the sum it is, formed in fp64
from pass 1's own dS' codes and psi."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,causal", [(1, 128, 2, 1, True), (1, 384, 3, 1, False), (1, 640, 2, 2, True), (2, 1280, 16, 4, True)])
def test_pass2_d256_is_the_sum_of_the_tiles(B, N, H, Hk, causal):
    q, k, v, dO = (t.cuda() for t in O.make_inputs(B, N, H, Hk, 256, 2012))
    Q8, Q8s = _lib.quant(0, q)
    K8, K8s = _lib.quant(1, k, _lib.kmean(k))
    V8, V8s = _lib.quant(2, v)
    o, lse = _lib.fwd_fp8(Q8, K8, V8, Q8s, K8s, V8s, B, H, Hk, causal)
    dO8, dO8s, delta = _lib.quant_do(dO, o)
    _, _, ws = _lib.bwd_pass1(Q8, K8, V8, dO8, Q8s, K8s, V8s, dO8s, lse, delta, B, H, Hk, causal)
    dq = _lib.bwd_pass2(ws, K8, B, H, Hk, N, 256, causal)
    assert _lib.device_status() == 0
    nb = N // 128
    codes = ws[0].view(torch.uint8).view(B * H, nb, nb, 128, 128).view(torch.float8_e4m3fn).double()      # [.., row block, key block, key, row]
    ds = codes.permute(0, 1, 4, 2, 3).reshape(B * H, N, N)
    ds = ds * ws[1].view(B * H, N // 64, N // 64).double().repeat_interleave(64, 1).repeat_interleave(64, 2)
    if causal:                                                     # tiles above the diagonal are never written
        keep = torch.ones(nb, nb, dtype=torch.bool, device=ds.device).tril().repeat_interleave(128, 0).repeat_interleave(128, 1)
        ds = torch.where(keep, ds, torch.zeros_like(ds))
    K = K8.view(B, Hk, N, 256).double().repeat_interleave(H // Hk, 1).reshape(B * H, N, 256)
    ref = (torch.bmm(ds, K) * (0.0625 / 256.0)).view(B, H, N, 256).permute(0, 2, 1, 3)
    assert O.rel(dq.cpu(), ref.cpu()) < 3e-3                       # bf16 rounding: 2^-9 of each element


def test_psi_at_any_multiple_of_4_bytes():
    """The workspace's psi is promised to be fp32 and no more aligned: passes 1 and 2 on views at 4, 8 and 12 bytes give the bits of a buffer of its own."""
    B, N, H, Hk = 1, 384, 2, 1
    q, k, v, dO = (t.cuda() for t in O.make_inputs(B, N, H, Hk, 256, 2013))
    Q8, Q8s = _lib.quant(0, q)
    K8, K8s = _lib.quant(1, k, _lib.kmean(k))
    V8, V8s = _lib.quant(2, v)
    o, lse = _lib.fwd_fp8(Q8, K8, V8, Q8s, K8s, V8s, B, H, Hk, True)
    dO8, dO8s, delta = _lib.quant_do(dO, o)
    args = (Q8, K8, V8, dO8, Q8s, K8s, V8s, dO8s, lse, delta, B, H, Hk, True)
    _, _, ws = _lib.bwd_pass1(*args)
    dq = _lib.bwd_pass2(ws, K8, B, H, Hk, N, 256, True)
    for off in (1, 2, 3):
        buf = torch.full((ws[1].numel() + 8,), float("nan"), device="cuda")
        assert buf.data_ptr() % 16 == 0
        view = (torch.empty_like(ws[0]), buf[off:off + ws[1].numel()].view(ws[1].shape))
        _lib.bwd_pass1(*args, ws=view)
        assert torch.equal(dq, _lib.bwd_pass2(view, K8, B, H, Hk, N, 256, True)), off
    assert _lib.device_status() == 0
