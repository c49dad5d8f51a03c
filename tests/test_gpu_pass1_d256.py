"""Pass 1 at head_dim 256 over items of one tile, several items per CTA and walks of a few tiles (an item is half a key block, its rings run
on across items): dK, dV, the dS' codes and psi against the oracle, and against the same call made one head at a time."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,causal", [(1, 128, 1, 1, True), (5, 128, 32, 8, True), (1, 256, 3, 1, False), (1, 640, 2, 1, True), (2, 384, 30, 10, True)])
def test_pass1_d256(B, N, H, Hk, causal):
    q, k, v, dO = O.make_inputs(B, N, H, Hk, 256, 2041)
    r = O.attention_fwd_bwd(q, k, v, dO, causal, "stale", fwd_tile_keys=128, pv="group", debug=True)
    args = [r[n].cuda() for n in ("Q8", "K8", "V8", "dO8", "Q8s", "K8s", "V8s", "dO8s", "LSE", "delta")]
    dk, dv, ws = _lib.bwd_pass1(*args, B, H, Hk, causal)
    assert _lib.device_status() == 0
    nb = N // 128
    psi = ws[1].view(B * H, 2 * nb, 2 * nb).cpu()
    seen = torch.ones(2 * nb, 2 * nb, dtype=torch.bool)
    if causal:
        seen = seen.tril()
        above = psi.view(B * H, nb, 2, nb, 2)[:, range(nb), 0, range(nb), 1]     # the quarter of a diagonal tile above the diagonal: a zero tile
        assert (above == 0).all()
    assert torch.allclose(psi[:, seen], r["psi"][:, seen], rtol=2e-3, atol=0)
    tiles = torch.ones(nb, nb, dtype=torch.bool)
    if causal:
        tiles = tiles.tril()                                                      # those above are not written
    # kernel tile [row block, key block, key 128, row 128]  <-  oracle [m-block, key half block, row 64, key 64]
    codes = ws[0].view(B * H, nb, nb, 128, 128)
    ref = r["dS8"].view(torch.uint8).view(B * H, nb, 2, nb, 2, 64, 64).permute(0, 1, 3, 4, 6, 2, 5).reshape(B * H, nb, nb, 128, 128)
    a, b = (t[:, tiles].contiguous().view(torch.float8_e4m3fn).float() for t in (codes.cpu(), ref))
    # a code that the approximate exponential moves goes one step, at most 2^-3 of itself: the bound is 0.16 % of them
    assert O.rel(a, b) < 5e-3, O.rel(a, b)
    if causal:
        masked = codes.cpu()[:, range(nb), range(nb), 64:, :64].contiguous().view(torch.float8_e4m3fn).float()
        assert (masked == 0).all(), "the quarter of a diagonal tile above the diagonal"
    for name, a, tol in (("dKh", dk, 3e-3), ("dVh", dv, 2e-3)):                   # bf16 rounding, and codes that the approximate exponential moves
        ref = r[name].to(torch.bfloat16).view(B, H, N, 256).permute(0, 2, 1, 3)
        assert O.rel(a.cpu(), ref) < tol, (name, O.rel(a.cpu(), ref))
    dk2, dv2 = torch.full_like(dk, float("nan")), torch.full_like(dv, float("nan"))
    rep, by_head, seen, tiles = H // Hk, codes.view(B, H, nb, nb, 128, 128), seen.cuda(), tiles.cuda()
    for h0 in range(0, H, rep):
        _, _, ws2 = _lib.bwd_pass1(*args, B, H, Hk, causal, h0=h0, hcount=rep, out=(dk2, dv2))
        part = ws2[0].view(B, rep, nb, nb, 128, 128)
        assert torch.equal(part[:, :, tiles], by_head[:, h0:h0 + rep][:, :, tiles]), "dS' codes of a head range"
        part = ws2[1].view(B, rep, 2 * nb, 2 * nb)
        assert torch.equal(part[:, :, seen], ws[1].view(B, H, 2 * nb, 2 * nb)[:, h0:h0 + rep][:, :, seen]), "psi of a head range"
    assert torch.equal(dk, dk2) and torch.equal(dv, dv2), "the walk over several items changed the bits"
