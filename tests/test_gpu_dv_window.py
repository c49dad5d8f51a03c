"""dV's sum over long walks (pass 1): walks of more than 64 row tiles keep it in windows, whose sum lives in the item's outputs until the
item's end.  With all-zero K codes and LSE 0 every visible P-hat is exactly 2^8, so dV is a sum of dO codes and dK one of the kernel's own
dS' codes: both are formed in 64 bits here."""
import pytest
import torch

from delta_matching_b200 import _lib

pytestmark = pytest.mark.gpu


def _inputs(N, H, Hk, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rq, rk = _lib.blocks(D)
    code = lambda h: torch.randn(h, N, D, generator=g, device="cuda").mul_(50).clamp_(-448, 448).to(torch.float8_e4m3fn)
    scale = lambda h, b: torch.rand(h, N // b, generator=g, device="cuda") + 0.5
    return {"Q8": code(H), "K8": torch.zeros(Hk, N, D, device="cuda").to(torch.float8_e4m3fn), "V8": code(Hk), "dO8": code(H), "Q8s": scale(H, rq),
            "K8s": scale(Hk, rk), "V8s": scale(Hk, rk), "dO8s": scale(H, rq), "lse": torch.zeros(H, N, device="cuda"),
            "delta": torch.randn(H, N, generator=g, device="cuda")}


def _dv(d, h, D):
    x = d["dO8"][h].double() * d["dO8s"][h].double().repeat_interleave(_lib.blocks(D)[0])[:, None]
    return x.flip(0).cumsum(0).flip(0)                             # a key's rows: its own and all below


# walks of 1 to 130 tiles: every remainder of a window, 64 / 65 and 128 / 129 among them
@pytest.mark.parametrize("D,out_fp32", [(128, False), (128, True), (256, False)])
def test_gradients_of_walks_up_to_two_windows(D, out_fp32):
    N, H, Hk = 130 * 128, 2, 1
    d = _inputs(N, H, Hk, D, 5)
    dk, dv, ws = _lib.bwd_pass1(*d.values(), 1, H, Hk, True, out_fp32=out_fp32)
    assert _lib.device_status() == 0
    nb, kb = N // 128, 128 if D == 128 else 64
    ds8 = ws[0].view(H, nb, nb, 128, 128).view(torch.float8_e4m3fn)                       # [head, row block, key block, key, row]
    psi = ws[1].view(H, N // 64, N // kb).double()
    keep = 2.0 ** -23 if out_fp32 else 2.0 ** -8                    # of an element, before the sums' own errors: its last rounding
    for h in range(H):
        ref = _dv(d, h, D)
        err = (dv[0, :, h].double() - ref).abs()
        # what the additions of a window (four a tile) and the window sums may lose, each a unit in the last place of the running sum
        size = d["dO8"][h].double().abs().mul_(d["dO8s"][h].double().repeat_interleave(_lib.blocks(D)[0])[:, None]).flip(0).cumsum(0).flip(0)
        assert (err <= keep * ref.abs() + 64 * 4 * 2.0 ** -24 * size).all()
        dkr = torch.zeros(N, D, device="cuda", dtype=torch.float64)
        qs = d["Q8s"][h].double().repeat_interleave(N // d["Q8s"].shape[1])
        for rb in range(nb):
            rows = slice(128 * rb, 128 * rb + 128)
            c = ds8[h, rb, :rb + 1].double()                                              # [key block, key, row]
            f = psi[h, 2 * rb:2 * rb + 2].repeat_interleave(64, 0).repeat_interleave(kb, 1)[:, :128 * (rb + 1)] / 256
            c = c.reshape(-1, 128) * f.T * qs[rows]
            dkr[:128 * (rb + 1)] += c @ d["Q8"][h, rows].double()
        dkr /= d["K8s"][0].double().repeat_interleave(N // d["K8s"].shape[1])[:, None]
        assert ((dk[0, :, h].double() - dkr).norm() <= (1e-6 if out_fp32 else 2e-3) * dkr.norm())


@pytest.mark.parametrize("D", [128, 256])
def test_the_outputs_do_not_depend_on_the_head_range(D):
    N, H, Hk = 72 * 128, 4, 2
    d = _inputs(N, H, Hk, D, 6)
    dk, dv, _ = _lib.bwd_pass1(*d.values(), 1, H, Hk, True)
    out = (torch.full_like(dk, float("nan")), torch.full_like(dv, float("nan")))
    for h0 in range(H):
        _lib.bwd_pass1(*d.values(), 1, H, Hk, True, h0=h0, hcount=1, out=out)
    assert torch.equal(dk, out[0]) and torch.equal(dv, out[1])


def test_the_sum_of_a_very_long_walk_does_not_drift():
    """512 tiles of gradients of one sign.  The tensor pipe's additions, four a tile, round towards zero: a sum that is never set down loses
    1.5e-5 here (measured), eight windows an eighth of that or less each of its own part."""
    N = 65536
    d = _inputs(N, 1, 1, 128, 7)
    d["dO8"] = d["dO8"].float().abs().to(torch.float8_e4m3fn)
    _, dv, _ = _lib.bwd_pass1(*d.values(), 1, 1, 1, True, out_fp32=True)
    ref = _dv(d, 0, 128)[:256]
    off = ((dv[0, :256, 0].double() - ref).sum() / ref.sum()).item()
    assert abs(off) <= 1.5e-5 / 8, off
