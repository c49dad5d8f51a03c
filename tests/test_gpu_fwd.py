"""The tcgen05 forward against the CPU oracle (same codes in, O and LSE out) and against fp32 attention."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


def _codes(q, k, v):
    Q8, Q8s = O.quant_q(q.transpose(1, 2))
    K8, K8s, _ = O.quant_k(k.transpose(1, 2))
    V8, V8s = O.quant_v(v.transpose(1, 2))
    return Q8, Q8s, K8, K8s, V8, V8s


@pytest.mark.parametrize("B,N,H,Hk,causal,D", [(1, 256, 2, 2, True, 128), (1, 512, 4, 2, True, 128), (2, 1024, 4, 1, True, 128),
                                                 (1, 512, 2, 2, False, 128), (1, 384, 2, 1, True, 256), (1, 512, 4, 2, False, 256),
                                                 (2, 256, 2, 2, True, 256)])
def test_forward_matches_oracle(B, N, H, Hk, causal, D):
    q, k, v, dO = O.make_inputs(B, N, H, Hk, D, 1001)
    c = _codes(q, k, v)
    o_ref, lse_ref = O.forward(*c, H, Hk, causal, tile_keys=128, pv="group")
    o, lse = _lib.fwd_fp8(*(t.cuda() for t in (c[0], c[2], c[4], c[1], c[3], c[5])), B, H, Hk, causal)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    o, lse = o.cpu(), lse.cpu()
    assert torch.isfinite(o.float()).all() and torch.isfinite(lse).all()
    assert (lse - lse_ref).abs().max() < 2e-4, (lse - lse_ref).abs().max()
    assert O.rel(o, o_ref) < 2e-3, O.rel(o, o_ref)
    ro = O.fp32_reference(q, k, v, dO, causal)[0]
    assert O.rel(o, ro) < 0.08
    # the reference's own tile geometry (D=128: 256-key tiles; rho chain) is the same sum in another rounding order
    o_ref2, _ = O.forward(*c, H, Hk, causal)
    assert O.rel(o, o_ref2) < 2e-3


def test_forward_head_range_and_determinism():
    B, N, H, Hk, D = 1, 512, 4, 2, 128
    q, k, v, _ = O.make_inputs(B, N, H, Hk, D, 3)
    c = [t.cuda() for t in _codes(q, k, v)]
    args = (c[0], c[2], c[4], c[1], c[3], c[5])
    o1, l1 = _lib.fwd_fp8(*args, B, H, Hk, True)
    o2, l2 = _lib.fwd_fp8(*args, B, H, Hk, True)
    assert torch.equal(o1, o2) and torch.equal(l1, l2)
    o3 = torch.zeros_like(o1)
    l3 = torch.zeros_like(l1)
    for h0 in range(0, H, 2):
        _lib.fwd_fp8(*args, B, H, Hk, True, h0=h0, hcount=2, out=(o3, l3))
    assert torch.equal(o1, o3) and torch.equal(l1, l3)


def _one_key_rows(Q8, K8, V8, Q8s, K8s, V8s, H, Hk):
    """O (bf16) and LSE of row 0 under the causal mask, every fp32 rounding of a row softmax over its single key written out.  Q / K codes are
    small integers, so the score's raw product is exact in any order of summation."""
    kv = O._kv_index(Q8.shape[0], H, Hk).to(Q8.device)
    l2, log2_448 = (torch.tensor(c, device=Q8.device, dtype=torch.float32) for c in (O.LOG2E, O.LOG2_448))
    fma = lambda a, b, c: (a.double() * b.double() + c.double()).float()       # the product of two fp32 numbers is exact in fp64
    raw = (Q8[:, 0].float() * K8[kv, 0].float()).sum(-1)
    dsc = Q8s[:, 0] * K8s[kv, 0]
    gm = raw * dsc
    ms = gm * l2 - log2_448
    p = torch.exp2(fma(raw, dsc * l2, -ms))
    code = p.clamp(max=448.0).to(torch.float8_e4m3fn).float()
    s0 = torch.exp2(fma(-gm, l2, ms))
    l = s0 * p
    o = (code[:, None] * V8[kv, 0].float()) * (V8s[kv, 0] * s0)[:, None]
    return (o * (1.0 / l)[:, None]).to(torch.bfloat16), gm + torch.log(l)


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("N,H,Hk", [(256, 8, 8), (768, 16, 4)])
def test_rows_of_one_key_round_as_a_row_softmax(N, H, Hk, seed):
    """V scales of few significant bits put half of a one-key row's products half way between two bf16 values: O's bits there are those of
    the row's softmax, and the stale delta and dQ built on them are the oracle's."""
    B, D = 2, 128
    g = torch.Generator().manual_seed(seed)
    ints = lambda h: torch.randint(-4, 5, (B * h, N, D), generator=g).float().to(torch.float8_e4m3fn)
    uni = lambda h, b, lo, hi: torch.rand(B * h, N // b, generator=g) * (hi - lo) + lo
    Q8, K8, V8 = ints(H), ints(Hk), torch.randn(B * Hk, N, D, generator=g).mul_(100).clamp_(-448, 448).to(torch.float8_e4m3fn)
    Q8s, K8s = uni(H, 128, 0.01, 0.03), uni(Hk, 64, 0.5, 1.0)
    V8s = torch.randint(9, 18, (B * Hk, N // 64), generator=g).float().mul_(2).add_(1).mul_(2.0 ** -12)         # odd, 19 .. 35
    dO = torch.randn(B, N, H, D, generator=g).to(torch.bfloat16)
    d = [t.cuda() for t in (Q8, K8, V8, Q8s, K8s, V8s)]
    o, lse = _lib.fwd_fp8(*d, B, H, Hk, True)
    o0, lse0 = _one_key_rows(*d, H, Hk)
    assert torch.equal(o[:, 0].reshape(B * H, D), o0)
    assert (lse[:, 0] - lse0).abs().max() <= 2.0 ** -23 * lse0.abs().max()            # logf of a denominator next to 1
    dO8, dO8s, delta = _lib.quant_do(dO.cuda(), o)
    o_ref = o.clone()
    o_ref[:, 0] = o0.view(B, H, D)
    delta_ref = O.stale_delta(dO, o_ref.cpu())
    dk, dv, ws = _lib.bwd_pass1(d[0], d[1], d[2], dO8, d[3], d[4], d[5], dO8s, lse, delta, B, H, Hk, True)
    dq = _lib.bwd_pass2(ws, d[1], B, H, Hk, N, D, True).cpu().float()
    assert _lib.device_status() == 0
    r = O.bwd_pass1(Q8, Q8s, K8, K8s, V8, V8s, dO8.cpu(), dO8s.cpu(), lse.cpu(), delta_ref, H, Hk, True)
    ref = O.bwd_pass2(r[2], r[3], K8, H, Hk, True).view(B, H, N, D).permute(0, 2, 1, 3)
    rms = ref.square().mean().sqrt()
    off = ((dq - ref).abs() / ref.abs().clamp_min(rms))[:, 0].max().item()
    assert off <= 1 / 8 + 1 / 256, off                 # one e4m3 step of the row's single dS' code, one bf16 rounding


@pytest.mark.parametrize("N,causal", [(512, True), (768, False)])
def test_the_floor_of_a_basis_hangs_on_the_threads_own_maximum(N, causal):
    """Every other 64-key group lies about 25 binades below its neighbours and carries values 2^24 times theirs.  Against the row's maximum,
    12 binades up, most of its codes would be subnormal or zero; against the maximum of its own thread's groups they are whole."""
    B, H, Hk, D = 1, 4, 2, 128
    g = torch.Generator().manual_seed(9)
    code = lambda h, f: torch.randn(B * h, N, D, generator=g).mul_(f).clamp_(-448, 448).to(torch.float8_e4m3fn)
    Q8, K8, V8 = code(H, 100.0), code(Hk, 100.0), code(Hk, 100.0)
    Q8s, V8s = torch.full((B * H, N // 128), 1.0 / 100), torch.full((B * Hk, N // 64), 2.0 ** -7)
    K8s = torch.full((B * Hk, N // 64), 0.7 / 100)
    K8s[:, 1::2] *= 0.05
    V8s[:, 1::2] *= 2.0 ** 24
    c = (Q8, Q8s, K8, K8s, V8, V8s)
    own, lse_ref = O.forward(*c, H, Hk, causal, tile_keys=128, pv="group", floor="own")
    row, _ = O.forward(*c, H, Hk, causal, tile_keys=128, pv="group")
    o, lse = _lib.fwd_fp8(*(t.cuda() for t in (Q8, K8, V8, Q8s, K8s, V8s)), B, H, Hk, causal)
    assert _lib.device_status() == 0
    assert (lse.cpu() - lse_ref).abs().max() < 2e-4
    assert O.rel(o.cpu(), own) < 2e-3, O.rel(o.cpu(), own)
    assert O.rel(row, own) > 2e-2, O.rel(row, own)          # the inputs tell the two forms apart
