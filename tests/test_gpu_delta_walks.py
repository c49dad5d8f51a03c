"""Pass 0: the persistent roles kernel over walks of one tile, of one item and of several items per CTA, against the
debug row sums: with delta subtracted the rows of P-hat * (dP - delta) cancel to round-off."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,unit", [(128, 256), (256, 128)])      # the unit of a sequence's length
@pytest.mark.parametrize("B,n,H,Hk,causal", [(1, 1, 2, 1, True), (1, 3, 3, 1, False), (1, 5, 2, 2, True), (2, 10, 16, 4, True),
                                             (16, 1, 64, 8, True)])
def test_delta_equals_and_cancels_the_row_sums(B, n, H, Hk, causal, D, unit):
    N = n * unit
    q, k, v, dO = (t.cuda() for t in O.make_inputs(B, N, H, Hk, D, 2011))
    Q8, Q8s = _lib.quant(0, q)
    K8, K8s = _lib.quant(1, k, _lib.kmean(k))
    V8, V8s = _lib.quant(2, v)
    o, lse = _lib.fwd_fp8(Q8, K8, V8, Q8s, K8s, V8s, B, H, Hk, causal)
    dO8, dO8s = _lib.quant_do(dO)[:2]
    ops = (Q8, K8, V8, dO8, Q8s, K8s, V8s, dO8s, lse)
    delta = _lib.delta_fp8(*ops, B, H, Hk, causal)
    rows, rows_abs = _lib.bwd_dbg_rowsum(*ops, delta, B, H, Hk, causal)
    plain, _ = _lib.bwd_dbg_rowsum(*ops, torch.zeros_like(delta), B, H, Hk, causal)      # the sums that delta is
    assert _lib.device_status() == 0
    assert (rows.double().norm() / rows_abs.double().norm()).item() < 1e-6
    assert O.rel(plain.cpu(), delta.cpu()) < 1e-5
    # a CTA's walk does not change a row's bits: the same heads, a few at a time
    part = torch.empty_like(delta)
    for h in range(0, H, 4):
        _lib.delta_fp8(*ops, B, H, Hk, causal, h0=h, hcount=min(4, H - h), out=part)
    assert torch.equal(part, delta)
