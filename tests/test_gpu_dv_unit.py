"""Pass 1 keeps dV's accumulator in units of the current dO scale block's scale (128 rows; head_dim 256: 64): gradients whose
blocks differ by many orders of magnitude, or are all zero (first, middle, last, everywhere), against the CPU oracle."""
import pytest
import torch

from delta_matching_b200 import _lib
from oracle import dm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,rows", [(128, 128), (256, 64)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("scales", [(1, 0, 1, 1), (0, 1, 0, 1), (1, 1, 1, 0), (0, 0, 0, 0), (1e-6, 1e6, 1, 1e-12), (1e12, 1e-6, 0, 1e3)])
def test_dv_over_blocks_of_very_different_scale(scales, causal, D, rows):
    B, N, H, Hk = 1, 512, 2, 1
    q, k, v, dO = O.make_inputs(B, N, H, Hk, D, 77)
    dO = (dO.float() * torch.tensor(scales, dtype=torch.float32).repeat_interleave(rows).repeat(N // (4 * rows))[None, :, None, None]).to(torch.bfloat16)
    r = O.attention_fwd_bwd(q, k, v, dO, causal, "stale", fwd_tile_keys=128, pv="group", debug=True)
    d = [r[n].cuda() for n in ("Q8", "K8", "V8", "dO8", "Q8s", "K8s", "V8s", "dO8s", "LSE", "delta")]
    dk, dv, _ = _lib.bwd_pass1(*d, B, H, Hk, causal)
    assert _lib.device_status() == 0
    ref = r["dVh"].to(torch.bfloat16).view(B, H, N, D).permute(0, 2, 1, 3).float()
    assert torch.isfinite(dv).all() and torch.isfinite(dk).all()
    for b in range(4):                     # per key block: a small block's gradient must not drown in a large one's
        got, want = dv[:, 128 * b:128 * (b + 1)].cpu().float(), ref[:, 128 * b:128 * (b + 1)]
        assert (got - want).norm() <= 2e-3 * want.norm(), b
