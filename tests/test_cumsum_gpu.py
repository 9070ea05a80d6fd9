"""Four warps per (batch, chunk, head) of the cumulative sums: lane, warp, chunk and head remainders, clamps and dt types, against
the oracle."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err, reference_with_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,G,P,N,Q,dt_dtype,limit", [
    (33, 1, 1, 16, 16, 32, torch.float32, (0.0, float("inf"))), (300, 9, 3, 32, 16, 40, torch.bfloat16, (0.01, 0.05)),
    (257, 8, 1, 64, 64, 128, torch.float32, (0.0, float("inf"))), (400, 10, 2, 64, 32, 136, torch.float16, (0.0, 0.04)),
    (513, 17, 1, 64, 128, 256, torch.bfloat16, (0.02, 0.06)), (250, 3, 1, 128, 64, 248, torch.float32, (0.0, 0.1))])
def test_cumsums(L, H, G, P, N, Q, dt_dtype, limit):
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator().manual_seed(L + Q)
    mk = lambda *s: torch.randn(*s, generator=g)
    b = 2
    x, B, C, dout = (t.bfloat16() for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N), mk(b, L, H, P)))
    dt, A, bias = (mk(b, L, H) - 3.0).to(dt_dtype), -torch.rand(H, generator=g) - 0.5, 0.1 * mk(H)
    wide = dt.new_zeros(b, L, H + 3)
    wide[..., 1:H + 1] = dt
    leaves = [x.cuda(), wide.cuda()[..., 1:H + 1], A.cuda(), B.cuda(), C.cuda(), bias.cuda()]
    leaves = [t.requires_grad_(True) for t in leaves]
    out = bimamba_chunk_scan_combined(*leaves[:5], Q, dt_bias=leaves[5], dt_softplus=True, dt_limit=limit)
    got = [out, *torch.autograd.grad(out, leaves, dout.cuda())]
    r = reference_with_grads(x, dt, A, B, C, Q, dout, dt_bias=bias, dt_softplus=True, dt_limit=limit)
    for a, name in zip(got, ("out", "dx", "ddt", "dA", "dB", "dC", "ddt_bias")):
        assert max_rel_err(a, r[name]) < 2e-2, name
