"""Heads summed in parts by several blocks (few tiles a row) or by one (many rows): the oracle, and the same bits either way."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err, reference_with_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,G,N,Q", [(300, 24, 1, 128, 256), (257, 16, 1, 64, 128), (200, 20, 2, 128, 256), (500, 34, 2, 128, 128)])
def test_parts_do_not_depend_on_the_batch(L, H, G, N, Q):
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator().manual_seed(L + H)
    b, P = 40, 64
    mk = lambda *s: torch.randn(*s, generator=g)
    x, B, C, dout = (t.bfloat16() for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N), mk(b, L, H, P)))
    ins = [x, mk(b, L, H) - 4.0, -torch.exp(torch.rand(H, generator=g) * 2.7), B, C, mk(H)]

    def run(rows):
        leaves = [(t[:rows] if t.dim() > 2 else t).cuda().requires_grad_(True) for t in ins]
        out = bimamba_chunk_scan_combined(*leaves[:5], Q, D=leaves[5], dt_softplus=True)
        return [out, *torch.autograd.grad(out, leaves, dout[:rows].cuda())]
    few, many = run(1), run(b)
    for k in (0, 1, 2, 4, 5):                            # out, dx, ddt, dB, dC
        assert torch.equal(few[k], many[k][:1]), k
    r = reference_with_grads(x[:1], ins[1][:1], ins[2], B[:1], C[:1], Q, dout[:1], D=ins[5], dt_softplus=True)
    for k, name in enumerate(("out", "dx", "ddt", "dA", "dB", "dC", "dD")):
        assert max_rel_err(few[k], r[name]) < 2e-2, name
