"""The chunk walk (states and their recurrence in one kernel): stage and tile edges, states in and out, against the fp64 oracle."""
import pytest
import torch
from oracle.bissd_oracle import chunked_reference, max_rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,b,L,H,G,P,N,Q", [
    (torch.bfloat16, 1, 100, 2, 1, 64, 128, 256), (torch.float16, 2, 200, 4, 2, 64, 64, 128),
    (torch.bfloat16, 1, 513, 6, 2, 64, 256, 256), (torch.float16, 8, 257, 3, 1, 128, 64, 256),
    (torch.bfloat16, 9, 600, 10, 2, 128, 128, 128), (torch.bfloat16, 8, 1100, 20, 1, 64, 128, 128),
    (torch.float16, 4, 300, 4, 1, 128, 256, 128)])
def test_walk(dtype, b, L, H, G, P, N, Q):
    from ssd import _cabi
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator().manual_seed(L + P + N)
    mk = lambda *s: torch.randn(*s, generator=g)
    x, B, C = (t.to(dtype) for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N)))
    ins = [x, torch.rand(b, L, H, generator=g) * 0.05, -torch.rand(H, generator=g) - 0.5, B, C, mk(b, H, P, N), mk(b, H, P, N)]
    gout, gf, gb = mk(b, L, H, P), mk(b, H, P, N), mk(b, H, P, N)

    def run(op, keys, dev, cast):
        leaves = [t.to(dev).to(cast or t.dtype).requires_grad_(True) for t in ins]
        r = op(*leaves[:5], Q, initial_states_f=leaves[5], initial_states_b=leaves[6], **{keys: True})
        outs = [r[k] for k in ("out", "final_f", "final_b")] if isinstance(r, dict) else list(r)
        loss = sum((o * w.to(dev).to(o.dtype)).sum() for o, w in zip(outs, (gout.to(dtype), gf, gb)))
        return outs + list(torch.autograd.grad(loss, leaves))
    _cabi.trace_enable(True)
    got = run(bimamba_chunk_scan_combined, "return_final_states", "cuda", None)
    torch.cuda.synchronize()
    ran = set(_cabi.trace_read())
    _cabi.trace_enable(False)
    assert {"tc_state_walk", "tc_dstate_walk"} <= ran, ran
    ref = run(chunked_reference, "return_intermediates", "cpu", torch.float64)
    for a, r, name in zip(got, ref, ("out", "final_f", "final_b", "dx", "ddt", "dA", "dB", "dC", "dinit_f", "dinit_b")):
        assert max_rel_err(a, r) < 2e-2, name
