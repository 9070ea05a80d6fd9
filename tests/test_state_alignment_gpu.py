"""Initial states and gradients of final states at any fp32 address: the same bits as at an aligned one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,H,G,P,N,Q,apart", [
    (torch.float32, 2, 1, 16, 20, 64, True), (torch.float32, 2, 1, 15, 17, 32, True), (torch.bfloat16, 2, 1, 64, 64, 128, True),
    (torch.float16, 2, 2, 32, 32, 64, True), (torch.bfloat16, 40, 1, 64, 128, 256, False)])
def test_states_at_any_address(dtype, H, G, P, N, Q, apart):
    from ssd import _cabi
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    b, L = 1, 5 * Q
    g = torch.Generator(device="cuda").manual_seed(P + N)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, B, C = (t.to(dtype) for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N)))
    rest = [x, mk(b, L, H) - 4.0, -torch.rand(H, generator=g, device="cuda"), B, C]
    states, grads = [mk(b, H, P, N) for _ in range(2)], [mk(b, H, P, N) for _ in range(2)]

    def moved(t, by):                                        # the same numbers, `by` floats past an aligned address
        buf = torch.empty(t.numel() + 4, device="cuda")[by:by + t.numel()]
        assert buf.data_ptr() % 16 == 4 * by
        return buf.copy_(t.flatten()).view(t.shape)

    def run(by):
        leaves = [t.clone().requires_grad_(True) for t in rest] + [moved(t, by).requires_grad_(True) for t in states]
        out, fin_f, fin_b = bimamba_chunk_scan_combined(*leaves[:5], Q, return_final_states=True, initial_states_f=leaves[5],
                                                        initial_states_b=leaves[6], dt_softplus=True)
        return [out, fin_f, fin_b, *torch.autograd.grad((fin_f, fin_b), leaves, [moved(t, by) for t in grads])]
    _cabi.trace_enable(True)
    want = run(0)
    torch.cuda.synchronize()
    assert ("state_passing_fwd" in _cabi.trace_read()) == apart
    _cabi.trace_enable(False)
    for by in (1, 2, 3):
        for a, w in zip(run(by), want):
            assert torch.equal(a, w)
