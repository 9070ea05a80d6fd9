"""The fused dCB / decay-gradient kernel: one, two, three and more heads a block (the depth of its buffers), parts of unequal length,
tiles with one row or column, both chunk sizes, decays beyond fp32's range across a strip - against the oracle."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err, reference_with_grads
from oracle.bissd_rounding_model import reduced_gradient_ok, reduced_gradient_scales

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,G,N,Q,steep,dtype", [
    (1, 8, 8, 64, 128, 0.0, torch.bfloat16), (129, 8, 4, 64, 128, 0.0, torch.bfloat16), (257, 9, 3, 128, 256, 0.0, torch.float16),
    (127, 8, 2, 64, 256, 0.0, torch.bfloat16), (385, 10, 1, 64, 128, 3.0, torch.bfloat16), (512, 18, 1, 128, 256, 6.0, torch.bfloat16),
    (300, 8, 1, 128, 256, 3.0, torch.float16)])
def test_against_the_oracle(L, H, G, N, Q, steep, dtype):
    from ssd import _cabi
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator().manual_seed(L + H + Q)
    mk = lambda *s: torch.randn(*s, generator=g)
    b, P = 2, 64
    x, B, C, dout = (t.to(dtype) for t in (0.5 * mk(b, L, H, P), 0.5 * mk(b, L, G, N), 0.5 * mk(b, L, G, N), mk(b, L, H, P)))
    dt, A = mk(b, L, H) - 4.0 + steep, -torch.exp(torch.rand(H, generator=g) * 2.7)
    leaves = [t.cuda().requires_grad_(True) for t in (x, dt, A, B, C)]
    _cabi.trace_enable(True)
    try:
        out = bimamba_chunk_scan_combined(*leaves, Q, dt_softplus=True)
        got = [out, *torch.autograd.grad(out, leaves, dout.cuda())]
        torch.cuda.synchronize()
        ran = _cabi.trace_read()
    finally:
        _cabi.trace_enable(False)
    assert "tc_intra_dcb_tile" in ran
    r = reference_with_grads(x, dt, A, B, C, Q, dout, dt_softplus=True)
    for k, name in ((0, "out"), (1, "dx"), (2, "ddt"), (4, "dB"), (5, "dC")):
        assert max_rel_err(got[k], r[name]) < 2e-2, name          # the bound of every 16-bit test of this operator
        # In the 2-norm a result is a sum of terms that went through at most a dozen roundings to 8 bits (C.B^T and V are bf16 for
        # fp16 too), each 2^-9 / sqrt(3) of its value in the mean: sqrt(12 / 3) 2^-9 = 3.9e-3 of the result
        want = r[name].double()
        assert (got[k].detach().double().cpu() - want).norm() <= 2.0 ** -8 * want.norm(), name
    # dA adds up the decay gradients of all tokens, this kernel's row and column sums of V among them
    scale = reduced_gradient_scales(x, dt, A, B, C, Q, dout, dt_softplus=True)["dA"]
    ok, err, bound = reduced_gradient_ok(got[3], r["dA"], scale, 2e-2)
    assert ok, (err, bound)
    # each term is off by one rounding to bf16 at most, 2^-9 of it, were they all to lie on one side
    assert err <= 2.0 ** -9 * scale.max(), (err, scale.max())
