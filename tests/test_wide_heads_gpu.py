"""headdim 128 and dstate above 128: slab counts, both chunk sizes, groups, ragged tails, against the oracle."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err, reference_with_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,L,H,G,P,N,Q,z", [
    (torch.float16, 130, 2, 1, 128, 64, 128, True), (torch.bfloat16, 257, 3, 3, 128, 128, 256, False),
    (torch.float16, 300, 4, 2, 128, 192, 128, True), (torch.bfloat16, 100, 5, 1, 128, 256, 256, True),
    (torch.float16, 513, 8, 2, 128, 256, 128, False), (torch.bfloat16, 390, 4, 1, 64, 256, 128, True),
    (torch.float16, 260, 3, 1, 64, 192, 256, False)])
def test_wide(dtype, L, H, G, P, N, Q, z):
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator().manual_seed(L + N)
    mk = lambda *s: torch.randn(*s, generator=g)
    b = 2
    x, B, C, dout = (t.to(dtype) for t in (mk(b, L, H, P), 0.5 * mk(b, L, G, N), 0.5 * mk(b, L, G, N), mk(b, L, H, P)))
    ins = dict(x=x, dt=torch.rand(b, L, H, generator=g) * 0.05, A=-torch.rand(H, generator=g) - 0.5, B=B, C=C, D=mk(H, P))
    if z:
        ins["z"] = mk(b, L, H, P).to(dtype)
    leaves = {k: t.cuda().requires_grad_(True) for k, t in ins.items()}
    out = bimamba_chunk_scan_combined(**leaves, chunk_size=Q)
    got = [out, *torch.autograd.grad(out, list(leaves.values()), dout.cuda())]
    r = reference_with_grads(*(ins[k] for k in ("x", "dt", "A", "B", "C")), Q, dout, D=ins["D"], z=ins.get("z"))
    for a, name in zip(got, ["out"] + ["d" + k for k in leaves]):
        assert max_rel_err(a, r[name]) < 2e-2, name
