"""The operator's native host path (csrc/torch_ops.cpp) against its Python path: the same library calls, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,opts,finals", [
    (torch.float32, (), False), (torch.float32, ("D", "z", "bias", "init"), True), (torch.bfloat16, ("D", "z", "bias"), False),
    (torch.bfloat16, ("strided", "init"), True), (torch.float16, ("z", "one_init", "only_x"), False)])
def test_native_path_equals_python_path(dtype, opts, finals):
    from ssd.bi.ssd_combined import MambaChunkScanCombinedFn, bimamba_chunk_scan_combined
    b, L, H, P, G, N, Q = 2, 150, 4, 64, 2, 64, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s, t=torch.float32: torch.randn(*s, generator=g, device="cuda").to(t)
    x = mk(b, L, H, P + (1 if "strided" in opts else 0), t=dtype)[..., :P]       # rows that miss the 16-byte alignment
    ins = dict(x=x, dt=mk(b, L, H), A=-mk(H).abs(), B=mk(b, L, G, N, t=dtype), C=mk(b, L, G, N, t=dtype),
               D=mk(H, P) if "D" in opts else None, z=mk(b, L, H, P, t=dtype) if "z" in opts else None,
               dt_bias=mk(H) if "bias" in opts else None, initial_states_f=mk(b, H, P, N) if "init" in opts else None,
               initial_states_b=mk(b, H, P, N) if "init" in opts or "one_init" in opts else None)
    leaves = [t for k, t in ins.items() if t is not None and ("only_x" not in opts or k == "x")]
    for t in leaves:
        t.requires_grad_(True)
    order = lambda i: (i["x"], i["dt"], i["A"], i["B"], i["C"], Q, i["D"], i["z"], i["dt_bias"], True, (0.0, 2.0), finals,
                       i["initial_states_f"], i["initial_states_b"])
    got, want = bimamba_chunk_scan_combined(*order(ins)), MambaChunkScanCombinedFn.apply(*order(ins))
    got, want = (r if finals else (r,) for r in (got, want))
    douts = [torch.randn(t.shape, generator=g, device="cuda").to(t.dtype) for t in want]
    ggot, gwant = (torch.autograd.grad(r, leaves, douts) for r in (got, want))
    with torch.no_grad():
        free = bimamba_chunk_scan_combined(*order(ins))
    for a, w in zip((*got, *ggot, *(free if finals else (free,))), (*want, *gwant, *want)):
        assert a.dtype == w.dtype and torch.equal(a, w)
    if finals:                                           # a gradient of the final states alone
        ggot, gwant = (torch.autograd.grad(r[1], leaves, douts[1]) for r in (
            bimamba_chunk_scan_combined(*order(ins)), MambaChunkScanCombinedFn.apply(*order(ins))))
        assert all(torch.equal(a, w) for a, w in zip(ggot, gwant))
