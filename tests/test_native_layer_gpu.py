"""The layer's native node (csrc/torch_ops.cpp) against its Python path, which calls the same kernels one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,ngroups,bias,seqlen,mem_eff,d_head", [
    (torch.bfloat16, 1, False, 333, False, 64), (torch.bfloat16, 2, True, 128, True, 64),
    (torch.float32, 1, True, 70, False, 32), (torch.float16, 1, False, 257, True, 128)])
def test_native_layer_equals_python_path(monkeypatch, dtype, ngroups, bias, seqlen, mem_eff, d_head):
    from ssd.modules import BiMamba2
    torch.manual_seed(5)
    layer = BiMamba2(512, d_state=64, headdim=d_head, ngroups=ngroups, bias=bias, chunk_size=128, use_mem_eff_path=mem_eff,
                     device="cuda").to(dtype)
    with torch.no_grad():
        layer.A_log.uniform_(0.0, 2.0)
        layer.norm.weight.uniform_(0.5, 1.5)
    u = torch.randn(2, seqlen, 512, device="cuda").to(dtype).requires_grad_(True)
    dout = torch.randn(2, seqlen, 512, device="cuda").to(dtype)
    names, leaves = zip(("u", u), *((n, p) for n, p in layer.named_parameters() if not n.startswith("fc_D")))

    def step():
        out = layer(u)
        return (out, *torch.autograd.grad(out, leaves, dout))
    got = step()
    with torch.no_grad():
        free = layer(u)
    monkeypatch.setattr(BiMamba2, "_native_ok", lambda self: False)
    import ssd.bi.split_conv1d_scan as split
    monkeypatch.setattr(split, "native_layer", lambda *a: None)
    want = step()
    assert torch.equal(free, got[0])
    # the same kernels on the same numbers; only A_log's gradient is one product rounded once instead of twice, by half an ulp each
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    for n, a, w in zip(("out", *names), got, want):
        assert a.dtype == w.dtype and a.shape == w.shape, n
        if n == "A_log":
            assert ((a.float() - w.float()).abs() <= 1.5 * ulp * w.float().abs() + 1e-7).all(), n
        else:
            assert torch.equal(a, w), n
