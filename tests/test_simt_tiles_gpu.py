"""Edges of the CUDA-core kernels' tiles: widths around 16 / 32 / 64, chunks around 64, sizes no four elements divide, heads
dealt to several blocks, unaligned 16-bit inputs."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err, reference_with_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,L,H,P,G,N,Q,dtype", [
    (1, 65, 2, 16, 1, 17, 64, torch.float32), (1, 40, 8, 15, 1, 33, 32, torch.float32), (2, 130, 4, 33, 2, 16, 65, torch.float32),
    (1, 255, 6, 64, 3, 65, 128, torch.float32), (1, 300, 2, 80, 1, 70, 256, torch.float32), (1, 70, 4, 1, 4, 1, 66, torch.float32),
    (1, 100, 2, 20, 1, 12, 40, torch.bfloat16), (2, 33, 16, 32, 2, 32, 64, torch.float32)])
def test_cuda_core_tiles(b, L, H, P, G, N, Q, dtype):
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined, kernel_path
    g = torch.Generator().manual_seed(L + P + N)
    mk = lambda *s: torch.randn(*s, generator=g)
    x, B, C, z = (t.to(dtype) for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N), mk(b, L, H, P)))
    ins = [x, mk(b, L, H) - 3.0, -torch.exp(torch.rand(H, generator=g) * 2.7), B, C, mk(H, P), z, mk(H) * 0.1]
    dout = mk(b, L, H, P).to(dtype)
    dev = [t.cuda().requires_grad_(True) for t in ins]
    assert kernel_path(dev[0], dev[1], dev[3], Q) == "simt"
    out = bimamba_chunk_scan_combined(*dev[:5], Q, D=dev[5], z=dev[6], dt_bias=dev[7], dt_softplus=True)
    got = [out, *torch.autograd.grad(out, dev, dout.cuda())]
    r = reference_with_grads(x, ins[1], ins[2], B, C, Q, dout, D=ins[5], z=z, dt_bias=ins[7], dt_softplus=True)
    for k, a in zip(("out", "dx", "ddt", "dA", "dB", "dC", "dD", "dz", "ddt_bias"), got):
        assert max_rel_err(a, r[k]) < (1e-4 if dtype == torch.float32 else 2e-2), k
