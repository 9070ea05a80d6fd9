"""Edges of the convolution's runs of rows and of the norm's blocks: lengths around a run and a round, channel counts that
leave a warp part empty, width 1, row counts around a step, one and several rows side by side in a block."""
import pytest
import torch
from oracle.bissd_oracle import max_rel_err
from oracle.layer_oracle import dwconv1d_silu_reference, rms_norm_gated_reference

pytestmark = pytest.mark.gpu


def _check(fn, ref_fn, leaves, dout, tol):
    dev = [t.cuda().requires_grad_(True) for t in leaves]
    ref = [t.float().requires_grad_(True) for t in leaves]
    got, want = fn(*dev), ref_fn(*ref)
    ggot, gwant = torch.autograd.grad(got, dev, dout.cuda()), torch.autograd.grad(want, ref, dout.float())
    for a, w in zip((got, *ggot), (want, *gwant)):
        assert max_rel_err(a, w) < tol


@pytest.mark.parametrize("L,C,K,dtype", [(31, 8, 1, torch.float32), (32, 136, 3, torch.float32), (33, 72, 7, torch.float32),
                                         (257, 264, 7, torch.bfloat16), (6, 64, 5, torch.float16), (1, 128, 7, torch.float32)])
def test_conv_runs(L, C, K, dtype):
    from ssd.bi.conv_silu import dwconv1d_silu
    g = torch.Generator().manual_seed(L * C + K)
    mk = lambda *s: torch.randn(*s, generator=g)
    _check(dwconv1d_silu, dwconv1d_silu_reference, [mk(2, L, C).to(dtype), 0.4 * mk(C, 1, K), 0.2 * mk(C)], mk(2, L, C).to(dtype),
           2e-5 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("rows,hidden,group,before,dtype", [(1, 256, 256, True, torch.float32), (17, 256, 256, False, torch.float32),
                                                            (3, 4096, 2048, True, torch.float32), (1500, 768, 256, False, torch.bfloat16),
                                                            (2399, 512, 512, True, torch.bfloat16)])
def test_norm_blocks(rows, hidden, group, before, dtype):
    from ssd.bi.layernorm_gated import rmsnorm_fn
    g = torch.Generator().manual_seed(rows + hidden)
    mk = lambda *s: torch.randn(*s, generator=g)
    kw = dict(eps=1e-5, group_size=group, norm_before_gate=before)
    _check(lambda x, w, z: rmsnorm_fn(x, w, None, z=z, **kw), lambda x, w, z: rms_norm_gated_reference(x, w, None, z=z, **kw),
           [mk(rows, hidden).to(dtype), 1.0 + 0.3 * mk(hidden), mk(rows, hidden).to(dtype)], mk(rows, hidden).to(dtype),
           2e-5 if dtype == torch.float32 else 2e-2)
