"""A row's results do not depend on how many rows there are: sizes where the batch changes the kernels, or how they share work."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rows(dtype, b, L, H, P, G, N, Q, z, few=1):
    """out, dx, ddt, dB, dC (and dz) of `few` rows run alone and of the same rows among b, with the kernels of each run."""
    from ssd import _cabi
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    g = torch.Generator(device="cuda").manual_seed(L + H + P)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, B, C, dout, gate = (t.to(dtype) for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N), mk(b, L, H, P), mk(b, L, H, P)))
    per_row, shared = [x, mk(b, L, H) - 4.0, B, C] + ([gate] if z else []), [-torch.exp(torch.rand(H, generator=g, device="cuda") * 2.7), mk(H)]
    results = []
    for n in (few, b):
        leaves = [t[:n].clone().requires_grad_(True) for t in per_row]
        _cabi.trace_enable(True)
        out = bimamba_chunk_scan_combined(leaves[0], leaves[1], shared[0], leaves[2], leaves[3], Q, D=shared[1], z=leaves[4] if z else None,
                                          dt_softplus=True)
        got = [out, *torch.autograd.grad(out, leaves, dout[:n])]
        torch.cuda.synchronize()
        ran = set(_cabi.trace_read())
        _cabi.trace_enable(False)
        results.append((dict(zip(("out", "dx", "ddt", "dB", "dC", "dz"), (t[:few] for t in got))), ran))
    return results


def check(*case, **kw):
    (alone, _), (among, _) = results = rows(*case, **kw)
    for k in alone:
        assert torch.equal(alone[k], among[k]), k
    return [ran for _, ran in results]


@pytest.mark.parametrize("case", [(torch.float16, 11, 916, 1, 128, 1, 128, 128, True), (torch.float32, 5, 175, 32, 32, 4, 16, 64, False),
                                  (torch.bfloat16, 8, 600, 12, 32, 1, 32, 64, True)])
def test_recurrence_with_chunks_in_flight(case):
    """Few threads keep eight chunks' loads in flight, many one: the same sums."""
    check(*case)


@pytest.mark.parametrize("case", [(torch.bfloat16, 16, 1000, 4, 128, 2, 64, 128, True), (torch.float16, 16, 1024, 4, 128, 2, 64, 128, False),
                                  (torch.bfloat16, 16, 2000, 4, 64, 4, 64, 256, False), (torch.bfloat16, 7, 517, 16, 128, 2, 64, 256, False)])
def test_walk_and_two_kernels_dstate_64(case):
    """Few rows: chunk states and the recurrence as two kernels; many: the walk.  The states round alike."""
    few, many = check(*case)
    assert "tc_chunk_state_tma" in few and "tc_state_walk" in many, (few, many)


@pytest.mark.parametrize("case", [(torch.bfloat16, 4, 8192, 8, 64, 1, 128, 256, False), (torch.bfloat16, 64, 1000, 4, 64, 2, 64, 128, True),
                                  (torch.float16, 14, 822, 4, 64, 4, 256, 128, True), (torch.bfloat16, 11, 842, 12, 128, 4, 128, 128, False),
                                  (torch.float16, 16, 1000, 4, 128, 2, 256, 128, True), (torch.bfloat16, 20, 585, 6, 128, 2, 64, 128, True)])
def test_walk_and_two_kernels(case):
    """The sums over a chunk's states that enter ddt are added up in one order, whichever computes them."""
    few, many = check(*case)
    assert "state_passing_bwd" in few and "tc_dstate_walk" in many, (few, many)


@pytest.mark.parametrize("case,few", [((torch.float32, 8, 1000, 8, 32, 1, 32, 128, True), 1), ((torch.float32, 6, 700, 8, 64, 2, 64, 128, False), 1),
                                      ((torch.float32, 30, 294, 12, 16, 1, 16, 64, True), 5), ((torch.float32, 9, 242, 48, 64, 4, 64, 64, True), 1),
                                      ((torch.float32, 9, 222, 9, 16, 1, 17, 66, False), 2), ((torch.bfloat16, 40, 200, 6, 20, 1, 12, 40, False), 1)])
def test_cuda_core_heads_in_parts(case, few):
    """Heads of a group dealt to several blocks, or all to one: dCB is summed in the same parts."""
    check(*case, few=few)


@pytest.mark.parametrize("P,N", [(64, 64), (64, 128), (64, 256), (128, 64), (128, 128), (128, 256)])
def test_one_pass_and_two_phases(P, N):
    """A whole backward pass walks; one in phases, as the sequence-sharded operator runs it, keeps its local gradients."""
    from ssd.bi import sequence_parallel as sp
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    b, L, H, G, Q = 4, 700, 24, 2, 128
    g = torch.Generator(device="cuda").manual_seed(P + N)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, B, C, dout = (t.bfloat16() for t in (mk(b, L, H, P), mk(b, L, G, N), mk(b, L, G, N), mk(b, L, H, P)))
    leaves = [t.requires_grad_(True) for t in (x, mk(b, L, H) - 4.0, -torch.rand(H, generator=g, device="cuda") - 0.1, B, C)]
    out = bimamba_chunk_scan_combined(*leaves, Q, dt_softplus=True)
    want = [out, *torch.autograd.grad(out, leaves, dout)]
    zero = torch.zeros(b, H, P, N, device="cuda")
    for boundary in (None, zero):                            # nothing enters the shard
        st = sp.local_forward(*(t.detach() for t in leaves), Q, dt_softplus=True)
        got = [sp.finish_forward(st, boundary, boundary)]
        sp.local_backward(st, dout)
        got += sp.finish_backward(st, boundary, boundary)[:5]
        for a, w, name in zip(got, want, ("out", "dx", "ddt", "dA", "dB", "dC")):
            assert torch.equal(a, w), name
