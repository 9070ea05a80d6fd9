"""Which sizes walk the chunks in one kernel and which take two, as the least scratch shows it (a walk has no fp32 local states): sizes
where one form is well ahead of the other (us a forward call, two kernels and walk)."""
import ctypes
import pytest

from ssd import _cabi


@pytest.mark.parametrize("b,L,H,P,N,Q,walks", [
    (1, 16747, 24, 64, 64, 128, True),        # 213, 153
    (5, 17696, 8, 64, 64, 128, True),         # 298, 207
    (2, 15326, 16, 64, 64, 128, True),        # 223, 170
    (8, 2048, 24, 64, 128, 256, True), (8, 1024, 16, 128, 256, 128, True),
    (1, 8192, 8, 64, 128, 256, False),        # 46, 69
    (1, 6260, 2, 128, 128, 128, False),       # 35, 93
    (1, 17397, 2, 128, 256, 128, False)])     # 85, 230
def test_walk_or_two_kernels(b, L, H, P, N, Q, walks):
    p = _cabi.Problem(batch=b, seqlen=L, nheads=H, headdim=P, ngroups=1, dstate=N, chunk_size=Q, x_dtype=_cabi.BF16, dt_dtype=_cabi.F32)
    lib, least, full = _cabi.load(), ctypes.c_size_t(), ctypes.c_size_t()
    assert lib.bissd_workspace_bytes_least(ctypes.byref(p), ctypes.byref(least), None) == 0
    assert lib.bissd_workspace_bytes(ctypes.byref(p), ctypes.byref(full), None) == 0
    local_states = 2 * b * -(-L // Q) * H * P * N * 4
    assert (full.value - least.value >= local_states) == walks


@pytest.mark.gpu
def test_a_pass_in_two_phases_does_not_walk_twice():
    """Where one walk pays and two do not, the phases take the two kernels, which repeat the recurrence only: the same bits."""
    import torch
    from ssd.bi import sequence_parallel as sp
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    b, L, H, P, N, Q = 1, 2048, 16, 64, 128, 256
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ins = [mk(b, L, H, P).bfloat16(), mk(b, L, H) - 4.0, -torch.rand(H, generator=g, device="cuda") - 0.1, mk(b, L, 1, N).bfloat16(), mk(b, L, 1, N).bfloat16()]
    start = [mk(b, H, P, N), mk(b, H, P, N)]
    outs, ran = [], []
    for phases in (False, True):
        _cabi.trace_enable(True)
        try:
            if phases:
                outs.append(sp.finish_forward(sp.local_forward(*ins, Q, dt_softplus=True), *start))
            else:
                outs.append(bimamba_chunk_scan_combined(*ins, Q, dt_softplus=True, initial_states_f=start[0], initial_states_b=start[1]))
            torch.cuda.synchronize()
            ran.append(_cabi.trace_read())
        finally:
            _cabi.trace_enable(False)
    assert "tc_state_walk" in ran[0] and "tc_state_walk" not in ran[1], ran
    assert torch.equal(*outs)
