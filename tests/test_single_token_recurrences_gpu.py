"""The delta rules' recurrences for one token a sequence: the bits of the form for any number of tokens (GPU)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from llmi_b200.ops import kernels
    return kernels


def _contexts(slots):
    S = len(slots)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731
    seq = [i if s >= 0 else -1 for i, s in enumerate(slots)]
    return [types.SimpleNamespace(n_seqs=S, decode=one, seq_q_start=i32(list(range(S + 1))), seq_slot=i32(slots), tok_seq=i32(seq),
                                  tok_pos=i32([5] * S), seq_kv_len=i32([6 if s >= 0 else 0 for s in slots])) for one in (True, False)]


@pytest.mark.parametrize("H,Hk,D,Dv", [(4, 4, 32, 32), (3, 3, 64, 48), (6, 2, 64, 64), (4, 2, 128, 128), (2, 1, 128, 16)])
@pytest.mark.parametrize("write", [True, False])
def test_single_tokens_same_bits(H, Hk, D, Dv, write):
    """Slots out of order, a padding sequence; key heads shared; a decay per head and one per channel; the state kept and not."""
    k = K()
    torch.manual_seed(H * D + Dv)
    slots = [3, 0, -1, 4, 1]
    S, taps = len(slots), 4
    outs = []
    for ctx in _contexts(slots):
        torch.manual_seed(7)
        row = []
        proj, prep = torch.randn(S, 2 * H * D + H * Dv + 8, device="cuda"), torch.rand(S, 3 * H * D + 4, device="cuda")
        state, o = torch.randn(6, H * D * Dv + 4, device="cuda"), torch.full((S, H * Dv), 7.0, device="cuda")
        k.dplr_recurrence(proj, prep, H, D, Dv, state, ctx, o, write)
        row += [state, o]
        nc = 2 * Hk * D + H * Dv
        for channel in (False, True):
            proj = torch.randn(S, nc + 2 * H + H * Dv, device="cuda")
            prep = torch.empty(S, nc + (H * D + 2 * H if channel else 2 * H), device="cuda")
            state, o = torch.randn(6, k.delta_state_floats(H, Hk, D, Dv, taps), device="cuda"), torch.full((S, H * Dv), 7.0, device="cuda")
            z = torch.randn(S, H * D, device="cuda") if channel else None
            k.delta_step(proj, (H, Hk, D, Dv, taps), torch.randn(nc, taps, device="cuda"), torch.randn(H, device="cuda") * 0.1,
                         torch.randn(H * D if channel else H, device="cuda"), state, ctx, prep, o, write, z)
            row += [state, o]
        outs.append(row)
    for i, (a, b) in enumerate(zip(*outs)):
        assert torch.equal(a, b), i
        assert bool(torch.isfinite(a).all())
    assert all(bool((o[2] == 7.0).all()) for o in outs[0][1::2])      # (nobody's row)
    k.check_device_errors("cuda:0")
