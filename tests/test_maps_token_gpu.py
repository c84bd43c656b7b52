"""Single tokens over several score maps a head: the newest row first, last and alone in its page, whatever the pages bring ahead."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("Hq,G,maps,dk,dv", [(4, 2, 2, 64, 64), (6, 2, 1, 64, 128), (3, 3, 2, 128, 128), (8, 2, 2, 32, 64)])
@pytest.mark.parametrize("window,chunk", [(0, 0), (70, 0), (64, 0), (0, 128)])
def test_positions_around_a_page(Hq, G, maps, dk, dv, window, chunk):
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt = Runtime(torch.bfloat16, "cuda")
    torch.manual_seed(Hq + window)
    for p in (0, 1, 62, 63, 64, 127, 128, 129, 640):
        n, P = p + 1, p // 64 + 2
        pages = torch.randperm(P, device="cuda").int().view(1, P)
        kc = torch.full((P, G * maps, 64, dk), float("nan"), device="cuda").bfloat16()      # (behind the newest row: no numbers)
        vc = torch.full((P, G, 64, dv), float("nan"), device="cuda").bfloat16()
        k, v = torch.randn(n, G * maps, dk, device="cuda").bfloat16(), torch.randn(n, G, dv, device="cuda").bfloat16()
        for j in range(n):
            kc[pages[0, j // 64], :, j % 64], vc[pages[0, j // 64], :, j % 64] = k[j], v[j]
        q = torch.randn(1, Hq * maps * dk, device="cuda").bfloat16()
        ctx = types.SimpleNamespace(decode=True, n_seqs=1, n_real_seqs=1, tok_seq=_i32([0]), tok_pos=_i32([p]), seq_q_start=_i32([0, 1]),
                                    seq_kv_len=_i32([n]), seq_slot=_i32([0]), host_q_lens=[1], host_kv_lens=[n])
        out = torch.full((1, Hq * maps * dv), float("nan"), device="cuda").bfloat16()
        kernels.attention_maps(q, out, kc, vc, ctx, pages, 64, Hq, G, maps, dk, dv, dk ** -0.5, None, window, chunk, rt=rt)
        lo = max(0, n - window) if window else p // chunk * chunk if chunk else 0
        kd, vd = k[lo:].double().view(n - lo, G, 1, maps, dk), v[lo:].double().view(n - lo, G, 1, dv)
        w = torch.softmax((q.double().view(1, G, Hq // G, maps, dk) * kd).sum(-1) * dk ** -0.5, dim=0)
        want = (w[..., None] * vd[:, :, :, None]).sum(0).reshape(1, -1)
        # weights and result rounded to bf16
        assert float((out.double() - want).abs().max()) <= 2.0 ** -7 * float(v.abs().max()), p
