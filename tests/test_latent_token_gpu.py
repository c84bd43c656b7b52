"""Latent attention of single tokens: the per-head products with the rotation, and the attention over rows up to the newest (GPU)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("K", [64, 128, 256, 512, 1024, 2048, 96])
@pytest.mark.parametrize("N", [2, 13, 130])
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9])
def test_per_head_products(K, N, M):
    """Every row length of the kernel and one that it does not have, rows that end inside a block, tokens around a batch of four and
    around the line to the tensor cores; operands that lie apart."""
    from llmi_b200.ops import kernels
    torch.manual_seed(K + N + M)
    B, bx, by = 3, K + 8, N + N % 2 + 2
    x = torch.randn(M, B * bx, device="cuda").bfloat16()
    w = (torch.randn(B, N, K, device="cuda") * K ** -0.5).bfloat16()
    for early in (False, True):
        out = torch.full((M, B * by), 7.0, device="cuda").bfloat16()
        kernels.linear_batched(x, bx, w, out, by, K, early=early)
        for b in range(B):
            want = x[:, b * bx:b * bx + K].double() @ w[b].double().T
            got = out[:, b * by:b * by + N].double()
            size = x[:, b * bx:b * bx + K].double().abs() @ w[b].double().abs().T
            # the result's rounding, and a sum of K exact products in 32 bits
            assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -23 * size).all())
            assert bool((out[:, b * by + N + N % 2:(b + 1) * by] == 7.0).all())


@pytest.mark.parametrize("D,C,R,rot_dims,pairing", [(64, 64, 16, 16, 1), (128, 512, 64, 64, 1), (64, 256, 32, 20, 0), (256, 64, 5, 4, 0), (128, 128, 64, 0, 1)])
@pytest.mark.parametrize("T", [1, 2, 7])
def test_queries_equal_the_two_launches(D, C, R, rot_dims, pairing, T):
    """The rotated part bit for bit, entries that do not turn, an odd number of them, a token row of no sequence."""
    from llmi_b200.ops import kernels
    torch.manual_seed(D + C + T)
    H = 3
    pad = -(H * (D + R)) % 8                                         # rows start on 16 bytes
    q, w = torch.randn(T, H * (D + R) + pad, device="cuda").bfloat16()[:, :H * (D + R)], torch.randn(H, C, D, device="cuda").bfloat16()
    inv = torch.rand(max(rot_dims // 2, 1), device="cuda")
    ctx = types.SimpleNamespace(tok_seq=_i32([0, -1, 1, 2, 3, 4, 5][:T]), tok_pos=_i32([5000, 0, 3, 64, 9, 10, 11][:T]))
    one, two = (torch.full((T, H * (C + R)), 7.0, device="cuda").bfloat16() for _ in range(2))
    kernels.latent_query(q, D, w, one, C, R, H, inv, rot_dims, ctx, pairing, 1.25)
    kernels.latent_q_rotate(q, D, two, C, R, H, inv, rot_dims, ctx, pairing, 1.25)
    a, b = one.view(T, H, C + R), two.view(T, H, C + R)
    assert torch.equal(a[..., C:], b[..., C:])
    want = torch.einsum("thd,hcd->thc", q.double().reshape(T, H, D + R)[..., :D], w.double())
    assert float((a[..., :C].double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())


@pytest.mark.parametrize("H,C,R", [(16, 512, 64), (8, 64, 32), (3, 256, 16), (20, 128, 64)])
@pytest.mark.parametrize("window", [0, 70])
def test_positions_around_a_page(H, C, R, window):
    """The newest row alone in its page, last in it, first of all; several sequences a block; a row of no sequence; whatever lies
    behind the newest row is no number."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt = Runtime(torch.bfloat16, "cuda")
    torch.manual_seed(H + C)
    at = [0, 63, -1, 64, 65, 300, 127, 128]
    S, P, Dk = len(at), 5, C + R
    pages = torch.randperm(S * P, device="cuda").int().view(S, P)
    cache = torch.full((S * P, 1, 64, Dk), float("nan"), device="cuda").bfloat16()
    rows = torch.randn(S, P * 64, Dk, device="cuda").bfloat16()
    for s, p in enumerate(at):
        for j in range(p + 1):
            cache[pages[s, j // 64], 0, j % 64] = rows[s, j]
    qa = (torch.randn(S, H * Dk, device="cuda") * 0.1).bfloat16()
    seqs = [s if p >= 0 else -1 for s, p in enumerate(at)]
    ctx = types.SimpleNamespace(decode=True, tok_seq=_i32(seqs), tok_pos=_i32([max(p, 0) for p in at]))
    out = torch.full((S, H * C), 7.0, device="cuda").bfloat16()
    kernels.attention_latent(qa, out, cache, ctx, pages, 64, H, C, R, 0.3, rt=rt, window=window)
    for s, p in enumerate(at):
        if p < 0:
            assert bool((out[s] == 0).all())
            continue
        lo = max(0, p - window + 1) if window else 0
        k = rows[s, lo:p + 1].double()
        w = torch.softmax(qa[s].double().view(H, Dk) @ k.T * 0.3, dim=-1)
        want = (w @ k[:, :C]).reshape(-1)
        # weights and result rounded to bf16
        assert float((out[s].double() - want).abs().max()) <= 2.0 ** -7 * float(k.abs().max())


@pytest.mark.parametrize("H,C,R,S,n", [(4, 256, 32, 64, 2000), (8, 64, 16, 64, 2000), (16, 512, 64, 8, 2000)])
def test_reading_ahead_is_no_slower(H, C, R, S, n):
    """Launches in a row: with the next launch let go ahead of the wait, 64 sequences took 1.1 times as long as with nothing read ahead."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt, P, Dk = Runtime(torch.bfloat16, "cuda"), n // 64 + 1, C + R
    pages, cache = torch.randperm(S * P, device="cuda").int().view(S, P), torch.randn(S * P, 1, 64, Dk, device="cuda").bfloat16()
    qa, out = (torch.randn(S, H * Dk, device="cuda") * 0.1).bfloat16(), torch.empty(S, H * C, device="cuda").bfloat16()
    ctx = types.SimpleNamespace(decode=True, tok_seq=_i32(list(range(S))), tok_pos=_i32([n] * S))

    def us(early):
        side, graph, times = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
        run = lambda: kernels.attention_latent(qa, out, cache, ctx, pages, 64, H, C, R, 0.3, rt=rt, early=early)      # noqa: E731
        with torch.cuda.stream(side):
            run()
            side.synchronize()
            with torch.cuda.graph(graph, stream=side):
                for _ in range(20):
                    run()
        for _ in range(9):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end) * 50.0)
        return min(times)
    assert us(True) < 1.05 * us(False)


@pytest.mark.parametrize("K", [64, 128, 256, 1024, 2048])
@pytest.mark.parametrize("N,M", [(13, 4), (130, 5), (64, 8), (2, 7)])
@pytest.mark.parametrize("token", [True, False])
def test_per_head_products_on_either_kernel(K, N, M, token, monkeypatch):
    """The kernel of a few tokens and the tensor cores' tiles, whichever the choice by sizes is: around the former's batch of four."""
    from llmi_b200.ops import kernels
    monkeypatch.setattr(kernels, "heads_token_faster", lambda *sizes: token)
    torch.manual_seed(K + N + M)
    B, bx, by = 3, K + 8, N + N % 2 + 2
    x, w = torch.randn(M, B * bx, device="cuda").bfloat16(), (torch.randn(B, N, K, device="cuda") * K ** -0.5).bfloat16()
    out = torch.full((M, B * by), 7.0, device="cuda").bfloat16()
    kernels.linear_batched(x, bx, w, out, by, K, early=True)
    for b in range(B):
        want, got = x[:, b * bx:b * bx + K].double() @ w[b].double().T, out[:, b * by:b * by + N].double()
        size = x[:, b * bx:b * bx + K].double().abs() @ w[b].double().abs().T
        # the result's rounding, and a sum of K exact products in 32 bits
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + K ** 0.5 * 2.0 ** -23 * size).all())
        assert bool((out[:, b * by + N + N % 2:(b + 1) * by] == 7.0).all())
