"""The 32-bit path's product and attention at the edges of their tiles: against 64 bits, and bit for bit between the kernels
that a call's size selects (a position must not depend on how many others are in the step) (GPU)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from llmi_b200.ops import kernels
    return kernels


@pytest.mark.parametrize("N,K_", [(8, 4), (2000, 520), (7, 256), (65, 260), (129, 576), (200, 1020), (71, 1028), (64, 2560), (9, 4100), (17, 8192)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 15, 17, 33, 64, 65, 130])
def test_linear_f32_every_kernel_same_bits(M, N, K_):
    k = K()
    torch.manual_seed(M * 7 + N + K_)
    x = torch.randn(M, K_ + 8, device="cuda")[:, :K_]
    w, b, s = torch.randn(N, K_, device="cuda") / K_ ** 0.5, torch.randn(N, device="cuda"), torch.rand(N, device="cuda") + 0.5
    y = torch.full((M, N + 3), 7.0, device="cuda")
    k.linear_simt(x, w, y[:, :N], b, k.OUT_STORE, s)
    ref = (x.double() @ w.double().T + b.double()) * s.double()
    # a chain of 256 additions and one of K / 256: (256 + K / 256 + 2) roundings of 6e-8 of the terms' root sum of squares, at most
    bound = 6e-8 * (258 + K_ / 256) * float((x.double().abs() @ w.double().abs().T).max()) * 1.5
    assert float((y[:, :N].double() - ref).abs().max()) < bound
    assert float((y[:, :N].double() - ref).norm() / ref.norm()) < 1e-6
    assert bool((y[:, N:] == 7.0).all())
    # the same rows one by one, and through the kernel that takes any alignment
    one = torch.empty(1, N, device="cuda")
    for r in {0, M // 2, M - 1}:
        k.linear_simt(x[r:r + 1], w, one, b, k.OUT_STORE, s)
        assert torch.equal(one, y[r:r + 1, :N])
    odd = torch.empty(M * (K_ + 5) + 1, device="cuda")[1:].view(M, K_ + 5)[:, :K_]
    odd.copy_(x)
    z = torch.empty(M, N, device="cuda")
    k.linear_simt(odd, w, z, b, k.OUT_STORE, s)
    assert torch.equal(z, y[:, :N])
    acc = torch.randn(M, N, device="cuda")
    both = acc.clone()
    k.linear_simt(x, w, acc, None, k.OUT_ADD_F32)
    k.linear_simt(odd, w, both, None, k.OUT_ADD_F32)
    assert torch.equal(acc, both)
    k.check_device_errors("cuda:0")


def test_linear_f32_batched_same_bits():
    k = K()
    for M in (2, 70):
        x, w = torch.randn(M, 3 * 300, device="cuda"), torch.randn(3, 50, 300, device="cuda")
        out = torch.empty(M, 150, device="cuda")
        k.linear_batched(x, 300, w, out, 50, 300)
        for b in range(3):
            one = torch.empty(M, 50, device="cuda")
            k.linear_simt(x[:, 300 * b:300 * b + 300], w[b], one)
            assert torch.equal(out[:, 50 * b:50 * b + 50], one)
    k.check_device_errors("cuda:0")


def _context(q_lens, kv_lens, decode):
    lens = torch.tensor(q_lens)
    start = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)])
    seq = torch.repeat_interleave(torch.arange(len(q_lens)), lens)
    pos = torch.cat([torch.arange(k - q, k) for q, k in zip(q_lens, kv_lens)])
    i32 = lambda t: t.to(torch.int32).cuda()      # noqa: E731
    return types.SimpleNamespace(decode=decode, host_q_lens=list(q_lens), host_kv_lens=list(kv_lens), tok_seq=i32(seq), tok_pos=i32(pos),
                                 seq_q_start=i32(start), seq_kv_len=i32(torch.tensor(kv_lens)))


@pytest.mark.parametrize("nh,nkv,hd", [(3, 1, 64), (4, 4, 64), (6, 2, 36), (8, 2, 128), (10, 2, 8), (2, 2, 100)])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_f32_prompt_and_decode(nh, nkv, hd, window):
    """Prompts of unequal lengths on top of what is there, against 64 bits; every query alone as a decode step gives the same bits.
    What no query sees is NaN."""
    k = K()
    torch.manual_seed(nh * hd + window)
    q_lens, kv_lens = [1, 31, 32, 33, 70, 64], [1, 31, 96, 700, 70, 65]
    ctx = _context(q_lens, kv_lens, False)
    T, scale = sum(q_lens), hd ** -0.5
    P = max((n + 63) // 64 for n in kv_lens)
    pages = torch.full((len(q_lens), P), -1, dtype=torch.int32)
    order = torch.randperm(64)
    kc = torch.full((64, nkv, 64, hd), float("nan"), device="cuda")
    vc = kc.clone()
    n = 0
    refs = []
    q = torch.randn(T, nh * hd + 4, device="cuda")[:, :nh * hd]
    at = 0
    for i, (ql, kl) in enumerate(zip(q_lens, kv_lens)):
        keys, vals = torch.randn(kl, nkv, hd, device="cuda") * 2, torch.randn(kl, nkv, hd, device="cuda")
        for p in range((kl + 63) // 64):
            pages[i, p] = order[n]
            rows = slice(64 * p, min(kl, 64 * p + 64))
            kc[order[n], :, :rows.stop - rows.start] = keys[rows].transpose(0, 1)
            vc[order[n], :, :rows.stop - rows.start] = vals[rows].transpose(0, 1)
            n += 1
        qi = q[at:at + ql].double().view(ql, nh, hd)
        s = torch.einsum("qhd,khd->hqk", qi, keys.double().repeat_interleave(nh // nkv, 1)) * scale
        qp, kp = torch.arange(kl - ql, kl, device="cuda")[:, None], torch.arange(kl, device="cuda")[None]
        s.masked_fill_((kp > qp) | ((kp <= qp - window) if window else torch.zeros_like(kp > qp)), -float("inf"))
        refs.append(torch.einsum("hqk,khd->qhd", s.softmax(-1), vals.double().repeat_interleave(nh // nkv, 1)).reshape(ql, -1))
        at += ql
    pages = pages.cuda()
    out = torch.full((T, nh * hd), 7.0, device="cuda")
    assert k.attention_f32_applies(q, out, ctx, 64, nh, nkv, hd)
    k.attention(q, out, kc, vc, ctx, pages, 64, nh, nkv, hd, scale, window)
    ref = torch.cat(refs)
    assert float((out.double() - ref).norm() / ref.norm()) < 1e-6
    # token j of every sequence that has one, as a decode step, with a padding row between
    for j in (0, 17, 31, 32, 69):
        who = [i for i, ql in enumerate(q_lens) if ql > j]
        if not who:
            continue
        rows = [sum(q_lens[:i]) + j for i in who]
        one = _context([1] * len(who), [kv_lens[i] - q_lens[i] + j + 1 for i in who], True)
        one.tok_seq = torch.cat([one.tok_seq, torch.tensor([-1], dtype=torch.int32, device="cuda")])
        one.tok_pos = torch.cat([one.tok_pos, torch.tensor([0], dtype=torch.int32, device="cuda")])
        qd = torch.cat([q[rows], q[:1]]).contiguous()
        got = torch.full((len(who) + 1, nh * hd), 7.0, device="cuda")
        k.attention(qd, got, kc, vc, one, pages[who].contiguous(), 64, nh, nkv, hd, scale, window)
        assert torch.equal(got[:-1], out[rows]) and bool((got[-1] == 0).all())
    k.check_device_errors("cuda:0")


@pytest.mark.parametrize("M", [1, 8, 24])
def test_a_matrix_that_the_launch_ahead_writes(M):
    """Without ``early`` the second matrix may come out of the product just ahead, which lets the next launch start before it has
    ended."""
    k = K()
    torch.manual_seed(M)
    N, K_ = 24, 4096
    base, x = torch.randn(N, 512, device="cuda"), torch.randn(M, K_, device="cuda")
    w, y = torch.zeros(N, K_, device="cuda"), torch.empty(M, N, device="cuda")
    for _ in range(50):
        a = torch.randn(K_, 512, device="cuda") / 512 ** 0.5
        w.zero_()
        k.linear_simt(base, a, w)                    # w [N, 4096]: the launch ahead
        k.linear_simt(x, w, y)
        ref = x.double() @ (base.double() @ a.double().T).T
        assert float((y.double() - ref).norm() / ref.norm()) < 2e-6
        b = w.view(2, N // 2, K_)
        out = torch.empty(M, N, device="cuda")
        w.zero_()
        k.linear_simt(base, a, w)
        k.linear_batched(x, 0, b, out, N // 2, K_)
        assert torch.equal(out, y)
    k.check_device_errors("cuda:0")


def _us(f, reps=9, calls=20):
    f()
    times = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(calls):
            f()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / calls)
    return min(times)


@pytest.mark.parametrize("M,N,K_", [(1000, 4096, 64), (1000, 4096, 256), (3000, 1024, 128), (1000, 4096, 320), (24, 65536, 64)])
def test_products_of_short_k_are_no_slower_than_the_kernel_for_any_rows(M, N, K_):
    """fp32 rows of 16 bytes against rows that lie anywhere, which one kernel of the file takes (it took 0.4 to 0.8 times as long)."""
    k = K()
    y = torch.empty(M, N, device="cuda")

    def call(odd):
        x, w = (torch.randn(n * K_ + odd, device="cuda")[odd:].view(n, K_) for n in (M, N))
        return _us(lambda: k.linear_simt(x, w, y))
    assert call(0) < 1.15 * call(1)


@pytest.mark.parametrize("nkv,group,hd,S,n,q,window", [(32, 1, 64, 64, 100, 1, 0), (1, 16, 128, 1, 40, 1, 0), (1, 8, 64, 1, 60, 1, 0), (8, 4, 128, 64, 100, 1, 0),
                                                       (8, 4, 128, 64, 100, 2, 0), (1, 16, 128, 64, 1500, 4, 100), (8, 4, 128, 64, 1500, 2, 100)])
def test_short_sequences_are_no_slower_than_on_the_generic_kernel(nkv, group, hd, S, n, q, window):
    """Sequences of a page or two, and prompts of a few tokens each, against a warp per query and head (it took 0.3 to 0.8 times as
    long); the same numbers."""
    from llmi_b200.engine.runtime import Runtime
    k = K()
    torch.manual_seed(n)
    ctx = _context([q] * S, [n] * S, q == 1)
    P, nh = (n + 63) // 64, nkv * group
    pages = torch.randperm(S * P).to(torch.int32).view(S, P).cuda()
    kc, vc = (torch.randn(S * P, nkv, 64, hd, device="cuda") for _ in range(2))
    x = torch.randn(S * q, nh * hd, device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)
    rt = Runtime(torch.float32, "cuda:0")
    new = _us(lambda: k.attention(x, a, kc, vc, ctx, pages, 64, nh, nkv, hd, hd ** -0.5, window, rt=rt))
    old = _us(lambda: k.attention_generic(x, b, kc, vc, ctx.tok_seq, ctx.tok_pos, pages, 64, nh, nkv, hd, hd ** -0.5, window))
    assert float((a - b).norm() / b.norm()) < 1e-6
    assert new < 1.1 * old
    k.check_device_errors("cuda:0")


@pytest.mark.parametrize("nh,nkv,hd", [(30, 1, 16), (7, 1, 64), (5, 1, 128), (12, 2, 100), (40, 1, 64)])
def test_attention_f32_many_heads_a_kv_head(nh, nkv, hd):
    """Heads of a kv head cut over blocks, four, two and one at a time, with a remainder; fewer pages than warps; a prompt token by
    token and by blocks of 32 queries: the same bits, and 64 bits' result."""
    from llmi_b200.engine.runtime import Runtime
    k = K()
    torch.manual_seed(nh)
    rt, scale = Runtime(torch.float32, "cuda:0"), hd ** -0.5
    for S, n, q in ((1, 70, 1), (3, 300, 2), (60, 130, 2), (40, 10, 1)):
        ctx = _context([q] * S, [n] * S, False)
        P = (n + 63) // 64
        pages = torch.randperm(S * P).to(torch.int32).view(S, P).cuda()
        kc, vc = (torch.randn(S * P, nkv, 64, hd, device="cuda") for _ in range(2))
        x = torch.randn(S * q, nh * hd, device="cuda")
        outs = []
        rule = k.f32_by_token
        try:
            for by_token in (True, False):
                k.f32_by_token = lambda *a: by_token
                outs.append(torch.full_like(x, 7.0))
                k.attention(x, outs[-1], kc, vc, ctx, pages, 64, nh, nkv, hd, scale, rt=rt)
        finally:
            k.f32_by_token = rule
        assert torch.equal(outs[0], outs[1])
        s = 0
        at = pages[s].long()
        keys, vals = (c[at].transpose(1, 2).reshape(-1, nkv, hd)[:n].double().repeat_interleave(nh // nkv, 1) for c in (kc, vc))
        sc = torch.einsum("qhd,khd->hqk", x[:q].double().view(q, nh, hd), keys) * scale
        sc.masked_fill_(torch.arange(n, device="cuda")[None] > torch.arange(n - q, n, device="cuda")[:, None], -float("inf"))
        ref = torch.einsum("hqk,khd->qhd", sc.softmax(-1), vals).reshape(q, -1)
        assert float((outs[0][:q].double() - ref).norm() / ref.norm()) < 1e-6
    k.check_device_errors("cuda:0")
