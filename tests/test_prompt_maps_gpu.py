"""The prompt attention on the tcgen05 tensor cores with several maps a head, values of their own size, factors per head and an
fp32 output, against 64 bits (GPU)."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,maps,dk,dv,f32", [(4, 2, 2, 64, 128, True), (6, 2, 1, 64, 64, False), (4, 4, 1, 128, 128, False), (3, 1, 2, 64, 64, True),
                                                (2, 1, 3, 64, 128, False)])
@pytest.mark.parametrize("scaled,window,chunk", [(False, 0, 0), (True, 0, 1024), (True, 100, 0)])
def test_attention_maps_prompt_on_tcgen05(H, G, maps, dk, dv, f32, scaled, window, chunk):
    """Prompts of unequal lengths, some on top of what is there; a head's factor positive, negative, zero; a chunk that no
    sequence leaves; positions of nobody NaN; key ranges in one piece and cut."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    dev = "cuda"
    torch.manual_seed(H * dk + dv + maps)
    q_lens, held = [1, 128, 129, 300, 65], [0, 0, 64, 37, 200]
    kv_lens = [a + b for a, b in zip(q_lens, held)]
    starts = np.concatenate([[0], np.cumsum(q_lens)])
    T, scale = int(starts[-1]), dk ** -0.5
    pages_of = [(k + 63) // 64 for k in kv_lens]
    order, at = torch.randperm(sum(pages_of)), 0
    table = torch.full((len(q_lens), max(pages_of)), -1, dtype=torch.int32)
    kc = torch.full((sum(pages_of), G * maps, 64, dk), float("nan"), device=dev, dtype=torch.bfloat16)
    vc = torch.full((sum(pages_of), G, 64, dv), float("nan"), device=dev, dtype=torch.bfloat16)
    q = torch.randn(T, H * maps * dk, device=dev).bfloat16()
    factor = torch.tensor([1.5, -0.7, 0.0, 2.0, -1.0, 0.3], device=dev)[:H].contiguous() if scaled else None
    refs = []
    for i, (ql, kl) in enumerate(zip(q_lens, kv_lens)):
        keys, vals = torch.randn(kl, G * maps, dk, device=dev).bfloat16(), torch.randn(kl, G, dv, device=dev).bfloat16()
        for p in range(pages_of[i]):
            table[i, p] = order[at]
            n = min(64, kl - 64 * p)
            kc[order[at], :, :n] = keys[64 * p:64 * p + n].transpose(0, 1)
            vc[order[at], :, :n] = vals[64 * p:64 * p + n].transpose(0, 1)
            at += 1
        qi = q[starts[i]:starts[i + 1]].double().view(ql, H, maps, dk)
        kk = keys.double().view(kl, G, maps, dk).repeat_interleave(H // G, 1)
        s = torch.einsum("qhmd,khmd->hmqk", qi, kk) * scale
        if scaled:
            s = s * factor.double()[:, None, None, None]
        qp, kp = torch.arange(kl - ql, kl, device=dev)[:, None], torch.arange(kl, device=dev)[None]
        s.masked_fill_((kp > qp) | ((kp <= qp - window) if window else torch.zeros_like(kp > qp)), -float("inf"))
        refs.append(torch.einsum("hmqk,khd->qhmd", s.softmax(-1), vals.double().repeat_interleave(H // G, 1)).reshape(ql, -1))
    ref = torch.cat(refs)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    ctx = types.SimpleNamespace(decode=False, seq_q_start=i32(starts), seq_kv_len=i32(kv_lens), n_q_blocks=sum((x + 127) // 128 for x in q_lens),
                                tok_seq=i32(np.repeat(np.arange(len(q_lens)), q_lens)),
                                tok_pos=i32(np.concatenate([np.arange(k - n, k) for n, k in zip(q_lens, kv_lens)])),
                                host_q_lens=None, host_kv_lens=None)
    rt, out = Runtime(torch.bfloat16, dev), torch.full((T, H * maps * dv), 7.0, device=dev, dtype=torch.float32 if f32 else torch.bfloat16)
    seen = []
    tc = K.attention_prefill_tc
    K.attention_prefill_tc = lambda *a, **kw: (seen.append(1), tc(*a, **kw))
    try:
        for cut in (False, True):
            if cut:
                ctx.host_q_lens, ctx.host_kv_lens = q_lens, kv_lens
            out.fill_(7.0)
            K.attention_maps(q, out, kc, vc, ctx, table.to(dev), 64, H, G, maps, dk, dv, scale, factor, window, chunk, rt=rt)
            # weights and output in bf16, 2^-9 each, 0.6 of that in norm
            assert float((out.double() - ref).norm() / ref.norm()) < 1.2 * 2 ** -9 * 2 ** 0.5
    finally:
        K.attention_prefill_tc = tc
    assert len(seen) == 2
    K.check_device_errors("cuda:0")


def test_a_factor_that_is_no_number_stays_one():
    """A head whose factor is NaN gives NaN, as in the general kernel; the heads beside it, one with a factor of 0 among them, do
    not."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    dev, H, d, n = "cuda", 4, 64, 150
    torch.manual_seed(2)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    q, kc, vc = (torch.randn(s, device=dev).bfloat16() for s in ((n, H * d), (3, H, 64, d), (3, H, 64, d)))
    factor = torch.tensor([1.5, float("nan"), 0.0, -2.0], device=dev)
    ctx = types.SimpleNamespace(decode=False, seq_q_start=i32([0, n]), seq_kv_len=i32([n]), n_q_blocks=2, tok_seq=i32([0] * n), tok_pos=i32(range(n)),
                                host_q_lens=[n], host_kv_lens=[n])
    out, plain = (torch.full((n, H * d), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(2))
    seen, tc = [], K.attention_prefill_tc
    K.attention_prefill_tc = lambda *a, **kw: (seen.append(1), tc(*a, **kw))
    try:
        K.attention_maps(q, out, kc, vc, ctx, i32([[0, 1, 2]]), 64, H, H, 1, d, d, d ** -0.5, factor, rt=Runtime(torch.bfloat16, dev))
    finally:
        K.attention_prefill_tc = tc
    K.attention_flex(q, plain, kc, vc, ctx, i32([[0, 1, 2]]), 64, H, H, 1, d, d, d ** -0.5, factor)
    assert seen and torch.equal(out.isnan(), plain.isnan()) and bool(out.view(n, H, d)[:, 1].isnan().all())
    rest = [0, 2, 3]
    a, b = out.view(n, H, d)[:, rest].double(), plain.view(n, H, d)[:, rest].double()
    assert float((a - b).norm() / b.norm()) < 1.2 * 2 ** -9 * 2 ** 0.5
    K.check_device_errors("cuda:0")


@pytest.mark.parametrize("maps", [16, 17, 40])
def test_any_number_of_maps(maps):
    """More maps a head than anybody has: the general kernel's result."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    dev, H, dk, dv, n = "cuda", 2, 64, 128, 100
    torch.manual_seed(maps)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    q, kc, vc = (torch.randn(s, device=dev).bfloat16() for s in ((n, H * maps * dk), (2, maps, 64, dk), (2, 1, 64, dv)))
    ctx = types.SimpleNamespace(decode=False, seq_q_start=i32([0, n]), seq_kv_len=i32([n]), n_q_blocks=1, tok_seq=i32([0] * n), tok_pos=i32(range(n)),
                                host_q_lens=[n], host_kv_lens=[n])
    out, plain = (torch.empty(n, H * maps * dv, device=dev) for _ in range(2))
    K.attention_maps(q, out, kc, vc, ctx, i32([[0, 1]]), 64, H, 1, maps, dk, dv, dk ** -0.5, rt=Runtime(torch.bfloat16, dev))
    K.attention_flex(q, plain, kc, vc, ctx, i32([[0, 1]]), 64, H, 1, maps, dk, dv, dk ** -0.5)
    assert float((out - plain).norm() / plain.norm()) < 1.2 * 2 ** -9 * 2 ** 0.5
    K.check_device_errors("cuda:0")
