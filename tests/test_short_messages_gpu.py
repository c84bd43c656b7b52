"""The attention of short messages on long histories at the edges of its tiles (GPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from llmi_b200.ops import kernels
    return kernels


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("group", [1, 3, 4, 16])
@pytest.mark.parametrize("window", [0, 100])
def test_attention_short(hd, group, window):
    """Messages of unequal lengths (one token, edges of the row tiles, none at all) on histories that end at the edges of
    pages, every way to share the pages, against 64 bits; positions that no query sees are NaN.  P and the output are bf16:
    a relative error of 2^-9 each, at most 0.6 of that in norm."""
    k = K()
    torch.manual_seed(hd + group + window)
    nkv, dev = 2, "cuda"
    nh = nkv * group
    q_lens = [1, 64 // group, 0, 7, 17, 48 if group < 4 else 31, 9]
    held = [0, 63, 0, 64, 700, 130, 1000]
    n_seqs, kv_lens = len(q_lens), [h + q for h, q in zip(held, q_lens)]
    pages_of = [(n + 63) // 64 for n in kv_lens]
    table = torch.full((n_seqs, max(pages_of) + 1), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(pages_of)), 0
    kc = torch.full((sum(pages_of), nkv, 64, hd), float("nan"), device=dev, dtype=torch.bfloat16)
    vc = kc.clone()
    starts = np.concatenate([[0], np.cumsum(q_lens)])
    T, scale = int(starts[-1]), hd ** -0.5
    q = torch.randn(T, nh * hd + 8, device=dev, dtype=torch.bfloat16)[:, :nh * hd]
    refs = []
    for i, (ql, kl) in enumerate(zip(q_lens, kv_lens)):
        keys, vals = (torch.randn(kl, nkv, hd, device=dev).to(torch.bfloat16) for _ in range(2))
        for p in range(pages_of[i]):
            table[i, p] = order[at]
            rows = slice(64 * p, min(kl, 64 * p + 64))
            kc[order[at], :, :rows.stop - rows.start] = keys[rows].transpose(0, 1)
            vc[order[at], :, :rows.stop - rows.start] = vals[rows].transpose(0, 1)
            at += 1
        if ql == 0:
            continue
        s = torch.einsum("qhd,khd->hqk", q[starts[i]:starts[i + 1]].double().view(ql, nh, hd), keys.double().repeat_interleave(group, 1)) * scale
        qp, kp = torch.arange(kl - ql, kl, device=dev)[:, None], torch.arange(kl, device=dev)[None]
        s.masked_fill_((kp > qp) | ((kp <= qp - window) if window else torch.zeros_like(kp > qp)), -float("inf"))
        refs.append(torch.einsum("hqk,khd->qhd", s.softmax(-1), vals.double().repeat_interleave(group, 1)).reshape(ql, -1))
    ref = torch.cat(refs)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    for parts in (1, 2, 4, 8):
        out = torch.full((T, nh * hd), 7.0, device=dev, dtype=torch.bfloat16)
        k.attention_short(q, out, kc, vc, table.to(dev), i32(starts), i32(kv_lens), max(q_lens), nh, nkv, hd, scale, window, parts)
        assert float((out.double() - ref).norm() / ref.norm()) < 1.2 * 2 ** -9 * 2 ** 0.5, parts
    k.check_device_errors("cuda:0")
