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


@pytest.mark.parametrize("hd,group", [(64, 1), (64, 3), (128, 4), (128, 16)])
@pytest.mark.parametrize("window,rot,write", [(0, True, True), (200, True, True), (0, False, True), (0, True, False)])
def test_attention_short_decode_same_bits(hd, group, window, rot, write):
    """A decode step with the position encoding inside gives, however the pages are shared, the bits of the same kernel behind the
    kernel that rotates and appends, and that kernel's cache: lengths at the edges of pages, a padding sequence, positions of
    nobody NaN.  (Against 64 bits: test_attention_short_small_tiles.)"""
    k = K()
    nkv = 2
    nh, dev = nkv * group, "cuda"
    torch.manual_seed(hd * group)
    lens, P = [1, 64, 65, 700, 0, 129, 1000, 128], 16                     # lengths after the step (0: padding)
    S, n_pages = len(lens), 48
    order = torch.randperm(n_pages)
    table, at = torch.full((S, P), -1, dtype=torch.int32), 0
    kc = torch.full((n_pages, nkv, 64, hd), float("nan"), device=dev, dtype=torch.bfloat16)
    vc = kc.clone()
    for s, n in enumerate(lens):
        for p in range((n + 63) // 64):
            table[s, p] = order[at]
            there = min(64, n - (1 if write else 0) - 64 * p)
            if there > 0:
                kc[order[at], :, :there] = torch.randn(nkv, there, hd, device=dev).bfloat16()
                vc[order[at], :, :there] = torch.randn(nkv, there, hd, device=dev).bfloat16()
            at += 1
    qkv = torch.randn(S, (nh + 2 * nkv) * hd, device=dev).bfloat16()
    inv = torch.rand(hd // 2, device=dev)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    pages, kvlen, starts = table.to(dev), i32(lens), i32(list(range(S + 1)))
    seq, pos = i32([i if n else -1 for i, n in enumerate(lens)]), i32([max(n - 1, 0) for n in lens])
    q_rot, kr, vr = qkv.clone(), kc.clone(), vc.clone()
    k.rope_store(q_rot, inv, hd if rot else 0, seq, pos, pages, 64, kr, vr, nh, nkv, hd, write)
    for parts in (1, 2, 4, 8):
        outs = [torch.full((S, nh * hd), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(2)]
        k.attention_short(q_rot, outs[0], kr, vr, pages, starts, kvlen, 1, nh, nkv, hd, hd ** -0.5, window, parts)
        k1, v1 = kc.clone(), vc.clone()
        k.attention_short(qkv, outs[1], k1, v1, pages, starts, kvlen, 1, nh, nkv, hd, hd ** -0.5, window, parts,
                          (inv, hd if rot else 0, write))
        assert torch.equal(outs[0], outs[1]) and bool((outs[1][4] == 7.0).all()) and bool(torch.isfinite(outs[1].float()).all())
        for a, b in ((kr, k1), (vr, v1)):
            assert torch.equal(torch.nan_to_num(a.float(), nan=-7.0), torch.nan_to_num(b.float(), nan=-7.0))
    k.check_device_errors("cuda:0")


@pytest.mark.parametrize("nkv,hd,S,pages,parts", [(32, 64, 24, 12, 0), (16, 128, 24, 3, 1), (16, 128, 4, 16, 4), (8, 128, 2, 52, 8)])
@pytest.mark.parametrize("fused", [True, False])
def test_ungrouped_decode_has_32_bit_weights(nkv, hd, S, pages, parts, fused):
    """A decode step of ungrouped heads, by the kernel that ``attention`` sends it to and by the one that has the other sizes:
    values whose weighted sum all but cancels, so that weights rounded to bf16 would be as wrong as the result is large.  With
    32-bit ones: the output's rounding (at most 2^-8; spread evenly over that, 1 / sqrt(3) of it in norm) and, of the terms' norm
    (at most 2^9.3 times the result's), the scores' and exponentials' 2^-21 in all."""
    import types
    from llmi_b200.engine.runtime import Runtime
    k = K()
    dev = "cuda"
    torch.manual_seed(nkv + S)
    lens = [64 * pages - 17 * (s % 3) for s in range(S)]
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    table = i32(torch.randperm(S * pages).view(S, pages))
    kc = torch.randn(S * pages, nkv, 64, hd, device=dev).bfloat16()
    vc = torch.full_like(kc, float("nan"))
    qkv = torch.randn(S, 3 * nkv * hd, device=dev).bfloat16()
    scale, ref, terms = hd ** -0.5, [], 0.0
    for s, n in enumerate(lens):
        at = table[s].long()
        keys = kc[at].transpose(1, 2).reshape(-1, nkv, hd)[:n].double()
        if fused:                                              # (nothing turns: the new key is the row's own)
            keys[-1] = qkv[s, nkv * hd:2 * nkv * hd].view(nkv, hd).double()
        p = (torch.einsum("hd,khd->hk", qkv[s, :nkv * hd].view(nkv, hd).double(), keys) * scale).softmax(-1)
        r = torch.randn(n, nkv, hd, device=dev, dtype=torch.float64)
        vals = (r - torch.einsum("hk,khd->hd", p, r)).bfloat16()
        if fused:
            qkv[s, 2 * nkv * hd:] = vals[-1].reshape(-1)
        full = torch.full((64 * pages, nkv, hd), float("nan"), device=dev, dtype=torch.bfloat16)
        full[:n] = vals
        vc[at] = full.view(pages, 64, nkv, hd).transpose(1, 2)
        ref.append(torch.einsum("hk,khd->hd", p, vals.double()).reshape(-1))
        terms = max(terms, float(torch.einsum("hk,khd->hd", p ** 2, vals.double() ** 2).sqrt().norm() / ref[-1].norm()))
    ref = torch.stack(ref)
    assert terms < 2 ** 9.3
    ctx = types.SimpleNamespace(decode=True, seq_q_start=i32(range(S + 1)), seq_kv_len=i32(lens), tok_seq=i32(range(S)),
                                tok_pos=i32([n - 1 for n in lens]), n_real_seqs=S, host_q_lens=None, host_kv_lens=None)
    assert k.decode_short_parts(S, nkv, pages, hd, 1) == parts
    rt, rope = Runtime(torch.bfloat16, dev), (None, 0, True) if fused else None
    errors = []
    rule = k.decode_short_parts
    try:
        for other in (False, True):
            if other:
                k.decode_short_parts = lambda *a: 0
            out = torch.full((S, nkv * hd), 7.0, device=dev, dtype=torch.bfloat16)
            k.attention(qkv, out, kc.clone(), vc.clone(), ctx, table, 64, nkv, nkv, hd, scale, rt=rt, rope=rope)
            errors.append(float((out.double() - ref).norm() / ref.norm()))
    finally:
        k.decode_short_parts = rule
    assert max(errors) < 2 ** -8 / 3 ** 0.5 + 2 ** (9.3 - 21), errors
    k.check_device_errors("cuda:0")


def _small_llama(tmp_path, heads, kv_heads, head_dim):
    import llmi_b200 as L
    d = str(tmp_path / f"m{heads}_{kv_heads}_{head_dim}")
    L.write_random_model(d, {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": 2, "hidden_size": 256, "num_attention_heads": heads,
                             "num_key_value_heads": kv_heads, "head_dim": head_dim, "intermediate_size": 512, "vocab_size": 300,
                             "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": True, "max_position_embeddings": 1024,
                             "hidden_act": "silu"}, 3, torch.bfloat16)
    return L.load(d, "bfloat16")


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(6, 2, 64), (4, 4, 64), (8, 2, 128), (4, 2, 32)])
def test_recorded_messages_of_one_padded_shape(tmp_path, heads, kv_heads, head_dim):
    """Messages of one padded shape (as many tokens in all, page tables as wide) but of other lengths, one step after another, so
    that recordings made for some meet others: the logits of steps that are neither padded nor recorded.  A recording is told
    apart by what its launches follow, so heads that attention_short does not take share one."""
    import llmi_b200 as L
    from llmi_b200.engine import graphs
    from llmi_b200.ops import kernels
    if not graphs.RECORD:
        pytest.skip("recording is switched off")
    model = _small_llama(tmp_path, heads, kv_heads, head_dim)
    rng = np.random.default_rng(1)
    held, messages = [260, 300, 280, 310], [[4, 4, 4, 4], [13, 1, 1, 1], [1, 1, 2, 12], [4, 3, 4, 4], [2, 12, 1, 1], [3, 4, 4, 4], [1, 2, 10, 2], [4, 4, 4, 4]]
    caches = [model.new_cache(4 * 1024) for _ in range(2)]
    slots = [[c.alloc_slot() for _ in held] for c in caches]
    toks = [rng.integers(0, 300, n).tolist() for n in held]
    for c, s in zip(caches, slots):
        for slot, t in zip(s, toks):
            model.step(c, [L.SequenceStep(slot, t, [])])
    g = model._prompt_graphs
    before, had = g.replays, set(g.graphs)
    plans = set()
    for lens in messages:
        new = [rng.integers(0, 300, n).tolist() for n in lens]
        got, want = (model.step(c, [L.SequenceStep(slot, t, list(range(len(t)))) for slot, t in zip(s, new)], **kw).clone()
                     for c, s, kw in ((caches[0], slots[0], {}), (caches[1], slots[1], {"pad_pages_to": 1})))
        # every row: bf16 roundings of another batch's products, two layers deep; a row that no launch wrote would be of another size
        assert bool(((got - want).norm(dim=1) < 2e-2 * want.norm(dim=1)).all()), lens
        short = 4 if max(lens) <= 4 else 16
        parts = kernels.attention_short_parts(4, kv_heads, short, heads // kv_heads, 8, head_dim) if head_dim != 32 else 0
        rows = short * heads // kv_heads
        plans.add((parts, 16 if rows <= 16 else 32 if rows <= 32 else -(-rows // 64) * 64) if parts else ())
    assert len(set(g.graphs) - had) == len(plans) and g.replays - before == len(messages) - 2 * len(plans)
    assert len(plans) == (1 if head_dim == 32 or heads == kv_heads else 2)
    kernels.check_device_errors("cuda:0")


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("group,max_q", [(1, 1), (4, 1), (16, 1), (1, 16), (3, 5), (5, 3), (1, 17), (3, 9), (8, 4), (16, 2), (2, 16)])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_short_small_tiles(hd, group, max_q, window):
    """The tiles of 16 and of 32 rows, whose warps share a page's keys: messages of up to so many tokens (decode steps among them,
    and the form with 32-bit weights) on histories that end at the edges of pages and of the warps' keys, every way to share
    the pages, against 64 bits; positions that no query sees are NaN."""
    k = K()
    torch.manual_seed(hd + group + max_q + window)
    nkv, dev = 2, "cuda"
    nh = nkv * group
    q_lens = [max_q, 1, max(1, max_q // 2), max_q, max_q, 1, max_q, max_q]
    held = [0, 15, 16, 31, 63, 64, 700, 1000]
    S, kv_lens = len(q_lens), [h + q for h, q in zip(held, q_lens)]
    pages_of = [(n + 63) // 64 for n in kv_lens]
    table = torch.full((S, max(pages_of) + 1), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(pages_of)), 0
    kc = torch.full((sum(pages_of), nkv, 64, hd), float("nan"), device=dev, dtype=torch.bfloat16)
    vc = kc.clone()
    starts = np.concatenate([[0], np.cumsum(q_lens)])
    T, scale = int(starts[-1]), hd ** -0.5
    q = torch.randn(T, nh * hd, device=dev, dtype=torch.bfloat16)
    refs = []
    for i, (ql, kl) in enumerate(zip(q_lens, kv_lens)):
        keys, vals = (torch.randn(kl, nkv, hd, device=dev).to(torch.bfloat16) for _ in range(2))
        for p in range(pages_of[i]):
            table[i, p] = order[at]
            n = min(64, kl - 64 * p)
            kc[order[at], :, :n], vc[order[at], :, :n] = keys[64 * p:64 * p + n].transpose(0, 1), vals[64 * p:64 * p + n].transpose(0, 1)
            at += 1
        s = torch.einsum("qhd,khd->hqk", q[starts[i]:starts[i + 1]].double().view(ql, nh, hd), keys.double().repeat_interleave(group, 1)) * scale
        qp, kp = torch.arange(kl - ql, kl, device=dev)[:, None], torch.arange(kl, device=dev)[None]
        s.masked_fill_((kp > qp) | ((kp <= qp - window) if window else torch.zeros_like(kp > qp)), -float("inf"))
        refs.append(torch.einsum("hqk,khd->qhd", s.softmax(-1), vals.double().repeat_interleave(group, 1)).reshape(ql, -1))
    ref = torch.cat(refs)
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    for parts in (1, 2, 4, 8):
        for wide in (False, True) if max_q == 1 and group == 1 and hd == 128 else (False,):
            out = torch.full((T, nh * hd), 7.0, device=dev, dtype=torch.bfloat16)
            k.attention_short(q, out, kc, vc, table.to(dev), i32(starts), i32(kv_lens), max_q, nh, nkv, hd, scale, window, parts, wide=wide)
            # row by row, so that no single row's mistake is lost in the others: weights and output in bf16, 2^-8 at most each
            assert bool(((out.double() - ref).norm(dim=1) < 2 ** -8 * 2 ** 0.5 * ref.norm(dim=1)).all()), (parts, wide)
    k.check_device_errors("cuda:0")
