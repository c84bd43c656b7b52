"""Latent attention of prompts in its expanded form at the edges of its tiles, against 64 bits (GPU)."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,D,R,C,rot_dims,pairing", [(3, 128, 64, 512, 64, 1), (4, 64, 32, 256, 32, 1), (2, 64, 64, 64, 40, 0), (5, 128, 8, 192, 8, 0),
                                                      (2, 128, 0, 128, 0, 1)])
@pytest.mark.parametrize("spare", [0, 3])
def test_attention_expanded(H, D, R, C, rot_dims, pairing, spare):
    """Prompts of unequal lengths, some on top of what is there, one sequence without tokens, rows of no sequence behind;
    positions and pages of nobody are NaN.  ``spare``: pages more than the sequences have (a step padded to a shape)."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    dev = "cuda"
    torch.manual_seed(H * D + R)
    q_lens, held = [1, 128, 0, 129, 300, 65], [0, 0, 0, 64, 37, 200]
    kv_lens = [a + b for a, b in zip(q_lens, held)]
    kv_lens[2] = 70                                                   # (it has rows, but brings nothing)
    starts = np.concatenate([[0], np.cumsum(q_lens)])
    n, T = int(starts[-1]), int(starts[-1]) + 5
    pages_of = [(k + 63) // 64 for k in kv_lens]
    order, at = torch.randperm(sum(pages_of) + 1), 0
    table = torch.full((len(q_lens), max(pages_of)), -1, dtype=torch.int32)
    cache = torch.full((sum(pages_of) + 1, 1, 64, C + R), float("nan"), device=dev, dtype=torch.bfloat16)
    q = torch.randn(T, H * (D + R), device=dev, dtype=torch.bfloat16)
    uk, uv = (torch.randn(H, D, C, device=dev) / C ** 0.5).bfloat16(), (torch.randn(H, D, C, device=dev) / C ** 0.5).bfloat16()
    inv = torch.from_numpy(np.power(1e4, -2.0 * np.arange(max(rot_dims // 2, 1)) / max(rot_dims, 1)).astype(np.float32)).to(dev)
    scale, amp = (D + R) ** -0.5, 1.25
    refs = []
    for i, (ql, kl) in enumerate(zip(q_lens, kv_lens)):
        rows = torch.randn(kl, C + R, device=dev).bfloat16()
        for p in range(pages_of[i]):
            table[i, p] = order[at]
            cache[order[at], 0, :min(64, kl - 64 * p)] = rows[64 * p:64 * p + 64]
            at += 1
        if not ql:
            continue
        qi = q[starts[i]:starts[i + 1]].view(ql, H, D + R).double()
        ang = torch.arange(kl - ql, kl, device=dev, dtype=torch.float32)[:, None] * inv[:rot_dims // 2]
        cos, sin = (ang.cos().double() * amp)[:, None], (ang.sin().double() * amp)[:, None]
        rot = qi[..., D:].clone()
        a, b = (slice(0, rot_dims, 2), slice(1, rot_dims, 2)) if pairing else (slice(0, rot_dims // 2), slice(rot_dims // 2, rot_dims))
        u, v = rot[..., a].clone(), rot[..., b].clone()
        rot[..., a], rot[..., b] = u * cos - v * sin, v * cos + u * sin
        c, r = rows[:, :C].double(), rows[:, C:].double()
        k, val = torch.einsum("hdc,sc->shd", uk.double(), c), torch.einsum("hdc,sc->shd", uv.double(), c)
        s = (torch.einsum("qhd,shd->hqs", qi[..., :D], k) + torch.einsum("qhr,sr->hqs", rot, r)) * scale
        s.masked_fill_(torch.arange(kl, device=dev)[None] > torch.arange(kl - ql, kl, device=dev)[:, None], -float("inf"))
        refs.append(torch.einsum("hqs,shd->qhd", s.softmax(-1), val).reshape(ql, -1))
    i32 = lambda x: torch.as_tensor(x).to(torch.int32).to(dev)      # noqa: E731
    seq = np.concatenate([np.repeat(np.arange(len(q_lens)), q_lens), [-1] * 5])
    pos = np.concatenate([np.arange(k - ql, k) for ql, k in zip(q_lens, kv_lens)] + [np.zeros(5, dtype=int)])
    ctx = types.SimpleNamespace(decode=False, seq_q_start=i32(starts), seq_kv_len=i32(kv_lens), tok_seq=i32(seq), tok_pos=i32(pos),
                                n_q_blocks=sum((x + 127) // 128 for x in q_lens) + spare, host_q_lens=q_lens, host_kv_lens=kv_lens)
    n_pages = K.latent_expanded_pages(ctx, T, table, H, D)
    assert n_pages == sum(p for p, ql in zip(pages_of, q_lens) if ql)
    rows = 64 * (n_pages + spare)
    rt = Runtime(torch.bfloat16, dev)
    assert K.attention_expanded_supported(rt, D, D, R, C, scale)
    xc, xr, qr = (torch.full(s, float("nan"), device=dev, dtype=torch.bfloat16) for s in ((rows, C), (rows, 64), (T, H * 64)))
    K.latent_expand_prepare(cache, ctx, table.to(dev), xc, xr, q, qr, H, D, R, inv, rot_dims, pairing, amp)
    kv = torch.empty(rows, H * 2 * D, device=dev, dtype=torch.bfloat16)
    K.linear(xc, torch.cat([uk, uv], dim=1).reshape(H * 2 * D, C).contiguous(), kv)
    out = torch.full((T, H * D), 7.0, device=dev, dtype=torch.bfloat16)
    K.attention_expanded(q, qr, kv, xr, out, ctx, H, D, R, scale)
    ref = torch.cat(refs)
    # rounded to bf16 (2^-9 each, 0.6 of that in norm): the rotated queries and the keys (through scores of size about 1), the
    # weights, the values and the output
    assert float((out[:n].double() - ref).norm() / ref.norm()) < 1.2 * 2 ** -9 * 5 ** 0.5
    assert bool((out[n:] == 7.0).all())
    K.check_device_errors("cuda:0")


@pytest.mark.parametrize("page_size", [16, 32, 64, 128])
def test_latent_part_on_pages_of_any_size(page_size):
    """A prompt of as many tokens as the expanded form takes, and a second one on top of it, through the mixer: what the cache's
    page size is does not matter (the expanded form is for pages of 64; the others keep the form on the latent rows)."""
    from llmi_b200.cache.storage import CacheBinding, SequenceCache
    from llmi_b200.engine.batch import SequenceStep, StepBuffers, plan_step
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    from llmi_b200.parts import PartSpec, get_part
    W, H, D, R, C, Q = 128, 2, 64, 32, 64, 64
    params = {"width": W, "heads": H, "dim": D, "rot_dim": R, "vdim": D, "kv_rank": C, "q_rank": Q, "scale": (D + R) ** -0.5, "rot_base": 1e4,
              "eps": 1e-6}
    make = get_part("mixer", "latent_attention")
    torch.manual_seed(5)
    tensors = {n: (torch.ones(d.shape) if n.endswith("norm") else torch.randn(d.shape) * d.shape[1] ** -0.5)
               for n, d in make.declare(PartSpec("latent_attention", params, "")).items()}
    h = torch.randn(300, W, device="cuda")
    outs = {}
    for dtype, size in ((torch.float32, 64), (torch.bfloat16, page_size)):
        rt = Runtime(dtype, "cuda:0")
        part = make(PartSpec("latent_attention", params, ""), {n: t.to(dtype).float() for n, t in tensors.items()}, rt)
        cache = SequenceCache([(part.cache_request(), 1)], [], 512, 512, dtype, "cuda:0", page_size=size)
        buffers, slot, rows = StepBuffers("cuda:0"), cache.alloc_slot(), []
        for a, b in ((0, 160), (160, 300)):
            ctx = plan_step(cache, [SequenceStep(slot, list(range(b - a)), [])], 1000, buffers)
            x = torch.zeros(b - a, W, device="cuda")
            part.forward(h[a:b].to(dtype), x, ctx, CacheBinding(cache.kv_groups[0], 0))
            rows.append(x)
        outs[dtype] = torch.cat(rows).double()
    ref = outs[torch.float32]
    # rounded to bf16 (2^-8 at most, 1 / sqrt(3) of that in norm), one after another: weights (five products deep), input, latents, rows,
    # queries, keys or folded queries, weights of the sum, values or sums, heads: at most 16 in all
    assert float((outs[torch.bfloat16] - ref).norm() / ref.norm()) < 4 * 2 ** -8 / 3 ** 0.5
    K.check_device_errors("cuda:0")


def test_expanded_form_keeps_no_more_than_its_bound(monkeypatch):
    """A prompt that grows portion by portion: the buffers of keys and values, which double as they grow, stop at the bound; beyond
    it the step works on the latent rows."""
    from llmi_b200.cache.storage import CacheBinding, SequenceCache
    from llmi_b200.engine.batch import SequenceStep, StepBuffers, plan_step
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels as K
    from llmi_b200.parts import PartSpec, get_part
    W, H, D, R, C = 128, 2, 64, 32, 64
    params = {"width": W, "heads": H, "dim": D, "rot_dim": R, "vdim": D, "kv_rank": C, "q_rank": 64, "scale": (D + R) ** -0.5, "rot_base": 1e4,
              "eps": 1e-6}
    make, spec = get_part("mixer", "latent_attention"), PartSpec("latent_attention", params, "")
    bound = 700 * H * 2 * D * 2                                   # 700 rows: ten pages of 64
    monkeypatch.setattr(K, "EXPANDED_MAX_BYTES", bound)
    rt = Runtime(torch.bfloat16, "cuda:0")
    part = make(spec, {n: (torch.ones(d.shape) if n.endswith("norm") else torch.randn(d.shape) * 0.1) for n, d in make.declare(spec).items()}, rt)
    cache = SequenceCache([(part.cache_request(), 1)], [], 1024, 1024, torch.bfloat16, "cuda:0")
    buffers, slot = StepBuffers("cuda:0"), cache.alloc_slot()
    for n in range(6):                                            # 2, 4, .. pages; 10 are the most, 12 are too many
        ctx = plan_step(cache, [SequenceStep(slot, [1] * 128, [])], 1000, buffers)
        part.forward(torch.randn(128, W, device="cuda").bfloat16(), torch.zeros(128, W, device="cuda"), ctx, CacheBinding(cache.kv_groups[0], 0))
        used = rt._buffers["latent_kv"].numel()
        assert min(128 * (n + 1), 640) * H * 2 * D <= used <= 640 * H * 2 * D and 2 * used <= bound
        assert rt._buffers["latent_xc"].numel() <= 640 * C and rt._buffers["latent_xr"].numel() <= 640 * 64
    K.check_device_errors("cuda:0")
