"""Kernels that may start before the launch ahead has ended, with that launch still at work (GPU).

Every test puts a launch of two blocks in front that lets the next ones start at once and takes longer than the host needs to
launch them all (half a millisecond); the kernel that writes the step's own row waits for it, and the reader under test is
launched directly behind the writer."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu

ROUNDS = 15


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _long_launch():
    from llmi_b200.ops import kernels
    K = 1 << 19
    x, w, y = torch.ones(1, K, device="cuda"), torch.ones(16, K, device="cuda"), torch.empty(1, 16, device="cuda")
    return lambda: kernels.linear_simt(x, w, y)


def _token_ctx(positions):
    """A step in which sequence s brings the token at ``positions[s]``."""
    S, kv = len(positions), [p + 1 for p in positions]
    return types.SimpleNamespace(decode=True, n_seqs=S, n_real_seqs=S, tok_seq=_i32(list(range(S))), tok_pos=_i32(positions),
                                 seq_q_start=_i32(list(range(S + 1))), seq_kv_len=_i32(kv), seq_slot=_i32(list(range(S))),
                                 host_q_lens=[1] * S, host_kv_lens=kv)


def _check(reset, steps):
    """``steps``: functions of one launch or more each.  Run with the device idle between them, then in a row."""
    hold = _long_launch()
    want = []
    reset()
    for step in steps:
        torch.cuda.synchronize()
        want.append(step().clone())
    assert all(bool(torch.isfinite(w).all()) for w in want)
    for _ in range(ROUNDS):
        reset()
        hold()
        got = [step() for step in steps]
        for g, w in zip(got, want):
            assert torch.equal(g, w)


POSITIONS = [0, 1, 62, 63, 64, 126, 127, 300]


@pytest.mark.parametrize("C,R", [(512, 64), (64, 16)])
@pytest.mark.parametrize("early", [True, False])
def test_latent_rows(C, R, early):
    """``early``: the newest row is still to be written when the reader starts.  Without: so is the row before it, which the step
    before makes in the same row of launches."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt = Runtime(torch.bfloat16, "cuda")
    torch.manual_seed(C)
    H, Q, S, P, Dk = 16, 128, len(POSITIONS), 6, C + R
    pages = torch.randperm(S * P, device="cuda").int().view(S, P)
    full = torch.randn(S * P, 1, 64, Dk, device="cuda").bfloat16()
    cache = torch.empty_like(full)
    wq, wc, inv = torch.ones(Q, device="cuda"), torch.ones(C, device="cuda"), torch.rand(R // 2, device="cuda")
    steps = []
    for s, p in enumerate(POSITIONS):                    # (what the steps do not write stays no number)
        for j in range(p, 64 * P):
            full[pages[s, j // 64], 0, j % 64] = float("nan")
    for positions in [POSITIONS] if early else [POSITIONS, [p + 1 for p in POSITIONS]]:
        ctx, down = _token_ctx(positions), torch.randn(S, Q + C + R, device="cuda")
        cq, qa = torch.empty(S, Q, device="cuda").bfloat16(), (torch.randn(S, H * Dk, device="cuda") * 0.1).bfloat16()
        out = torch.empty(S, H * C, device="cuda").bfloat16()

        def step(ctx=ctx, down=down, cq=cq, qa=qa, out=out):
            kernels.latent_prepare(down, Q, C, R, wq, wc, 1e-5, inv, R, ctx, pages, 64, cache, cq)
            kernels.attention_latent(qa, out, cache, ctx, pages, 64, H, C, R, 0.3, rt=rt, early=early)
            return out
        steps.append(step)
    _check(lambda: cache.copy_(full), steps)


@pytest.mark.parametrize("Hq,G,maps,dk,dv,window", [(4, 2, 2, 64, 64, 0), (16, 8, 1, 128, 128, 0), (6, 2, 2, 64, 128, 70)])
@pytest.mark.parametrize("early", [True, False])
def test_rows_of_several_maps(Hq, G, maps, dk, dv, window, early):
    """As above, for keys and values in pages of their own."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt = Runtime(torch.bfloat16, "cuda")
    torch.manual_seed(Hq + dk)
    S, P, N, Nk, Nv = len(POSITIONS), 6, Hq * maps * dk, G * maps * dk, G * dv
    pages = torch.randperm(S * P, device="cuda").int().view(S, P)
    k_full, v_full = torch.randn(S * P, G * maps, 64, dk, device="cuda").bfloat16(), torch.randn(S * P, G, 64, dv, device="cuda").bfloat16()
    for s, p in enumerate(POSITIONS):
        for j in range(p, 64 * P):
            k_full[pages[s, j // 64], :, j % 64] = v_full[pages[s, j // 64], :, j % 64] = float("nan")
    kc, vc = torch.empty_like(k_full), torch.empty_like(v_full)
    steps = []
    for positions in [POSITIONS] if early else [POSITIONS, [p + 1 for p in POSITIONS]]:
        ctx, proj = _token_ctx(positions), torch.randn(S, N + Nk + Nv, device="cuda")
        q, out = torch.empty(S, N, device="cuda").bfloat16(), torch.empty(S, Hq * maps * dv, device="cuda").bfloat16()

        def step(ctx=ctx, proj=proj, q=q, out=out):
            kernels.qkv_prepare(proj, Hq * maps, G * maps, dk, G, dv, None, None, 1e-5, None, 0, ctx, pages, 64, kc, vc, q)
            kernels.attention_maps(q, out, kc, vc, ctx, pages, 64, Hq, G, maps, dk, dv, dk ** -0.5, None, window, 0, rt=rt, early=early)
            return out
        steps.append(step)

    def reset():
        kc.copy_(k_full)
        vc.copy_(v_full)
    _check(reset, steps)


@pytest.mark.parametrize("dims,ranks", [((4, 2, 64, 64, 4), (16, 24)), ((3, 3, 160, 96, 3), (8, 8)), ((2, 1, 32, 64, 6), (4, 4))])
@pytest.mark.parametrize("early", [True, False])
def test_channel_states(dims, ranks, early):
    """The row that a step works on is still to be written when it starts; without ``early`` so are the carried inputs and the state,
    which the step before leaves in the same row of launches."""
    from llmi_b200.ops import kernels
    torch.manual_seed(dims[2])
    H, Hk, D, Dv, taps = dims
    S, n_conv = 5, 2 * Hk * D + H * Dv
    at, width = n_conv + H, n_conv + H + sum(ranks)
    full = torch.randn(S, kernels.delta_state_floats(*dims), device="cuda") * 0.1
    state, conv = torch.empty_like(full), torch.randn(n_conv, taps, device="cuda") * 0.5
    a_log, dt_bias, weight = torch.randn(H, device="cuda"), torch.randn(H * D, device="cuda"), torch.ones(Dv, device="cuda")
    w_a, w_g = (torch.randn(r, -(-n // 64) * 64, device="cuda") * r ** -0.5 for r, n in zip(ranks, (H * D, H * Dv)))
    ctx, eye, steps = _token_ctx([3, 9, 64, 700, 5]), torch.eye(width, device="cuda"), []
    eye = torch.nn.functional.pad(eye, (0, -width % 4))
    proj_a = torch.empty(S, width, device="cuda")
    for _ in range(1 if early else 3):
        rows = torch.nn.functional.pad(torch.randn(S, width, device="cuda"), (0, -width % 4))
        proj, gate, out = torch.empty_like(proj_a), torch.empty(S, H * Dv, device="cuda"), torch.empty(S, H * Dv, device="cuda")
        pitch = n_conv + H * D + H
        prep = torch.empty(S, pitch + -pitch % 4, device="cuda")

        def step(rows=rows, proj=proj, gate=gate, out=out, prep=prep):
            kernels.linear_simt(rows, eye, proj)                         # (the rows as they are: the launch ahead)
            kernels.channel_token(proj, dims, (at, ranks[0]), (at + ranks[0], ranks[1]), conv, a_log, dt_bias, w_a, w_g, state, ctx,
                                  prep, gate, weight, 1e-5, out, early=early)
            return out
        steps.append(step)
    projs = [s.__defaults__[1] for s in steps]

    def reset():
        state.copy_(full)
        for p in projs:
            p.fill_(float("nan"))
    _check(reset, steps)


@pytest.mark.parametrize("nh,nkv,hd,window", [(9, 3, 64, 0), (15, 5, 64, 70), (16, 4, 128, 0), (8, 8, 128, 0)])
@pytest.mark.parametrize("early", [True, False])
def test_step_that_appends_its_own_row(nh, nkv, hd, window, early):
    """A decode step whose kernel rotates and appends: its projection is still to be written when it starts; without ``early`` so is
    the row before it."""
    from llmi_b200.engine.runtime import Runtime
    from llmi_b200.ops import kernels
    rt = Runtime(torch.bfloat16, "cuda")
    torch.manual_seed(nh + hd)
    first = POSITIONS[-4:] if nh == nkv else POSITIONS
    S, P = len(first), 13 if nh == nkv else 6
    assert kernels.decode_short_parts(S, nkv, P, hd, nh // nkv, window) > 0
    pages = torch.randperm(S * P, device="cuda").int().view(S, P)
    k_full, v_full = (torch.randn(S * P, nkv, 64, hd, device="cuda").bfloat16() for _ in range(2))
    for s, p in enumerate(first):
        for j in range(p, 64 * P):
            k_full[pages[s, j // 64], :, j % 64] = v_full[pages[s, j // 64], :, j % 64] = float("nan")
    kc, vc, inv = torch.empty_like(k_full), torch.empty_like(v_full), torch.rand(hd // 2, device="cuda")
    steps, projections = [], []
    for positions in [first] if early else [first, [p + 1 for p in first]]:
        ctx, rows = _token_ctx(positions), torch.randn(S, (nh + 2 * nkv) * hd, device="cuda")
        qkv, out = torch.empty(rows.shape, device="cuda").bfloat16(), torch.empty(S, nh * hd, device="cuda").bfloat16()
        projections.append(qkv)

        def step(ctx=ctx, rows=rows, qkv=qkv, out=out):
            kernels.cast_rows(rows, qkv)
            kernels.attention(qkv, out, kc, vc, ctx, pages, 64, nh, nkv, hd, hd ** -0.5, window, rt=rt, rope=(inv, hd, True), early=early)
            return out
        steps.append(step)

    def reset():
        kc.copy_(k_full)
        vc.copy_(v_full)
        for p in projections:
            p.fill_(float("nan"))
    _check(reset, steps)
    kernels.check_device_errors("cuda:0")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,top", [(1, 1), (3, 2)])
def test_experts_chosen_by_the_launch_ahead(dtype, T, top):
    """The down product asks for weights ahead of its wait, by experts that the router has yet to choose when it is launched."""
    from llmi_b200.ops import kernels
    torch.manual_seed(T)
    E, W, F = 16, 512, 256
    h, wg, wu = torch.randn(T, W, device="cuda").to(dtype), *(torch.randn(E, F, W, device="cuda").to(dtype) for _ in range(2))
    wd, ctx = torch.randn(E, W, F, device="cuda").to(dtype), _token_ctx(list(range(T)))
    router, logits = torch.randn(E, W, device="cuda").to(dtype), torch.empty(T, E, device="cuda")
    idx, wt = torch.empty(T, top, dtype=torch.int32, device="cuda"), torch.empty(T, top, device="cuda")
    a, y = torch.empty(T, top, F, device="cuda"), torch.empty(T, W, device="cuda")

    def step():
        kernels.linear_simt(h, router, logits, mode=kernels.OUT_STORE_F32)
        kernels.moe_route(logits, top, ctx, idx, wt)
        kernels.moe_experts_streamed(h, wg, wu, wd, idx, wt, kernels.ACT_SILU, a, y)
        return y

    def reset():                                         # (other experts, whose rows there are)
        logits.copy_(torch.rand(T, E, device="cuda"))
        idx.copy_(torch.randint(0, E, (T, top), device="cuda"))
        wt.fill_(float("nan"))
    _check(reset, [step])
