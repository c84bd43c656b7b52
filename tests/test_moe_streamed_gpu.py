"""Routed experts whose weights are streamed, a handful of tokens: against 64 bits, at the edges of a lane's batch of loads (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("W,F", [(8, 8), (256, 2040), (2048, 264), (2056, 2048), (4100, 24), (20, 4104), (7, 13)])
@pytest.mark.parametrize("top,gated", [(1, True), (3, True), (2, False)])
def test_streamed_experts(dtype, W, F, top, gated):
    """Rows shorter than one load, ending inside a batch of eight, one entry into the next, and rows that 16-byte loads do not
    take; a token of no sequence and a choice that is nobody's; stored and added; the same launches again give the same bits."""
    from llmi_b200.ops import kernels
    T, E = 3, 4
    gen = torch.Generator(device="cuda").manual_seed(W * F + top)

    def rnd(*shape, gain=1.0):
        return (torch.randn(*shape, generator=gen, device="cuda") * gain).to(dtype)
    h, wd = rnd(T, W), rnd(E, W, F, gain=F ** -0.5)
    wg, wu = (rnd(E, F, W, gain=W ** -0.5) if gated else None), rnd(E, F, W, gain=W ** -0.5)
    idx = torch.stack([torch.randperm(E, generator=gen, device="cuda")[:top] for _ in range(T)]).to(torch.int32).contiguous()
    idx[1] = -1
    if top > 1:
        idx[2, top - 1] = -1
    wt = torch.rand(T, top, generator=gen, device="cuda")
    start = torch.randn(T, W, generator=gen, device="cuda")
    act = kernels.ACT_SILU if gated else kernels.EXPERT_ACTIVATIONS["relu2"]
    exact = start.double().clone()
    size = torch.zeros_like(exact)
    for t in range(T):
        for j in range(top):
            e = int(idx[t, j])
            if e < 0:
                continue
            u = wu[e].double() @ h[t].double()
            g = wg[e].double() @ h[t].double() if gated else None
            a = g * torch.sigmoid(g) * u if gated else torch.relu(u) ** 2
            exact[t] += float(wt[t, j]) * (wd[e].double() @ a)
            size[t] += float(wt[t, j]) * (wd[e].double().abs() @ a.abs())
    got = []
    for _ in range(2):
        y, a = start.clone(), torch.empty(T, top, F, device="cuda")
        kernels.moe_experts_streamed(h, wg, wu, wd, idx, wt, act, a, y, add=True)
        got.append(y)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0][1], start[1])
    # products of the inputs are exact in 32 bits or rounded once; sums of W and F terms in 32 bits, each ahead of one more
    bound = (max(W, 32) ** 0.5 + max(F, 32) ** 0.5 + 8) * 2.0 ** -23
    assert float((got[0].double() - exact).abs().max()) <= bound * float((size + exact.abs()).max())
    y, a = torch.full((T, W), float("nan"), device="cuda"), torch.empty(T, top, F, device="cuda")
    kernels.moe_experts_streamed(h, wg, wu, wd, idx, wt, act, a, y)
    assert float((y.double() + start.double() - exact).abs().max()) <= bound * float((size + exact.abs()).max()) and float(y[1].abs().max()) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("W,F", [(64, 64), (256, 128), (2048, 128), (512, 512), (1024, 256), (128, 520)])
def test_forms_agree(dtype, W, F):
    """A token's result bit for bit, whichever product asks for its rows ahead, alone, among six tokens and among eight."""
    from llmi_b200.ops import kernels
    T, E, top = 8, 6, 3
    gen = torch.Generator(device="cuda").manual_seed(W + F)
    h = torch.randn(T, W, generator=gen, device="cuda").to(dtype)
    wg, wu = ((torch.randn(E, F, W, generator=gen, device="cuda") * W ** -0.5).to(dtype) for _ in range(2))
    wd = (torch.randn(E, W, F, generator=gen, device="cuda") * F ** -0.5).to(dtype)
    idx = torch.stack([torch.randperm(E, generator=gen, device="cuda")[:top] for _ in range(T)]).to(torch.int32).contiguous()
    idx[4], idx[5, 1] = -1, -1
    wt = torch.rand(T, top, generator=gen, device="cuda")

    def run(lo, hi):
        y, a = torch.empty(hi - lo, W, device="cuda"), torch.empty(hi - lo, top, F, device="cuda")
        kernels.moe_experts_streamed(h[lo:hi], wg, wu, wd, idx[lo:hi], wt[lo:hi], kernels.ACT_SILU, a, y)
        return y
    want = run(0, T)
    assert torch.equal(run(0, 6), want[:6]) and all(torch.equal(run(t, t + 1), want[t:t + 1]) for t in range(T))
    rule = kernels.moe_streamed_ahead
    try:
        for form in range(4):
            kernels.moe_streamed_ahead = lambda *sizes, form=form: form
            assert torch.equal(run(0, T), want)
    finally:
        kernels.moe_streamed_ahead = rule


@pytest.mark.parametrize("dtype,T,W,F,top", [(torch.float32, 256, 256, 128, 4), (torch.float32, 128, 64, 64, 2), (torch.float32, 128, 1024, 512, 2),
                                             (torch.bfloat16, 3, 64, 64, 4)])
def test_many_tokens_and_short_rows_are_no_slower_than_one_load_behind_the_other(dtype, T, W, F, top):
    """(They took 1.1 to 2 times as long with their rows asked for ahead.)"""
    from llmi_b200.ops import kernels
    E = 16
    h, wd = torch.randn(T, W, device="cuda").to(dtype), torch.randn(E, W, F, device="cuda").to(dtype)
    wg, wu = (torch.randn(E, F, W, device="cuda").to(dtype) for _ in range(2))
    idx = torch.stack([torch.randperm(E, device="cuda")[:top] for _ in range(T)]).to(torch.int32).contiguous()
    wt, a, y = torch.rand(T, top, device="cuda"), torch.empty(T, top, F, device="cuda"), torch.empty(T, W, device="cuda")

    def us():
        side, graph, times = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
        run = lambda: kernels.moe_experts_streamed(h, wg, wu, wd, idx, wt, kernels.ACT_SILU, a, y)      # noqa: E731
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
            times.append(start.elapsed_time(end))
        return min(times)
    rule = kernels.moe_streamed_ahead
    mine = us()
    try:
        kernels.moe_streamed_ahead = lambda *sizes: 0
        plain = us()
    finally:
        kernels.moe_streamed_ahead = rule
    assert mine < 1.08 * plain
