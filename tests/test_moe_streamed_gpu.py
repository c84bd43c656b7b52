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
