"""The kernels between a projection and attention or a recurrence, four entries a thread: against 64 bits and the general forms (GPU)."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ctx(seqs, positions):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")      # noqa: E731
    return types.SimpleNamespace(tok_seq=i32(seqs), tok_pos=i32(positions))


@pytest.mark.parametrize("H,D,Dv", [(3, 32, 32), (2, 64, 64), (17, 64, 128), (5, 128, 64), (2, 48, 48), (2, 64, 6)])
@pytest.mark.parametrize("R", [1, 7, 16, 130])
@pytest.mark.parametrize("walk", [True, False])
def test_general_delta_vectors(H, D, Dv, R, walk):
    """W2's rows walked and their product given; a row of no sequence; sizes and pitches that four entries a thread do not take."""
    from llmi_b200.ops import kernels
    torch.manual_seed(H * D + R)
    T, N = 3, H * D
    for extra in (0, 4, 3):
        width = 3 * N + 2 * H * Dv + R
        proj = torch.randn(T, width + extra + (-width) % 4, device="cuda")
        w2t, w0, ab = torch.randn(R, N, device="cuda") * R ** -0.5, torch.randn(N, device="cuda"), torch.randn(N, device="cuda")
        low = torch.tanh(proj[:, 3 * N + 2 * H * Dv:width].double())
        z = low @ w2t.double()
        prep = torch.full((T, 3 * N + 4), 7.0, device="cuda")
        kernels.gdelta_prepare(proj, H, D, Dv, w2t, w0, ab, _ctx([0, -1, 1], [5, 0, 9]), prep, None if walk else z.float())
        k = proj[:, N:2 * N].double().view(T, H, D)
        u = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).reshape(T, N)
        at = 2 * N + H * Dv
        want = torch.cat([torch.exp(-0.6065306597126334 * torch.sigmoid(w0.double() + z)), u,
                          -torch.sigmoid(proj[:, at:at + N].double() + ab.double()) * u], dim=1)
        assert (prep[1] == 7.0).all() and (prep[:, 3 * N:] == 7.0).all()
        # sums of R and D products in 32 bits, then a handful of roundings; every entry is at most 1
        assert float((prep[[0, 2], :3 * N].double() - want[[0, 2]]).abs().max()) < (R ** 0.5 + D ** 0.5 + 8) * 2.0 ** -23


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nk,dk,nv,dv", [(32, 8, 64, 8, 64), (64, 2, 64, 2, 64), (65, 2, 64, 2, 64), (3, 1, 4, 2, 12), (3, 1, 6, 1, 6), (6, 2, 100, 2, 100)])
@pytest.mark.parametrize("v_from_k", [False, True])
def test_norms_over_whole_parts(dtype, nq, nk, dk, nv, dv, v_from_k):
    """Parts up to the registers' size, one head beyond it, and sizes that whole fours do not divide; one norm, the other, both;
    keys and values not kept; rows of no sequence."""
    from llmi_b200.ops import kernels
    if v_from_k and (nv, dv) != (nk, dk):
        nv, dv = nk, dk
    torch.manual_seed(nq + dk)
    T, page, eps = 4, 64, 1e-5
    n_v = 0 if v_from_k else nv * dv
    proj = torch.randn(T, nq * dk + nk * dk + n_v, device="cuda")
    wq, wk = 1 + 0.2 * torch.randn(nq * dk, device="cuda"), 1 + 0.2 * torch.randn(nk * dk, device="cuda")
    seqs, at, pages = [0, 1, -1, 1], [3, 70, 0, 71], torch.tensor([[4, 0], [2, 5]], dtype=torch.int32, device="cuda")
    ctx = _ctx(seqs, at)
    for uq, uk, write in ((wq, wk, True), (wq, None, True), (None, wk, True), (wq, wk, False)):
        kc = torch.full((6, nk, page, dk), 7.0, dtype=dtype, device="cuda")
        vc = torch.full((6, nv, page, dv), 7.0, dtype=dtype, device="cuda")
        kw, vw, out = kc.double(), vc.double(), torch.full((T, nq * dk), float("nan"), dtype=dtype, device="cuda")
        kernels.qkv_prepare(proj, nq, nk, dk, nv, dv, uq, uk, eps, None, 0, ctx, pages, page, kc, vc, out, write_kv=write, v_from_k=v_from_k)
        x = proj.double()
        q, k, v = x[:, :nq * dk], x[:, nq * dk:nq * dk + nk * dk], x[:, nq * dk + nk * dk:]
        norm = lambda y, w: y if w is None else y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * w.double()      # noqa: E731
        q, k = norm(q, uq), norm(k, uk)
        v = k if v_from_k else v
        q[2] = 0
        if write:
            for t in (0, 1, 3):
                pg = int(pages[seqs[t], at[t] // page])
                kw[pg, :, at[t] % page], vw[pg, :, at[t] % page] = k[t].view(nk, dk), v[t].view(nv, dv)
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20      # of an entry's own size: the type's rounding, a sum's
        for got, want in ((out, q), (kc, kw), (vc, vw)):
            assert bool(((got.double() - want).abs() <= tol * want.abs()).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norms_without_an_epsilon(dtype):
    """eps 0: a row of no sequence has no length to divide by and is zeros all the same; the others are normed."""
    from llmi_b200.ops import kernels
    torch.manual_seed(2)
    T, nq, nk, d = 3, 4, 2, 64
    proj, wq, wk = torch.randn(T, (nq + 2 * nk) * d, device="cuda"), torch.ones(nq * d, device="cuda"), torch.ones(nk * d, device="cuda")
    kc, vc = (torch.zeros(2, nk, 64, d, dtype=dtype, device="cuda") for _ in range(2))
    out, pages = torch.full((T, nq * d), 7.0, dtype=dtype, device="cuda"), torch.tensor([[0], [1]], dtype=torch.int32, device="cuda")
    kernels.qkv_prepare(proj, nq, nk, d, nk, d, wq, wk, 0.0, None, 0, _ctx([0, -1, 1], [3, 0, 5]), pages, 64, kc, vc, out)
    q = proj[:, :nq * d].double()
    want = q / torch.sqrt((q * q).mean(-1, keepdim=True))
    want[1] = 0
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20         # the type's rounding, a sum's
    assert bool(((out.double() - want).abs() <= tol * want.abs()).all())


def _us(run):
    side, graph, times = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
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


@pytest.mark.parametrize("T,H,D,R", [(16, 64, 64, 16), (4, 64, 64, 8), (16, 64, 32, 32), (16, 16, 128, 4)])
def test_short_walks_are_no_slower_than_in_the_general_form(T, H, D, R):
    """Rows that whole fours do not divide take the general form (it took 0.6 to 0.9 times as long)."""
    from llmi_b200.ops import kernels
    N = H * D
    w2t, w0, ab, prep = torch.randn(R, N, device="cuda"), torch.randn(N, device="cuda"), torch.randn(N, device="cuda"), torch.empty(T, 3 * N, device="cuda")
    ctx = _ctx(list(range(T)), list(range(T)))

    def call(pitch):
        proj = torch.randn(T, pitch, device="cuda")
        return _us(lambda: kernels.gdelta_prepare(proj, H, D, D, w2t, w0, ab, ctx, prep))
    assert call(5 * N + R) < 1.08 * call(5 * N + R + 1)


@pytest.mark.parametrize("T,nq,nk,dk", [(3000, 4, 2, 32), (4000, 8, 2, 64), (2000, 2, 1, 64), (600, 8, 1, 16), (3000, 2, 1, 8)])
def test_norms_of_small_parts_are_no_slower_than_in_the_general_form(T, nq, nk, dk):
    """Rows that whole fours do not divide take the general form (many tokens took 0.4 to 0.9 times as long)."""
    from llmi_b200.ops import kernels
    wq, wk = torch.ones(nq * dk, device="cuda"), torch.ones(nk * dk, device="cuda")
    kc, vc = (torch.zeros(T // 64 + 1, nk, 64, dk, device="cuda").bfloat16() for _ in range(2))
    out, pages = torch.empty(T, nq * dk, device="cuda").bfloat16(), torch.arange(T // 64 + 1, device="cuda").int().view(1, -1)
    ctx = _ctx([0] * T, list(range(T)))

    def call(pitch):
        proj = torch.randn(T, pitch, device="cuda")
        return _us(lambda: kernels.qkv_prepare(proj, nq, nk, dk, nk, dk, wq, wk, 1e-5, None, 0, ctx, pages, 64, kc, vc, out))
    assert call((nq + 2 * nk) * dk) < 1.08 * call((nq + 2 * nk) * dk + 1)


@pytest.mark.parametrize("heads,dim", [(24, 64), (32, 64), (33, 64), (64, 64), (20, 128)])
def test_norms_are_as_near_to_64_bits_as_in_the_general_form(heads, dim):
    """fp32, 3,000 rows: whole fours (the part in registers) against a pitch that they do not divide (the general form)."""
    from llmi_b200.ops import kernels
    torch.manual_seed(heads)
    T, N = 3000, heads * dim
    wq, wk = 1 + 0.2 * torch.randn(N, device="cuda"), torch.ones(dim, device="cuda")
    x = torch.randn(T, N + 2 * dim, device="cuda")
    kc, vc = (torch.zeros(T // 64 + 1, 1, 64, dim, device="cuda") for _ in range(2))
    ctx, pages = _ctx([0] * T, list(range(T))), torch.arange(T // 64 + 1, device="cuda").int().view(1, -1)
    q = x[:, :N].double()
    want = q / torch.sqrt((q * q).mean(-1, keepdim=True) + 1e-5) * wq.double()

    def error(pad):
        out = torch.empty(T, N, device="cuda")
        kernels.qkv_prepare(torch.nn.functional.pad(x, (0, pad)), heads, 1, dim, 1, dim, wq, wk, 1e-5, None, 0, ctx, pages, 64, kc, vc, out)
        return float((out.double() - want).norm() / want.norm())
    # (two sums' roundings over 3,000 rows: their means differ by no more than a hundredth where neither is the better one)
    assert error(0) <= 1.01 * error(1)
