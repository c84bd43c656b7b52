"""The sampler's two ways to the kept set at their edges (GPU)."""
import numpy as np
import pytest
import torch

import plain_llama as P

pytestmark = pytest.mark.gpu


def K():
    from llmi_b200.ops import kernels
    return kernels


@pytest.mark.parametrize("V", [1, 7, 1024, 4099, 49152, 430003])
@pytest.mark.parametrize("top_k,top_p", [(50, 0.95), (1, 0.5), (512, 0.9), (513, 0.9), (40, 1.0), (0, 0.9)])
def test_sample_both_ways(V, top_k, top_p):
    """Few candidates and the general way, rows in shared memory and in scratch, values with and without many ties (a tie at
    the bound of more values than the candidates' list holds): the plain sampler's id."""
    k = K()
    torch.manual_seed(V + top_k)
    logits = torch.randn(6, V + 1, device="cuda")[:, :V] * 2.5
    logits[2] = (logits[2] * 2).round() / 2
    logits[3] = logits[3].clamp(max=1.0)
    logits[4] = -float("inf")
    logits[4, V // 2] = 0.0
    u = torch.tensor([0.0001, 0.3, 0.6, 0.95, 0.5, 0.999], dtype=torch.float64, device="cuda")
    out = torch.empty(6, dtype=torch.int32, device="cuda")
    k.sample(logits, 0.8, top_k, top_p, u, torch.empty(6, V, device="cuda"), out)
    for i in range(6):
        row = logits[i].cpu().numpy()
        prob = P.sampling_probabilities(row, 0.8, top_k, top_p)
        cum = np.cumsum(prob.astype(np.float64))
        got = int(out[i])
        assert prob[got] > 0
        # the draw's own interval holds the number, up to the rounding of the 32-bit probabilities
        slack = 1e-6 + 2e-7 * V ** 0.5
        assert cum[got] - prob[got] - slack <= float(u[i]) <= cum[got] + slack, (i, got)


@pytest.mark.parametrize("above", [1, 2, 10, 49, 50, 51, 400, 3000])
@pytest.mark.parametrize("top_p", [0.9, 1.0])
def test_sample_peaked_rows(above, top_p):
    """Rows with so many probabilities above 0, fewer and more than top_k, spread over the vocabulary or side by side: the plain
    sampler's id."""
    k = K()
    V, top_k = 49152, 50
    torch.manual_seed(above)
    logits = torch.full((4, V), -1e4, device="cuda")
    logits[0, torch.randperm(V)[:above].cuda()] = torch.randn(above, device="cuda")
    logits[1, :above] = torch.randn(above, device="cuda")
    logits[2, V - above:] = torch.randn(above, device="cuda")
    logits[3, torch.randperm(V)[:above].cuda()] = 1.0
    u = torch.tensor([0.3, 0.9999, 0.0001, 0.7], dtype=torch.float64, device="cuda")
    out = torch.empty(4, dtype=torch.int32, device="cuda")
    k.sample(logits, 1.0, top_k, top_p, u, torch.empty(4, V, device="cuda"), out)
    for i in range(4):
        prob = P.sampling_probabilities(logits[i].cpu().numpy(), 1.0, top_k, top_p)
        cum = np.cumsum(prob.astype(np.float64))
        got = int(out[i])
        assert prob[got] > 0
        assert cum[got] - prob[got] - 1e-6 <= float(u[i]) <= cum[got] + 1e-6, (i, got)      # (see test_sample_both_ways)


def test_sample_peaked_rows_are_no_slower():
    """A low temperature leaves a few dozen probabilities above 0: such rows take the way of ordinary ones, in about its time (the
    way past a full list took five times as long)."""
    k = K()
    n, V = 64, 49152
    torch.manual_seed(0)
    logits, u = torch.randn(n, V, device="cuda") * 2.5, torch.rand(n, dtype=torch.float64, device="cuda")
    probs, out = torch.empty(n, V, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")

    def us(temperature):
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                k.sample(logits, temperature, 50, 0.95, u, probs, out)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 100)
        return sorted(times)[3]
    us(0.8)
    assert us(0.01) < 2 * us(0.8)
