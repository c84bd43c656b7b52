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
