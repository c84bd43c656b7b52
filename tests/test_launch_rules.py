"""The rules by which a step's launches are chosen from its sizes, on the CPU."""
import types

import pytest

from llmi_b200.ops import kernels as K


@pytest.fixture(autouse=True)
def sms(monkeypatch):
    monkeypatch.setattr(K, "sm_count", lambda: 148)


@pytest.mark.parametrize("kv,group,hd", [(32, 1, 64), (3, 3, 64), (8, 4, 128), (16, 1, 128), (8, 2, 64), (4, 8, 64)])
@pytest.mark.parametrize("window", [1, 64, 128, 512, 2048])
def test_a_window_is_planned_by_what_it_spans(kv, group, hd, window):
    """However long the history, the plan is that of the pages that the window's positions lie on."""
    for n_seqs in (1, 8, 32, 64):
        span = (window - 1 + 63) // 64 + 1
        one = -(-window // 64) + 1
        assert span <= one <= span + 1
        for pages in (one, one + 1, 126, 500):
            if pages < one:
                continue
            assert K.decode_short_parts(n_seqs, kv, pages, hd, group, window) == K.decode_short_parts(n_seqs, kv, one, hd, group)
            ctx = types.SimpleNamespace(decode=True, n_real_seqs=n_seqs)
            if K.decode_short_parts(n_seqs, kv, one, hd, group):
                K._plan_cache[(n_seqs, pages, kv, hd, group)] = (pages, 0)          # (what the other kernel would do needs the library)
                assert K.decode_plan_token(ctx, n_seqs, pages, 64, kv, hd, group, window) == ("short", K.decode_short_parts(n_seqs, kv, one, hd, group))
        for max_q in (4, 16, 64):
            seen = -(-(window + max_q - 1) // 64) + 1
            assert K.attention_short_parts(n_seqs, kv, max_q, group, 500, hd, window) == K.attention_short_parts(n_seqs, kv, max_q, group, seen, hd)
    K._plan_cache.clear()


def test_ungrouped_decode_steps():
    """Heads of 64 stay with the kernel that has 32-bit weights and is the faster one; of 128 the clusters begin where they win."""
    assert not any(K.decode_short_parts(s, h, p, 64, 1) for s in (1, 8, 24, 28, 64, 96) for h in (3, 12, 32) for p in (1, 4, 12, 35, 125))
    assert [K.decode_short_parts(1, 16, p, 128, 1) for p in (4, 8, 16, 17, 32, 47, 48, 63)] == [0, 0, 4, 0, 0, 0, 8, 8]
    assert [K.decode_short_parts(1, 32, p, 128, 1) for p in (16, 32, 63)] == [4, 8, 8]
    assert [K.decode_short_parts(1, 8, p, 128, 4) for p in (1, 4, 5, 8, 16)] == [1, 1, 2, 2, 4]
