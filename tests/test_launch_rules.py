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


@pytest.mark.parametrize("layout,n_seqs,held,max_q,parts", [
    # (the prompt kernel against this one in the best number of blocks, us)
    ((1, 8, 64), 16, 250, 48, (0,)),           # 7.6 against 8.7
    ((8, 8, 64), 4, 1500, 64, (0,)),           # 29.9 against 41.3
    ((3, 3, 64), 16, 250, 32, (0,)),           # 7.9 against 8.7
    ((2, 16, 64), 8, 500, 64, (0,)),           # 14.1 against 17.7
    ((32, 1, 64), 8, 500, 64, (0,)),           # 15.6 against 19.3
    ((3, 3, 64), 4, 1500, 16, (8,)),           # 22.0 against 8.8
    ((3, 3, 64), 64, 150, 16, (1,)),           # 35.9 against 8.0
    ((32, 1, 64), 64, 500, 16, (1,)),          # 138 against 55
    ((8, 4, 128), 16, 2000, 8, (1, 2)),        # 115 against 31 and 29
])
def test_messages_go_where_they_are_faster(layout, n_seqs, held, max_q, parts):
    kv, group, hd = layout
    assert K.attention_short_parts(n_seqs, kv, max_q, group, (held + max_q + 63) // 64, hd) in parts


def test_a_cut_prompt_is_weighed_as_one():
    """A step whose lengths are known lets the prompt kernel cut its key ranges: 8 x 8 x 64, one sequence of 4,000, 64 tokens, 24.9 us
    cut and 54.5 whole against 31.7 here."""
    assert K.attention_short_parts(1, 8, 64, 8, 64, 64) == 4 and K.attention_short_parts(1, 8, 64, 8, 64, 64, cut=True) == 0


def test_prompts_of_a_few_tokens_in_32_bits():
    """Token by token where blocks of 32 queries would be all but empty, by blocks otherwise; decode steps always by token."""
    import torch

    def by_token(q_lens, pages, kv, group, window=0, decode=False):
        ctx = types.SimpleNamespace(decode=decode, host_q_lens=q_lens)
        return K.f32_by_token(ctx, sum(q_lens), torch.zeros(len(q_lens), pages), kv * group, kv, window)
    assert by_token([1] * 8, 1, 4, 1, decode=True)
    assert by_token([2] * 64, 24, 8, 4) and by_token([2] * 64, 24, 32, 1, 100) and by_token([4] * 64, 24, 1, 16, 100)
    assert not by_token([4] * 64, 24, 32, 1, 100) and not by_token([4] * 64, 24, 8, 4) and not by_token([30] * 8, 24, 1, 16, 100)
    assert not by_token([300], 6, 3, 3) and not by_token([2], 1, 8, 4) and not by_token([2] * 40000, 2, 1, 1)
