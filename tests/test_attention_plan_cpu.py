"""How the attention launches divide their work: host rules, checked without a GPU."""
import pytest

from odc_b200 import _ext

SMS = 148


def _plan(tokens, seqs, longest, n_q, n_kv, d=128, causal=True):
    return _ext.load().attn_plan(tokens, seqs, longest, n_q, n_kv, d, causal, SMS)


@pytest.mark.parametrize("d", [64, 128])
def test_parts_divide_the_group_and_keep_the_scratch_small(d):
    for n_kv, rep in ((1, 1), (1, 7), (2, 6), (8, 4), (8, 5), (4, 16)):
        for tokens in (0, 1, 127, 128, 1000, 20000, 200000):
            for seqs in (1, 2, 40, 1000):
                for longest in (0, 1, 128, 5000, 10 ** 9):   # the caller's word, right or wrong
                    for causal in (True, False):
                        parts = _plan(tokens, seqs, longest, n_kv * rep, n_kv, d, causal)[1]
                        assert parts >= 1 and rep % parts == 0
                        if parts > 1:   # fp32 partial dK and dV: up to a few hundred MB
                            assert parts * 2 * tokens * n_kv * d * 4 < 1 << 30


def test_few_tiles_are_taken_one_at_a_time_and_divided():
    assert _plan(1000, 1, 1000, 12, 2) == (False, 6)
    assert _plan(8000, 1, 8000, 1, 1) == (False, 1)
    assert _plan(32768, 1, 32768, 40, 8) == (True, 1)
    assert _plan(16384, 20, 4000, 32, 8) == (True, 1)
    assert _plan(1000, 1, 1000, 12, 2, d=64)[0] is False       # one tile per CTA in any case


def test_short_sequences_are_not_divided_for_nothing():
    assert _plan(6000, 300, 20, 14, 2)[1] == 1
    assert _plan(6000, 300, 20, 14, 2, d=64)[1] == 1
    assert _plan(12000, 40, 300, 5, 1)[1] == 1
