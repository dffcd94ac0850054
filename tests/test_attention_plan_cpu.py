"""How the attention launches divide their work: host rules, checked without a GPU."""
from odc_b200 import _ext

SMS = 148


def _plan(tokens, seqs, longest, n_q, n_kv, d=128, causal=True):
    return _ext.load().attn_plan(tokens, seqs, longest, n_q, n_kv, d, causal, SMS)


def test_few_tiles_are_taken_one_at_a_time():
    assert _plan(1000, 1, 1000, 12, 2) == (False, 6)
    assert _plan(8000, 1, 8000, 1, 1) == (False, 1)
    assert _plan(32768, 1, 32768, 40, 8) == (True, 1)
    assert _plan(16384, 20, 4000, 32, 8) == (True, 1)
    assert _plan(1000, 1, 1000, 12, 2, d=64)[0] is False       # one tile per CTA in any case

