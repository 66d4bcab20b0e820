"""The rule that sends a prefill to tcgen05 or to mma.sync: steps at whose sizes both kernels were timed go to the faster
one, and the choice is the same for the record of a pass as for the pass."""
from types import SimpleNamespace

import pytest

from llm_b200 import ops
from llm_b200.ops import prefill


def diff(dim, vdim, heads, seqs, new, behind, window=0, keep=0):
    return prefill.on_tcgen05(("diff", dim, vdim), heads, seqs * new, seqs, new, behind + new, window, keep)


def window(dim, heads, size, seqs, new, behind):
    return prefill.on_tcgen05(("window", dim), heads, seqs * new, seqs, new, behind + new, size)


def sigmoid(dim, heads, groups, size, seqs, new, behind):
    return prefill.sigmoid_on_tcgen05(heads, groups, dim, seqs * new, seqs, new, behind + new, size)


@pytest.mark.parametrize("choice,mma,tcgen05", [
    # (microseconds of both kernels on a B200, more than a tenth apart)
    (lambda: diff(64, 128, 32, 1, 3001, 0), 438.6, 221.0), (lambda: diff(64, 128, 32, 8, 16, 0), 9.3, 17.8),
    (lambda: diff(64, 128, 32, 1, 2, 8000), 319.4, 142.0), (lambda: diff(64, 128, 32, 8, 2, 2000, 1024, 4), 56.4, 77.9),
    (lambda: diff(64, 128, 32, 1, 100, 0), 10.6, 12.5), (lambda: diff(32, 64, 16, 1, 200, 0), 9.8, 13.9),
    (lambda: diff(32, 64, 16, 32, 2, 500), 33.0, 62.4), (lambda: diff(32, 64, 16, 8, 128, 2000), 73.7, 50.7),
    (lambda: diff(64, 64, 16, 8, 300, 0), 33.4, 38.6), (lambda: diff(128, 128, 16, 1, 512, 0), 44.0, 21.9),
    (lambda: window(64, 32, 1024, 1, 65, 0), 4.7, 5.8), (lambda: window(64, 64, 128, 32, 2, 500), 28.8, 49.6),
    (lambda: window(64, 64, 128, 1, 3001, 0), 53.9, 44.7), (lambda: window(128, 32, 2048, 1, 3001, 0), 252.0, 90.8),
    (lambda: window(128, 32, 2048, 8, 64, 0), 7.8, 6.8), (lambda: sigmoid(64, 4, 1, 0, 1, 100, 0), 10.7, 15.6),
    (lambda: sigmoid(128, 32, 8, 2048, 1, 2500, 0), 2147, 325), (lambda: sigmoid(128, 16, 2, 300, 32, 2, 500), 55.2, 81.6),
    (lambda: sigmoid(64, 4, 1, 0, 1, 128, 8000), 330.3, 285.8)])
def test_the_faster_kernel_is_chosen(choice, mma, tcgen05):
    assert choice() == (tcgen05 < mma)


def test_a_record_of_a_pass_is_not_run_where_the_other_kernel_would_be():
    spec = SimpleNamespace(n_heads=32, n_kv_heads=8, head_dim=64, value_dim=128, window=0, keep_first=0, talk=True)
    short, far = (SimpleNamespace(decode=False, new_counts=[20], n_tokens=20, n_seqs=1, max_len=length) for length in (20, 8000))
    assert ops.diff_attention_replay_key(short, spec) != ops.diff_attention_replay_key(far, spec)
    narrow = SimpleNamespace(n_heads=4, n_kv_heads=1, head_dim=64, value_dim=64, window=0, talk=True)
    assert ops.sigmoid_attention_replay_key(short, narrow) != ops.sigmoid_attention_replay_key(far, narrow)
    assert ops.attention_replay_key(short, 32, 8, 2048) != ops.attention_replay_key(far, 32, 8, 2048)
    assert ops.attention_replay_key(short, 32, 8) == ops.attention_replay_key(far, 32, 8)
