"""Which of two prefill kernels serves a step: the one on tcgen05 or the one on mma.sync.

The kernels on mma.sync take tiles of 64 queries, two or three blocks an SM; those on tcgen05 take
tiles of 128, one or two blocks an SM, pay more for their start (tensor memory, tensor maps) and
less for every page of keys. So tcgen05 wins on long walks and full tiles, mma.sync on short steps
and on many sequences that bring few tokens each. The rule compares two estimates: the turns that
the blocks take on the GPU's SMs, times (start + pages of the longest walk x cost of a page). The
numbers are fitted to both kernels' times at 36 steps (1 to 32 sequences, 2 to 3,001 new tokens
behind 0 to 8,000) of 16 combinations of heads, sizes and windows: the worst of the 576 choices
takes 13 % longer than the better kernel (0.9 us), all others at most 6 %. With tcgen05 at every
step, up to 1.9 times as long as mma.sync (8 sequences of 16 tokens, 32 heads of 2 x 64: 17.8 us for
9.3); with mma.sync at every step, up to 7.6 times as long as tcgen05 (8 sequences of 128 tokens
behind 2,000, 32 mixed heads of 128 over 8: 1,583 us for 210). Since then the tcgen05 kernels' loops are
issued by whole warps and long walks on them take 5 to 7 % less; the numbers are still those of the 36 steps,
so that a step near the line may be on mma.sync by that much.
"""
from __future__ import annotations

from functools import lru_cache

from .. import native

PAGE = native.plan_constant("page")
SMS = 148

# (blocks an SM, start, a page) on mma.sync, and the same on tcgen05; differential attention by the sizes of
# a map and a value, windowed attention by the head size
_COSTS = {
    ("diff", 32, 64): ((2, 1.8, 2.43), (1, 11.6, 1.08)),
    ("diff", 64, 64): ((2, 3.2, 2.19), (1, 8.1, 1.22)),
    ("diff", 64, 128): ((3, 4.4, 5.2), (1, 11.2, 2.1)),
    ("diff", 128, 128): ((2, 4.0, 3.4), (1, 4.8, 1.05)),
    ("window", 64): ((3, 5.7, 2.42), (2, 10.7, 1.21)),
    ("window", 128): ((2, 3.0, 2.4), (2, 4.0, 1.08)),
}
_MARGIN = 0.95           # tcgen05 only where its estimate is below this share of the other


def _turns(n_heads: int, n_tokens: int, n_seqs: int, max_new: int, tile: int, an_sm: int) -> int:
    """How often the SMs take a block, for the tiles of a step of unequal sequences."""
    tiles = min(n_seqs * -(-max_new // tile), n_tokens // tile + n_seqs)
    return -(-n_heads * tiles // (SMS * an_sm))


def _pages(max_new: int, max_len: int, window: int, keep_first: int, tile: int) -> int:
    """Pages that the longest walk of a tile of queries passes."""
    keys = max(max_len, max_new)
    if window > 0:
        seen, kept = window + min(tile, max_new) - 1, -(-keep_first // PAGE)
        if seen + kept * PAGE < keys:
            return -(-seen // PAGE) + 1 + kept
    return -(-keys // PAGE)


@lru_cache(maxsize=4096)
def on_tcgen05(kind: tuple, n_heads: int, n_tokens: int, n_seqs: int, max_new: int, max_len: int, window: int = 0,
               keep_first: int = 0) -> bool:
    """Whether a step of n_tokens new tokens, at most max_new of one of its n_seqs sequences, none longer than max_len
    behind the step, runs on tcgen05. `kind`: a row of _COSTS."""
    narrow, wide = _COSTS[kind]
    pages = [_pages(max_new, max_len, window, keep_first, tile) for tile in (64, 128)]
    if kind == ("window", 128) and pages[0] == 1 and max_new <= 32:
        return False                                       # (5.0 us for 4.6 to 4.9; from 33 tokens on it is ahead)
    mma = _turns(n_heads, n_tokens, n_seqs, max_new, 64, narrow[0]) * (narrow[1] + narrow[2] * pages[0])
    tc = _turns(n_heads, n_tokens, n_seqs, max_new, 128, wide[0]) * (wide[1] + wide[2] * pages[1])
    return tc < _MARGIN * mma


@lru_cache(maxsize=4096)
def sigmoid_on_tcgen05(n_heads: int, n_kv_heads: int, dim: int, n_tokens: int, n_seqs: int, max_new: int, max_len: int,
                       window: int) -> bool:
    """The same for the sigmoid attention with mixed heads, whose scores are a contraction over all key heads: on mma.sync a
    tile forms its mixed queries (a cost by its queries and the contraction's length) and pays for a page by that length."""
    length = n_kv_heads * dim / 64
    pages = [_pages(max_new, max_len, window, 0, tile) for tile in (64, 128)]
    mma = _turns(n_heads, n_tokens, n_seqs, max_new, 64, 2) * (
        5.7 + length * (1.37 + 1.98 * min(max_new, 64) / 64) + (pages[0] - 1) * (2.35 + 0.55 * length))
    tc = _turns(n_heads, n_tokens, n_seqs, max_new, 128, 1) * (9.91 + 0.28 * length + 2.15 * pages[1])
    return tc < _MARGIN * mma
