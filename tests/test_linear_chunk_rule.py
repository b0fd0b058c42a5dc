"""The rule by which linear attention with gated decays is walked in chunks or token by token, against what both were
measured to take (B200, us of the whole call in a graph: launched one by one, the short ones are as long as the host's work; bfloat16)."""

from types import SimpleNamespace

import pytest

from thing_htn_2026_b200 import ops

# heads, (tokens, single tokens beside them, prompts): token by token, in chunks
MEASURED = [(16, (16, 0, 1), 6, 13), (16, (64, 0, 1), 12, 17), (16, (128, 0, 1), 19, 24), (16, (300, 0, 1), 40, 38), (16, (2048, 0, 1), 255, 125),
            (16, (16, 60, 1), 41, 75), (16, (512, 60, 1), 93, 111), (16, (2048, 60, 1), 327, 235), (16, (512, 0, 2), 92, 54),
            (16, (512, 0, 8), 354, 172), (16, (16, 0, 8), 18, 25), (16, (33, 0, 64), 213, 161), (16, (16, 0, 64), 122, 97), (32, (16, 0, 1), 7, 16),
            (32, (64, 0, 1), 15, 23), (32, (128, 0, 1), 26, 33), (32, (300, 0, 1), 55, 44), (32, (2048, 0, 1), 358, 184), (32, (16, 60, 1), 97, 146),
            (32, (512, 60, 1), 174, 183), (32, (2048, 60, 1), 409, 400), (32, (512, 0, 8), 639, 337), (32, (16, 0, 8), 30, 36),
            (32, (16, 0, 64), 238, 176), (64, (33, 0, 1), 17, 32), (64, (64, 0, 1), 27, 32), (64, (300, 0, 1), 106, 56), (64, (512, 60, 1), 337, 356),
            (64, (2048, 60, 1), 793, 805), (64, (128, 0, 32), 1296, 672)]


@pytest.mark.parametrize("heads,what,by_token,in_chunks", MEASURED)
def test_the_faster_way_is_taken(heads, what, by_token, in_chunks):
    tokens, singles, prompts = what
    rows = SimpleNamespace(max_q_len=tokens, n_rows=tokens * prompts + singles, n_seqs=prompts + singles)
    taken = in_chunks if ops._LINEAR_COST.chunks_pay(rows, heads, 128) else by_token
    assert taken <= 1.06 * min(by_token, in_chunks)


def test_long_prompts_alone_are_walked_in_chunks():
    for tokens in (400, 2048, 20000):
        for prompts in (1, 2, 8):
            for heads in (8, 32, 128):
                rows = SimpleNamespace(max_q_len=tokens, n_rows=tokens * prompts, n_seqs=prompts)
                assert ops._LINEAR_COST.chunks_pay(rows, heads, 128), (tokens, prompts, heads)
