"""The rule by which linear attention with gated decays is walked in chunks or token by token, against what both were
measured to take (B200, us of the whole call, bfloat16)."""

from types import SimpleNamespace

import pytest

from thing_htn_2026_b200 import ops

# heads, (tokens, single tokens beside them, prompts): token by token, in chunks
MEASURED = [(16, (16, 0, 1), 13, 24), (16, (64, 0, 1), 20, 26), (16, (128, 0, 1), 28, 30), (16, (300, 0, 1), 50, 42), (16, (2048, 0, 1), 263, 155),
            (16, (16, 60, 1), 58, 111), (16, (512, 60, 1), 103, 155), (16, (2048, 60, 1), 335, 259), (16, (512, 0, 2), 101, 65), (16, (512, 0, 8), 364, 185),
            (16, (16, 0, 8), 28, 32), (16, (33, 0, 64), 222, 173), (16, (16, 0, 64), 130, 103), (32, (16, 0, 1), 15, 24), (32, (64, 0, 1), 24, 28),
            (32, (128, 0, 1), 36, 32), (32, (300, 0, 1), 65, 50), (32, (2048, 0, 1), 368, 222), (32, (16, 60, 1), 103, 155), (32, (512, 60, 1), 181, 241),
            (32, (2048, 60, 1), 419, 439), (32, (512, 0, 8), 650, 362), (32, (16, 0, 8), 42, 40), (32, (16, 0, 64), 247, 183), (64, (33, 0, 1), 26, 32),
            (64, (64, 0, 1), 36, 32), (64, (300, 0, 1), 118, 69), (64, (512, 60, 1), 347, 368), (64, (2048, 60, 1), 802, 765), (64, (128, 0, 32), 1308, 679)]


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
