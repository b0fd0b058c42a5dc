"""The rules by which a step's recurrence is walked in chunks or token by token, against what both were
measured to take (B200, us of the whole call, bfloat16)."""

from types import SimpleNamespace

import pytest

from thing_htn_2026_b200 import ops

# (tokens, single tokens beside them or None, sequences): token by token, in chunks
DELTA = [((16, 0, 1), 65, 52), ((16, 8, 1), 67, 67), ((16, 60, 1), 91, 187), ((33, 8, 1), 77, 71), ((33, 60, 1), 101, 187),
         ((128, 0, 1), 99, 52), ((128, 8, 1), 116, 79), ((128, 60, 1), 142, 192), ((512, 8, 1), 267, 152), ((512, 60, 1), 296, 224),
         ((2048, 0, 1), 658, 241), ((2048, 60, 1), 1054, 542), ((16, 0, 8), 83, 69), ((16, 0, 64), 183, 189), ((33, 0, 64), 294, 319),
         ((128, 0, 32), 511, 341)]
MLSTM = [((16, 0, 1), 17, 15), ((16, 8, 1), 26, 21), ((16, 60, 1), 52, 69), ((33, 0, 1), 24, 17), ((33, 8, 1), 36, 26), ((33, 60, 1), 62, 71),
         ((128, 0, 1), 60, 20), ((128, 60, 1), 116, 73), ((512, 60, 1), 337, 114), ((2048, 60, 1), 1223, 390), ((16, 0, 8), 36, 23),
         ((16, 0, 64), 173, 77), ((33, 0, 64), 331, 120), ((128, 0, 32), 601, 126)]
SPACE = [((128, 0, 1), 44, 42), ((128, 8, 1), 52, 58), ((128, 60, 1), 108, 171), ((512, 0, 1), 106, 79), ((512, 8, 1), 142, 122),
         ((512, 60, 1), 151, 198), ((2048, 0, 1), 368, 222), ((2048, 8, 1), 513, 386), ((2048, 60, 1), 517, 460), ((128, 0, 32), 568, 349)]
MEASURED = [("_DELTA_COST", 16, 128, *m) for m in DELTA] + [("_MLSTM_COST", 16, 128, *m) for m in MLSTM] + [("_SPACE_COST", 64, 64, *m) for m in SPACE]


@pytest.mark.parametrize("name,heads,size,what,by_token,in_chunks", MEASURED)
def test_the_faster_way_is_taken(name, heads, size, what, by_token, in_chunks):
    tokens, singles, prompts = what
    rows = SimpleNamespace(max_q_len=tokens, n_rows=tokens * prompts + singles, n_seqs=prompts + singles)
    taken = in_chunks if getattr(ops, name).chunks_pay(rows, heads, size) else by_token
    assert taken <= 1.05 * min(by_token, in_chunks)


@pytest.mark.parametrize("name", ["_DELTA_COST", "_MLSTM_COST", "_SPACE_COST"])
def test_long_prompts_alone_are_walked_in_chunks(name):
    for tokens in (128, 500, 2048, 20000):
        for prompts in (1, 2, 8):
            for heads in (8, 32, 128):
                rows = SimpleNamespace(max_q_len=tokens, n_rows=tokens * prompts, n_seqs=prompts)
                assert getattr(ops, name).chunks_pay(rows, heads, getattr(ops, name).size), (tokens, prompts, heads)


# the same with the kernels of today, in a graph (launched one by one, the short ones are as long as the host's work)
DELTA_IN_GRAPH = [((16, 0, 1), 52, 27), ((16, 8, 1), 57, 37), ((16, 60, 1), 78, 143), ((33, 8, 1), 64, 45), ((33, 60, 1), 88, 146),
                  ((128, 0, 1), 84, 32), ((128, 8, 1), 100, 50), ((128, 60, 1), 123, 150), ((512, 8, 1), 255, 78), ((512, 60, 1), 290, 184),
                  ((2048, 0, 1), 658, 177), ((2048, 60, 1), 971, 330), ((16, 0, 8), 66, 39), ((16, 0, 64), 174, 168), ((33, 0, 64), 284, 293),
                  ((128, 0, 32), 520, 300)]
MLSTM_IN_GRAPH = [((16, 0, 1), 10, 8), ((16, 8, 1), 16, 17), ((16, 60, 1), 40, 60), ((33, 0, 1), 16, 10), ((33, 8, 1), 26, 19), ((33, 60, 1), 50, 60),
                  ((128, 0, 1), 51, 14), ((128, 60, 1), 103, 62), ((512, 60, 1), 345, 91), ((2048, 60, 1), 1292, 210), ((16, 0, 8), 27, 16),
                  ((16, 0, 64), 158, 66), ((33, 0, 64), 314, 108), ((128, 0, 32), 585, 113)]
SPACE_IN_GRAPH = [((128, 0, 1), 32, 34), ((128, 8, 1), 41, 51), ((128, 60, 1), 97, 164), ((512, 0, 1), 93, 66), ((512, 8, 1), 129, 112),
                  ((512, 60, 1), 139, 187), ((2048, 0, 1), 349, 184), ((2048, 8, 1), 493, 194), ((2048, 60, 1), 495, 321), ((128, 0, 32), 540, 313)]
IN_GRAPH = [("_DELTA_COST", 16, 128, *m) for m in DELTA_IN_GRAPH] + [("_MLSTM_COST", 16, 128, *m) for m in MLSTM_IN_GRAPH] \
    + [("_SPACE_COST", 64, 64, *m) for m in SPACE_IN_GRAPH]


@pytest.mark.parametrize("name,heads,size,what,by_token,in_chunks", IN_GRAPH)
def test_the_faster_way_is_taken_in_a_graph(name, heads, size, what, by_token, in_chunks):
    tokens, singles, prompts = what
    rows = SimpleNamespace(max_q_len=tokens, n_rows=tokens * prompts + singles, n_seqs=prompts + singles)
    taken = in_chunks if getattr(ops, name).chunks_pay(rows, heads, size) else by_token
    assert taken <= 1.07 * min(by_token, in_chunks)
