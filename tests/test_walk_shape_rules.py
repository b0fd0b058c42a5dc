"""The rules by which the walks over chunks take their blocks, against what each shape was measured to take (B200, us of the whole call in a graph,
bfloat16, values of 128; state-space duality: of 64)."""

import pytest

from thing_htn_2026_b200 import ops

# heads, (tokens, single tokens beside them, prompts): us of the shapes from 1 on
LINEAR = [(4, (16, 60, 24), (62.9, 47.0, 39.8, 40.4)), (4, (40, 60, 48), (97.3, 74.4, 63.3, 57.2)), (4, (100, 8, 1), (19.2, 28.8, 24.4, 27.1)),
          (4, (300, 8, 8), (49.8, 40.1, 54.2, 63.2)), (4, (512, 0, 1), (32.9, 39.6, 55.7, 67.8)), (4, (600, 0, 8), (76.7, 60.2, 79.6, 95.9)),
          (8, (40, 60, 48), (188.7, 141.7, 116.7, 100.9)), (8, (300, 60, 2), (96.2, 71.3, 62.4, 69.2)), (8, (512, 0, 3), (64.8, 53.2, 63.8, 75.3)),
          (8, (2048, 0, 1), (107.3, 129.0, 189.4, 239.4)), (16, (16, 60, 32), (242.7, 174.8, 139.7, 114.5)), (16, (40, 8, 1), (37.7, 30.7, 33.3, 33.1)),
          (16, (512, 0, 8), (229.2, 193.2, 171.0, 177.8)), (16, (600, 0, 1), (49.7, 51.9, 69.4, 82.9)), (24, (128, 0, 2), (35.7, 30.6, 31.3, 34.0)),
          (24, (128, 0, 8), (95.9, 81.3, 70.2, 71.6)), (24, (300, 60, 16), (646.2, 491.8, 420.2, 397.2)), (32, (40, 0, 1), (20.9, 22.7, 19.8, 20.5)),
          (32, (40, 0, 2), (28.5, 27.9, 31.5, 32.6)), (32, (128, 60, 6), (393.6, 282.9, 229.9, 199.3)), (64, (40, 0, 2), (50.7, 38.5, 39.8, 38.9)),
          (64, (40, 8, 64), (1194.9, 924.3, 745.6, 664.9)), (64, (64, 0, 1), (27.9, 28.3, 31.6, 33.0)), (64, (600, 0, 16), (2076.2, 1665.5, 1473.9, 1501.6))]
MEASURED = [("thn_linear_attention_walk_shape", 128, *m) for m in LINEAR]


@pytest.mark.parametrize("rule,size,heads,what,us", MEASURED)
def test_the_fast_blocks_are_taken(rule, size, heads, what, us):
    tokens, singles, prompts = what
    shape = getattr(ops.lib(), rule)(tokens * prompts + singles, tokens, prompts + singles, heads, size)
    assert us[shape - 1] <= 1.15 * min(us)


@pytest.mark.parametrize("rule", sorted({m[0] for m in MEASURED}))
def test_blocks_fit_the_values(rule):
    for columns, shapes in ((16, {1}), (32, {1, 2}), (96, {1, 2}), (64, {1, 2, 3, 4})):
        for tokens in (1, 31, 33, 500, 100000):
            for seqs in (1, 3, 40, 5000):
                for heads in (1, 7, 32, 500):
                    assert getattr(ops.lib(), rule)(min(tokens * seqs, (1 << 31) - 1), tokens, seqs, heads, columns) in shapes
