"""Prompt attention on tensor memory: which keys a row sees, where windows, kept first keys and chunks begin or end at the edges of a
tile of 64 keys or one beside them, against a softmax in 64 bits."""

import pytest
import torch

from test_kernels_gpu import DEV, PagedFixture, rand, write_kv
from thing_htn_2026_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,keep_first,chunk", [
    (None, 0, None), (1, 0, None), (63, 0, None), (64, 0, None), (65, 0, None), (130, 0, None), (1, 1, None), (5, 64, None), (64, 65, None), (70, 200, None),
    (None, 0, 1), (None, 0, 63), (None, 0, 64), (None, 0, 65), (None, 0, 128)])
def test_matches_64_bits(window, keep_first, chunk):
    lens, n_q, n_kv, D, bf16 = [150, 64, 1, 321], 2, 1, 128, torch.bfloat16
    fix = PagedFixture(n_kv, D, lens, bf16)
    rows, cu = fix.rows(lens)
    q, k, v = (rand((cu[-1], n, D), bf16, seed) for n, seed in ((n_q, 1), (n_kv, 2), (n_kv, 3)))
    write_kv(fix, rows, k, v, n_q)
    err = ops.new_error_word(DEV)
    got = ops.attention_prefill_tcgen05(q.reshape(cu[-1], -1).to(DEV), rows, rows.tiles, fix.kv, n_q, D ** -0.5, window, err, keep_first, chunk)
    assert int(err.item()) == 0
    got = got.double().cpu().view(cu[-1], n_q, D)
    for a, b in zip(cu, cu[1:]):
        i, j = torch.arange(b - a)[:, None], torch.arange(b - a)[None]
        seen = (j <= i) & ((i - j < window) | (j < keep_first) if window else i // chunk == j // chunk if chunk else j <= i)
        for h in range(n_q):
            values = v[a:b, 0].double()
            p = torch.softmax((q[a:b, h].double() @ k[a:b, 0].double().T * D ** -0.5).masked_fill(~seen, -torch.inf), -1)
            want = p @ values
            # weights and results are rounded to bfloat16 once (2^-9 each), the rest is float32
            assert ((got[a:b, h] - want).abs() <= 2 ** -8 * (p @ values.abs()) + 2 ** -8 * want.abs()).all()
