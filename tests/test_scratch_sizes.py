"""Sizes of scratch memory as the kernel library states them, beyond 2^31 and 2^32 bytes: they reach Python with their 64 bits, and an entry point
refuses a scratch that is too small."""

import glob
import os
import re

import pytest

from thing_htn_2026_b200 import ops
from thing_htn_2026_b200.ops import library

KEY, SCORE = 2 * (128 + 8), 2 * (32 + 8)      # bytes of a row of keys and of a row of G in one plane
ROWS = (18 * 2048, 36 * 2048, 64 * 8192)      # many prompts in one step


def chunk_places(rows, seqs):
    return rows // 32 + seqs


# of n rows in n / 2,048 sequences; sizes that the recurrences pad to themselves
FORMULAS = {
    "thn_linear_attention_chunks_scratch_bytes": (lambda n: (n, n // 2048, 32), lambda n, s, h: h * n * 3 * (2 * KEY + SCORE) + chunk_places(n, s) * h * 512),
    "thn_mlstm_chunks_scratch_bytes": (lambda n: (n, n // 2048, 32), lambda n, s, h: h * n * (3 * SCORE + 16) + chunk_places(n, s) * h * 512),
    "thn_delta_chunks_scratch_bytes": (lambda n: (n, 32, 16, 128), lambda n, h, kv, e: 6 * kv * n * KEY + h * n * (3 * KEY + 3 * SCORE + 4 * e + 24)),
    "thn_state_space_chunks_scratch_bytes": (lambda n: (n, 128, 64, 8), lambda n, h, e, g: n * (6 * g * KEY + h * (3 * SCORE + 20 + 4 * e))),
    "thn_linear_attention_scratch_floats": (lambda n: (n, 32, 128, 128, 1), lambda n, h, d, e, mode: n * h * (3 * d + e)),
    "thn_state_space_scratch_floats": (lambda n: (n, 128, 64, 128, 8), lambda n, h, e, d, g: n * (g * 2 * d + h * (e + 4))),
    "thn_wkv_scratch_floats": (lambda n: (n, 64, 64), lambda n, h, d: n * h * (4 * d + 4)),
    "thn_choose_tokens_scratch_floats": (lambda n: (n * 256, 151936), lambda n, v: 64 * n),
    "thn_attention_decode_scratch_floats": (lambda n: (n, 32, 64, 128), lambda n, q, k, d: n * q * k * (d + 2)),
}


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("name", sorted(FORMULAS))
def test_sizes(name, rows):
    arguments, size = FORMULAS[name]
    arguments = arguments(rows)
    assert getattr(ops.lib(), name)(*arguments) == size(*arguments)
    assert rows < ROWS[-1] or size(*arguments) > 1 << 32


def test_every_64_bit_result_is_read_as_one():
    names = set()
    for path in glob.glob(os.path.join(os.path.dirname(library.__file__), "..", "csrc", "*.cu")):
        with open(path) as handle:
            names |= set(re.findall(r"THN_API (?:long long|size_t|int64_t) (\w+)\(", handle.read()))
    assert names == set(FORMULAS) and all(name.endswith(ops._SIZES) for name in names)


def test_a_scratch_that_is_too_small_is_refused():
    n, seqs, heads = 36 * 2048, 36, 32
    at = 1 << 20          # an address that nothing reads
    need = ops.lib().thn_linear_attention_chunks_scratch_bytes(n, seqs, heads)
    with pytest.raises(ops.KernelError, match=f"{need - 1} bytes of scratch, {need} needed"):
        ops._call("thn_linear_attention_chunks", at, at, at, need - 1, at, 3 * heads * 128, 0, heads * 128, 2 * heads * 128, at, heads * 128, None, 1.0,
                  at, at, n, 2048, seqs, heads, 128, 128, 1.0, 0, None, None)
    need = ops.lib().thn_mlstm_chunks_scratch_bytes(n, seqs, heads)
    with pytest.raises(ops.KernelError, match=f"{need - 1} bytes of scratch, {need} needed"):
        ops._call("thn_mlstm_chunks", at, at, at, at, need - 1, at, 3 * heads * 128, at, at, at, 15.0, at, at, n, 2048, seqs, heads, 128, 128, 1.0, 1e-6,
                  None)
    need = ops.lib().thn_delta_chunks_scratch_bytes(n, heads, 16, 128)
    shape = ops.DeltaShape(heads, 16, 128, 128, 4)
    with pytest.raises(ops.KernelError, match=f"{need - 1} bytes of scratch, {need} needed"):
        ops._call("thn_delta_chunks", at, at, at, need - 1, at, at, at, at, at, at, at, at, at, at, n, 2048, seqs, heads, 16, 128, 128, 4,
                  shape.proj_width, 1e-6, None, None)
    need = ops.lib().thn_state_space_chunks_scratch_bytes(n, 128, 64, 8)
    inner = 128 * 64
    with pytest.raises(ops.KernelError, match=f"{need - 1} bytes of scratch, {need} needed"):
        ops._call("thn_state_space_chunks", at, at, at, need - 1, at, 2 * inner + 16 * 128, inner, at, at, at, at, at, at, at, at, at, at, at, at, n, 2048,
                  seqs, 128, 64, 128, 8, 4, None, None)
