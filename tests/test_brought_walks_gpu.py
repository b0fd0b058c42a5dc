"""Walks whose operands more warps bring by bulk copies: many long sequences (blocks of 64 columns) against the same sequences one by one
(narrow blocks, other sums over the keys), with last chunks of one token, of 31 and of 32."""

import pytest
import torch

from test_chunk_recurrences_gpu import BF16, step
from test_chunk_recurrences_gpu import test_matrix_memory_matches_64_bits as matrix_memory_matches_64_bits
from thing_htn_2026_b200 import ops

pytestmark = pytest.mark.gpu
LENS = [224, 225, 255, 256, 1, 600, 231, 240]


def close(a, b):
    # the same sums of up to 128 and 32 products in another order, a state rounded once a chunk: 2^-18 of the size
    assert torch.isfinite(a).all() and (a.double() - b.double()).abs().max() <= 2 ** -18 * b.abs().max()


def alone(run, state, slots, cu):
    """The sequences one by one from the same states."""
    outs, states = [], state.clone()
    for i, slot in enumerate(slots):
        rows, lens, _, _ = step([cu[i + 1] - cu[i]])
        own = torch.zeros(2, *state.shape[1:], device=state.device)
        own[1] = state[slot]
        outs.append(run(slice(cu[i], cu[i + 1]), own, rows, lens))
        states[slot] = own[1]
    return torch.cat(outs), states


@pytest.mark.parametrize("heads,vdim", [(16, 128), (32, 64)])
def test_delta_rule(heads, vdim):
    rows, lens, cu, slots = step(LENS)
    g = torch.Generator(device="cuda").manual_seed(vdim)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    shape = ops.DeltaShape(heads, 4, 128, vdim, 4)
    proj, w, a_log, dt = draw(cu[-1], shape.proj_width).to(BF16), draw(shape.conv_channels, 4) * 0.5, draw(heads), draw(heads)
    state = draw(len(LENS) + 1, heads, vdim, 128) * 0.2
    err = ops.new_error_word(torch.device("cuda"))

    def run(part, s, r, n, word=err):
        ring = torch.zeros(s.shape[0], 4, shape.conv_channels, dtype=BF16, device="cuda")
        return ops.delta_rule(proj[part].contiguous(), w, a_log, dt, s, ring, r, n, shape, 1e-6, word)
    together = state.clone()
    o = run(slice(0, cu[-1]), together, rows, lens)
    want, states = alone(run, state, slots, cu)
    close(o, want)
    close(together[1:], states[1:])
    assert int(err.item()) == 0
    # without an error word the warps copy themselves: the same to the bit, in wide blocks and in narrow ones
    copied = state.clone()
    assert torch.equal(run(slice(0, cu[-1]), copied, rows, lens, None), o) and torch.equal(copied, together)
    narrow, copied = state[:2].clone(), state[:2].clone()
    r, n, _, _ = step([cu[1]])
    assert torch.equal(run(slice(0, cu[1]), narrow, r, n), run(slice(0, cu[1]), copied, r, n, None)) and torch.equal(narrow, copied)


@pytest.mark.parametrize("heads,vdim", [(16, 64), (8, 128)])
def test_state_space(heads, vdim):
    rows, lens, cu, slots = step(LENS)
    g = torch.Generator(device="cuda").manual_seed(heads)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")      # noqa: E731
    inner, channels = heads * vdim, heads * vdim + 4 * 128
    shape = ops.StateSpace(heads, vdim, 128, 2, draw(channels, 4) * 0.5, draw(channels) * 0.02, draw(heads) - 2, torch.exp(draw(heads)), draw(heads))
    proj, dt = draw(cu[-1], inner + channels).to(BF16), draw(cu[-1], heads)
    state = draw(len(LENS) + 1, heads, vdim, 128) * 0.1
    err = ops.new_error_word(torch.device("cuda"))

    def run(part, s, r, n, word=err):
        ring = torch.zeros(s.shape[0], 4, channels, dtype=BF16, device="cuda")
        return ops.state_space(proj[part].contiguous(), inner, dt[part].contiguous(), shape, s, ring, r, n, word)
    together = state.clone()
    o = run(slice(0, cu[-1]), together, rows, lens)
    want, states = alone(run, state, slots, cu)
    close(o, want)
    close(together[1:], states[1:])
    assert int(err.item()) == 0
    # without an error word the warps copy themselves: the same to the bit, in wide blocks and in narrow ones
    copied = state.clone()
    assert torch.equal(run(slice(0, cu[-1]), copied, rows, lens, None), o) and torch.equal(copied, together)
    narrow, copied = state[:2].clone(), state[:2].clone()
    r, n, _, _ = step([cu[1]])
    assert torch.equal(run(slice(0, cu[1]), narrow, r, n), run(slice(0, cu[1]), copied, r, n, None)) and torch.equal(narrow, copied)


# the blocks' shapes of the matrix memory (thn_mlstm_walk_shape)
@pytest.mark.parametrize("lens,heads,vdim,shape", [([70], 16, 128, 1), ([40, 33], 16, 128, 2), ([40] * 4, 16, 128, 3), ([64, 31, 64, 64], 24, 96, 4),
                                                   ([40] * 6, 16, 128, 4), ([33, 16], 32, 64, 2), ([40] * 9, 16, 128, 5)])
def test_matrix_memory(monkeypatch, lens, heads, vdim, shape):
    monkeypatch.setattr(ops, "_MLSTM_COST", ops._MLSTM_COST._replace(lead=1e9))
    assert ops.lib().thn_mlstm_walk_shape(sum(lens), max(lens), len(lens), heads, vdim) == shape
    matrix_memory_matches_64_bits(lens, heads, vdim)
