"""Linear attention with gated decays in chunks of 32 tokens, against the same token by token in 64 bits: lengths at the
edges of chunks, values at the edges of a block's columns, every block shape, decays from nearly one to nothing."""

import pytest
import torch

from test_chunk_recurrences_gpu import BAD, close, same_reach, step
from thing_htn_2026_b200 import ops

pytestmark = pytest.mark.gpu
BF16, KEY = torch.bfloat16, 128


@pytest.fixture(autouse=True)
def chunks_always_pay(monkeypatch):
    monkeypatch.setattr(ops, "_LINEAR_COST", ops._LINEAR_COST._replace(lead=1e9))


def operands(lens, heads, vdim, seed, spread=2.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj = draw(sum(lens), heads * (2 * KEY + vdim) + 16).to(BF16)
    return proj, draw(sum(lens), heads * KEY + 4) * spread, draw(heads * KEY) + 2, draw(len(lens) + 1, heads, vdim, KEY)


def run(proj, gate, bias, state, rows, heads, vdim, tau, want_bits=0):
    state, err = state.clone(), ops.new_error_word(torch.device("cuda"))
    o = ops.linear_attention(proj, (8, 8 + heads * KEY, 16 + 2 * heads * KEY), state, rows, heads, KEY, vdim, gate=gate, gate_bias=bias, tau=tau,
                             q_scale=KEY ** -0.5, err=err)
    assert int(err.item()) == want_bits
    return o, state


@pytest.mark.parametrize("shape", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("lens,heads,vdim,tau,spread", [
    ([16], 2, 128, 16.0, 2.0), ([31, 1, 33], 3, 16, 16.0, 2.0), ([32, 64, 65, 2], 2, 96, 1.0, 2.0), ([97], 4, 256, 16.0, 30.0),
    ([40] * 8, 16, 128, 16.0, 2.0), ([70, 35], 1, 64, 0.1, 2.0), ([200], 2, 128, 100.0, 2.0)])
def test_matches_64_bits(monkeypatch, shape, lens, heads, vdim, tau, spread):
    rows, _, cu, slots = step(lens)
    proj, gate, bias, state = operands(lens, heads, vdim, sum(lens) + vdim, spread)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape)
    if not ops._linear_in_chunks(proj, (8, 8 + heads * KEY, 16 + 2 * heads * KEY), state, rows, heads, KEY, vdim, gate, bias):
        pytest.fail("not walked in chunks")
    o, got = run(proj, gate, bias, state, rows, heads, vdim, tau)
    decay = torch.exp(torch.nn.functional.logsigmoid(gate[:, :heads * KEY].double() + bias.double()) / tau).view(-1, heads, KEY)
    wide = proj.double()
    for i, slot in enumerate(slots):
        S = state[slot].double()
        want = []
        for r in range(cu[i], cu[i + 1]):
            q, k = (wide[r, at:at + heads * KEY].view(heads, KEY) for at in (8, 8 + heads * KEY))
            v = wide[r, 16 + 2 * heads * KEY:16 + heads * (2 * KEY + vdim)].view(heads, vdim)
            S = S * decay[r][:, None, :] + v[:, :, None] * k[:, None, :]
            want.append(torch.einsum("hek,hk->he", S, q) * KEY ** -0.5)
        close(o[cu[i]:cu[i + 1]], torch.stack(want), lens[i])
        close(got[slot], S, lens[i])


@pytest.mark.parametrize("bad", BAD + (-float("inf"),))
@pytest.mark.parametrize("what", ["q", "k", "v", "gate", "state"])
@pytest.mark.parametrize("lens,at,heads,vdim", [([70, 40], 37, 2, 128), ([33], 16, 2, 16), ([64], 32, 2, 64)])
def test_keeps_what_is_not_finite_to_itself(monkeypatch, bad, what, lens, at, heads, vdim):
    rows, _, cu, _ = step(lens)
    proj, gate, bias, state = operands(lens, heads, vdim, at)
    if what == "gate":
        gate[at, KEY + 9] = bad           # an infinity is a decay of one or of nothing
    elif what == "state":
        state[len(lens), 1, 5, 77] = bad
    else:
        proj[at, {"q": 8 + KEY + 5, "k": 8 + (heads + 1) * KEY + 7, "v": 16 + 2 * heads * KEY + vdim + 3}[what]] = bad
    chunks = run(proj, gate, bias, state, rows, heads, vdim, 16.0)
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 1 << 30)
    same_reach(chunks, run(proj, gate, bias, state, rows, heads, vdim, 16.0))


def test_what_the_rule_leaves_to_the_tokens():
    rows, _, _, _ = step([40])
    proj, gate, bias, state = operands([40], 2, 128, 1)
    offsets = (8, 8 + 2 * KEY, 16 + 4 * KEY)
    ask = lambda p=proj, o=offsets, s=state, r=rows, d=KEY, e=128, g=gate, b=bias: ops._linear_in_chunks(p, o, s, r, 2, d, e, g, b)      # noqa: E731
    assert ask() and ask(b=None)
    assert not ask(p=proj.float()) and not ask(d=64) and not ask(e=120) and not ask(r=step([15])[0])
    assert not ask(o=(8, 8 + 2 * KEY, 12 + 4 * KEY)) and not ask(o=(6, 8 + 2 * KEY, 16 + 4 * KEY))
    assert not ask(p=torch.empty(40, proj.shape[1] + 4, dtype=BF16, device="cuda")) and not ask(g=torch.empty(40, gate.shape[1] + 2, device="cuda"))
    assert not ask(b=torch.empty(2 * KEY + 1, device="cuda")[1:])


@pytest.mark.parametrize("shape", [1, 2, 3])
def test_a_wait_that_runs_out_sets_its_bit_and_the_kernel_returns(monkeypatch, shape):
    """With nothing brought the walk's wait ends after 20 ms, the bit is set, the state stays, and the next launch is right again."""
    rows, _, _, _ = step([70, 33])
    proj, gate, bias, state = operands([70, 33], 2, 128, 5)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape)
    want = run(proj, gate, bias, state, rows, 2, 128, 16.0)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape + 16)
    _, untouched = run(proj, gate, bias, state, rows, 2, 128, 16.0, ops.ERR_WAIT_TIMEOUT)
    assert torch.equal(untouched, state)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape)
    again = run(proj, gate, bias, state, rows, 2, 128, 16.0)
    assert torch.equal(again[0], want[0]) and torch.equal(again[1], want[1])


@pytest.mark.parametrize("shape", [1, 2, 3, 4])
def test_without_an_error_word_no_warp_waits_for_another(monkeypatch, shape):
    """A walk that has no word to say so cannot run out of a wait: with nothing brought its results are the same to the bit."""
    rows, _, _, _ = step([70, 33, 1])
    proj, gate, bias, state = operands([70, 33, 1], 2, 128, 6)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape)
    want, want_state = run(proj, gate, bias, state, rows, 2, 128, 16.0)
    monkeypatch.setattr(ops, "LINEAR_CHUNK_SHAPE", shape + 16)
    o = ops.linear_attention(proj, (8, 8 + 2 * KEY, 16 + 4 * KEY), state, rows, 2, KEY, 128, gate=gate, gate_bias=bias, tau=16.0, q_scale=KEY ** -0.5)
    assert torch.equal(o, want) and torch.equal(state, want_state)
