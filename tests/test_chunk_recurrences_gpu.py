"""Recurrences that are walked in chunks of 32 tokens on the tensor cores, against the same token by token
in 64 bits: lengths at the edges of chunks, a prompt that goes on from a state, values at the edges of a
block's columns."""

import pytest
import torch

from thing_htn_2026_b200 import ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def step(lens, held=0):
    dev = torch.device("cuda", 0)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    seq_lens = torch.full((len(lens) + 1,), held, dtype=torch.int32, device=dev)
    slots = torch.arange(len(lens), 0, -1, dtype=torch.int32, device=dev)      # sequence i in slot len - i
    rows = ops.step_rows(torch.tensor(cu, dtype=torch.int32, device=dev), slots, seq_lens, cu[-1], max(lens))
    return rows, seq_lens, cu, slots.cpu().tolist()


def close(got, want, tokens):
    """float32 sums of a few dozen products per token and a state that is rounded once per token or chunk:
    2^-20 of the result's size, and a token's roundings add up at most linearly."""
    scale = want.abs().amax()
    assert torch.isfinite(got).all()
    assert (got.double() - want).abs().max() <= (8 + tokens / 8) * 2 ** -23 * scale


@pytest.mark.parametrize("lens,held,n_heads,n_kv,vdim", [
    ([16], 0, 2, 1, 128), ([31, 1, 33], 0, 4, 2, 16), ([32, 64, 65, 2], 0, 2, 2, 48), ([100], 7, 4, 1, 128),
    ([40, 17], 1, 2, 1, 256), ([70] * 8, 0, 16, 4, 64), ([35] * 5, 2, 16, 4, 96), ([20, 97], 64, 2, 2, 160),
    ([70] * 10, 0, 16, 4, 64), ([40] * 12, 5, 32, 8, 48)])
def test_delta_matches_64_bits(lens, held, n_heads, n_kv, vdim):
    g = torch.Generator().manual_seed(sum(lens) + vdim)
    rows, seq_lens, cu, slots = step(lens, held)
    dev, key, taps, eps = rows.slots.device, 128, 4, 1e-6
    shape = ops.DeltaShape(n_heads, n_kv, key, vdim, taps)
    draw = lambda *s: torch.randn(*s, generator=g)
    proj, w = draw(cu[-1], shape.proj_width).to(BF16), draw(shape.conv_channels, taps) * 0.5
    a_log, dt_bias = torch.rand(n_heads, generator=g) * 4 - 2, draw(n_heads)
    state, ring = draw(len(lens) + 1, n_heads, vdim, key) * 0.2, draw(len(lens) + 1, taps, shape.conv_channels).to(BF16)
    got_state, got_ring = state.to(dev), ring.to(dev)
    assert ops._delta_in_chunks(proj.to(dev), w.to(dev), got_state, got_ring, rows, shape)
    got = ops.delta_rule(proj.to(dev), w.to(dev), a_log.to(dev), dt_bias.to(dev), got_state, got_ring, rows, seq_lens, shape, eps)
    want, want_state = torch.zeros(cu[-1], n_heads, vdim, dtype=torch.float64), state.double()
    qk, gate_end = n_kv * key, shape.gate_offset + n_heads * vdim
    for i, slot in enumerate(slots):
        S = want_state[slot]
        for r in range(cu[i], cu[i + 1]):
            pos, acc = held + r - cu[i], torch.zeros(shape.conv_channels, dtype=torch.float64)
            for back in range(min(taps - 1, pos) + 1):
                raw = proj[r - back, :shape.conv_channels] if back <= r - cu[i] else ring[slot, (pos - back) % taps]
                acc += w[:, taps - 1 - back].double() * raw.double()
            y = torch.nn.functional.silu(acc)
            q, k = y[:qk].view(n_kv, key), y[qk:2 * qk].view(n_kv, key)
            q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + eps) * key ** -0.5).repeat_interleave(n_heads // n_kv, 0)
            k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + eps)).repeat_interleave(n_heads // n_kv, 0)
            b = torch.sigmoid(proj[r, gate_end:gate_end + n_heads].double())
            step_size = torch.nn.functional.softplus(proj[r, gate_end + n_heads:gate_end + 2 * n_heads].double() + dt_bias.double())
            S = torch.exp(-torch.exp(a_log.double()) * step_size)[:, None, None] * S
            u = b[:, None] * (y[2 * qk:].view(n_heads, vdim) - torch.einsum("hek,hk->he", S, k))
            S = S + u[:, :, None] * k[:, None, :]
            want[r] = torch.einsum("hek,hk->he", S, q)
        want_state[slot] = S
    close(got.cpu(), want, max(lens))
    close(got_state.cpu(), want_state, max(lens))
    for i, slot in enumerate(slots):
        for r in range(max(cu[i], cu[i + 1] - (taps - 1)), cu[i + 1]):
            assert torch.equal(got_ring[slot, (held + r - cu[i]) % taps].cpu(), proj[r, :shape.conv_channels])


@pytest.mark.parametrize("n_seqs,held", [(65535, 3), (65537, 2)])
def test_the_ring_of_very_many_sequences(n_seqs, held):
    """Two rows a sequence, as many sequences as a grid's second and third axes cannot count."""
    dev = torch.device("cuda", 0)
    shape, lens = ops.DeltaShape(1, 1, 4, 4, 4), torch.full((n_seqs,), held, dtype=torch.int32, device=dev)
    rows = ops.step_rows(torch.arange(0, 2 * n_seqs + 1, 2, dtype=torch.int32, device=dev), torch.arange(n_seqs, dtype=torch.int32, device=dev),
                         lens, 2 * n_seqs, 2)
    g = torch.Generator(device=dev).manual_seed(n_seqs)
    draw = lambda *s: torch.randn(*s, generator=g, device=dev)
    proj, ring = draw(2 * n_seqs, shape.proj_width).to(BF16), draw(n_seqs, 4, shape.conv_channels).to(BF16)
    want = ring.clone()
    for i in range(2):
        want[:, (held + i) % 4] = proj[i::2, :shape.conv_channels]
    ops.delta_rule(proj, draw(shape.conv_channels, 4), draw(1), draw(1), torch.zeros(n_seqs, 1, 4, 4, device=dev), ring, rows, lens, shape, 1e-6)
    assert torch.equal(ring, want)


@pytest.mark.parametrize("lens,n_heads,vdim", [
    ([16], 2, 128), ([31, 1, 33], 3, 16), ([32, 64, 65, 2], 2, 48), ([97], 4, 256), ([40] * 8, 16, 128), ([70, 35], 1, 64)])
def test_matrix_memory_matches_64_bits(lens, n_heads, vdim):
    g = torch.Generator().manual_seed(sum(lens) + vdim)
    rows, _, cu, slots = step(lens)
    dev, key, cap, scale = rows.slots.device, 128, 15.0, 128 ** -0.5
    draw = lambda *s: torch.randn(*s, generator=g)
    proj = draw(cu[-1], n_heads * (2 * key + vdim) + 8 * (n_heads % 2)).to(BF16)
    pre, bias_i, bias_f = draw(cu[-1], 2 * n_heads) * 3, draw(n_heads) * 2, draw(n_heads) * 2 + 1
    state = draw(len(lens) + 1, n_heads, vdim, key)
    normaliser = draw(len(lens) + 1, n_heads, 1, key + 1).expand(-1, -1, vdim // 16, -1).contiguous()
    got_state, got_normaliser = state.to(dev), normaliser.to(dev)
    assert ops._mlstm_in_chunks(proj.to(dev), got_state, rows, n_heads, key, vdim)
    got = ops.mlstm(proj.to(dev), pre.to(dev), bias_i.to(dev), bias_f.to(dev), cap, got_state, got_normaliser, rows, n_heads, key,
                    vdim, scale).cpu()
    gi = cap * torch.tanh((pre[:, :n_heads].double() + bias_i.double()) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((pre[:, n_heads:].double() + bias_f.double()) / cap))
    parts = proj.double()
    for i, slot in enumerate(slots):
        S, n, m = state[slot].double(), normaliser[slot, :, 0, :key].double(), normaliser[slot, :, 0, key].double()
        for r in range(cu[i], cu[i + 1]):
            q, k = parts[r, :n_heads * key].view(n_heads, key) * scale, parts[r, n_heads * key:2 * n_heads * key].view(n_heads, key)
            v = parts[r, 2 * n_heads * key:n_heads * (2 * key + vdim)].view(n_heads, vdim)
            top = torch.maximum(gf[r] + m, gi[r])
            keep, take, m = torch.exp(gf[r] + m - top), torch.exp(gi[r] - top), top
            S = keep[:, None, None] * S + take[:, None, None] * v[:, :, None] * k[:, None, :]
            n = keep[:, None] * n + take[:, None] * k
            below = torch.maximum((n * q).sum(-1).abs(), torch.exp(-m)) + 1e-6
            want = torch.einsum("hek,hk->he", S, q) / below[:, None]
            # the maximum is of the order of ten, so its roundings (2^-21 a step) weigh on every exponential; a denominator
            # that cancels magnifies the error of n . q by |n| |q| over itself
            slack = (1 + (n.norm(dim=-1) * q.norm(dim=-1) / below))[:, None] * want.abs().amax(dim=-1, keepdim=True)
            assert ((got[r].double() - want).abs() <= (64 + 2 * len(range(cu[i], r + 1))) * 2 ** -23 * slack).all()
        scale_s = S.abs().amax()
        bound = (64 + 2 * lens[i]) * 2 ** -23
        assert (got_state[slot].cpu().double() - S).abs().max() <= bound * scale_s
        copies = got_normaliser[slot].cpu().double()
        assert (copies[:, :, :key] - n[:, None]).abs().max() <= bound * n.abs().amax()
        assert (copies[:, :, key] - m[:, None]).abs().max() <= bound * m.abs().amax().clamp(min=1)


def test_matrix_memory_of_many_short_sequences():
    """What a step of long and short sequences needs grows with its rows, not with the longest times their number."""
    bytes_for = ops.lib().thn_mlstm_chunks_scratch_bytes
    assert bytes_for(100999, 1000, 16) <= 1.05 * bytes_for(100999, 1, 16)
    test_matrix_memory_matches_64_bits([33] + [1] * 9 + [70, 32, 1, 64], 2, 64)


@pytest.mark.parametrize("lens,held,n_heads,groups,vdim", [
    ([112], 0, 4, 2, 64), ([1, 129, 33], 0, 2, 2, 16), ([160, 2], 3, 8, 1, 96), ([115, 64], 1, 64, 8, 128), ([113] * 3, 0, 128, 4, 64)])
def test_state_space_matches_64_bits(lens, held, n_heads, groups, vdim):
    g = torch.Generator().manual_seed(sum(lens) + vdim)
    rows, seq_lens, cu, slots = step(lens, held)
    dev, n, taps, offset = rows.slots.device, 128, 4, 8
    draw = lambda *s: torch.randn(*s, generator=g)
    inner = n_heads * vdim
    channels = inner + 2 * groups * n
    shape = ops.StateSpace(n_heads, vdim, n, groups, draw(channels, taps) * 0.5, draw(channels) * 0.1, draw(n_heads) - 2,
                           torch.exp(draw(n_heads)), draw(n_heads))
    there = ops.StateSpace(n_heads, vdim, n, groups, *(t.to(dev) for t in (shape.conv_w, shape.conv_b, shape.dt_bias, shape.rate, shape.skip)))
    proj, dt = draw(cu[-1], offset + channels).to(BF16), draw(cu[-1], n_heads)
    state, ring = draw(len(lens) + 1, n_heads, vdim, n) * 0.2, draw(len(lens) + 1, taps, channels).to(BF16)
    got_state, got_ring = state.to(dev), ring.to(dev)
    assert ops._space_in_chunks(proj.to(dev), offset, got_state, got_ring, rows, there)
    got = ops.state_space(proj.to(dev), offset, dt.to(dev), there, got_state, got_ring, rows, seq_lens)
    want, want_state = torch.zeros(cu[-1], n_heads, vdim, dtype=torch.float64), state.double()
    size = torch.nn.functional.softplus(dt.double() + shape.dt_bias.double())
    decay = torch.exp(-shape.rate.double() * size)
    for i, slot in enumerate(slots):
        S = want_state[slot]
        for r in range(cu[i], cu[i + 1]):
            pos, acc = held + r - cu[i], shape.conv_b.double()
            for back in range(min(taps - 1, pos) + 1):
                raw = proj[r - back, offset:] if back <= r - cu[i] else ring[slot, (pos - back) % taps]
                acc = acc + shape.conv_w[:, taps - 1 - back].double() * raw.double()
            y = torch.nn.functional.silu(acc)
            x = y[:inner].view(n_heads, vdim)
            B, C = (y[inner + a * groups * n:inner + (a + 1) * groups * n].view(groups, n).repeat_interleave(n_heads // groups, 0) for a in (0, 1))
            S = decay[r][:, None, None] * S + (size[r][:, None] * x)[:, :, None] * B[:, None, :]
            want[r] = torch.einsum("hek,hk->he", S, C) + shape.skip.double()[:, None] * x
        want_state[slot] = S
    close(got.cpu(), want, max(lens))
    close(got_state.cpu()[1:], want_state[1:], max(lens))


# What is not finite must reach what it reaches token by token and nothing else: in particular no token ahead of it.
BAD = (float("nan"), float("inf"))


def same_reach(chunks, tokens):
    """The same entries are finite, and those are close: two float32 ways to take the same sums."""
    for a, b in zip(chunks, tokens):
        there = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), there) and there.any()
        assert (a[there] - b[there]).abs().max() <= 2 ** -16 * b[there].abs().max()


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("what", ["q", "k", "v", "b", "a", "a_log"])
@pytest.mark.parametrize("lens,at,vdim", [([70, 40], 37, 128), ([33], 16, 16), ([40], 31, 160)])
def test_delta_keeps_what_is_not_finite_to_itself(monkeypatch, bad, what, lens, at, vdim):
    rows, seq_lens, cu, _ = step(lens)
    dev, shape = rows.slots.device, ops.DeltaShape(4, 2, 128, vdim, 4)
    g = torch.Generator(device=dev).manual_seed(at)
    draw = lambda *s: torch.randn(*s, generator=g, device=dev)
    proj, w, a_log, dt_bias = draw(cu[-1], shape.proj_width).to(BF16), draw(shape.conv_channels, 4) * 0.5, draw(4), draw(4)
    gate_end = shape.gate_offset + 4 * vdim
    column = {"q": 5, "k": 256 + 128 + 7, "v": 512 + vdim + 3, "b": gate_end + 1, "a": gate_end + 4 + 2}.get(what)
    if column is None:
        a_log[1] = bad          # an infinite one is a decay of zero, a NaN a NaN
    else:
        proj[at, column] = bad
    state, ring = draw(len(lens) + 1, 4, vdim, 128) * 0.2, torch.zeros(len(lens) + 1, 4, shape.conv_channels, dtype=BF16, device=dev)
    results = []
    for lanes in (0, 8):
        monkeypatch.setattr(ops, "DELTA_LANES", lanes)
        s = state.clone()
        assert ops._delta_in_chunks(proj, w, s, ring, rows, shape) == (lanes == 0)
        results.append((ops.delta_rule(proj, w, a_log, dt_bias, s, ring.clone(), rows, seq_lens, shape, 1e-6), s))
    same_reach(*results)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("what", ["q", "k", "v", "i", "f"])
@pytest.mark.parametrize("lens,at,heads,vdim", [([70, 40], 37, 2, 128), ([33], 16, 2, 16), ([40] * 8, 50, 16, 128)])
def test_matrix_memory_keeps_what_is_not_finite_to_itself(bad, what, lens, at, heads, vdim):
    rows, _, cu, _ = step(lens)
    dev = rows.slots.device
    g = torch.Generator(device=dev).manual_seed(at)
    draw = lambda *s: torch.randn(*s, generator=g, device=dev)
    proj, pre = draw(cu[-1], heads * (256 + vdim)).to(BF16), draw(cu[-1], 2 * heads)
    if what in "if":
        pre[at, 1 + (heads if what == "f" else 0)] = bad       # (the cap makes a large number of an infinity)
    else:
        proj[at, {"q": 128 + 5, "k": (heads + 1) * 128 + 7, "v": heads * 256 + vdim + 3}[what]] = bad
    state, normaliser = draw(len(lens) + 1, heads, vdim, 128), draw(len(lens) + 1, heads, 1, 129).expand(-1, -1, vdim // 16, -1).contiguous()
    results = []
    for lanes in (0, 8):
        ops.set_mlstm_kernel(True, lanes)
        try:
            s, n = state.clone(), normaliser.clone()
            assert ops._mlstm_in_chunks(proj, s, rows, heads, 128, vdim) == (lanes == 0)
            results.append((ops.mlstm(proj, pre, torch.zeros(heads, device=dev), torch.ones(heads, device=dev), 15.0, s, n, rows, heads,
                                      128, vdim, 128 ** -0.5), s, n[..., :128]))     # (behind a NaN gate the maximum says nothing)
        finally:
            ops.set_mlstm_kernel(True, 0)
    same_reach(*results)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("what", ["x", "B", "C", "step", "rate"])
@pytest.mark.parametrize("lens,at,heads,groups,vdim", [([130, 40], 37, 4, 2, 64), ([113], 63, 2, 1, 16), ([128] * 8, 200, 64, 8, 64)])
def test_state_space_keeps_what_is_not_finite_to_itself(monkeypatch, bad, what, lens, at, heads, groups, vdim):
    rows, seq_lens, cu, _ = step(lens)
    dev, inner = rows.slots.device, heads * vdim
    g = torch.Generator(device=dev).manual_seed(at)
    draw = lambda *s: torch.randn(*s, generator=g, device=dev)
    channels = inner + 256 * groups
    shape = ops.StateSpace(heads, vdim, 128, groups, draw(channels, 4) * 0.5, draw(channels) * 0.1, draw(heads) - 2, torch.exp(draw(heads)), draw(heads))
    proj, dt = draw(cu[-1], channels).to(BF16), draw(cu[-1], heads)
    if what == "rate":
        shape.rate[1] = bad     # an infinite one is a decay of zero
    elif what == "step":
        dt[at, 1] = bad
    else:
        proj[at, {"x": vdim + 3, "B": inner + 7, "C": inner + groups * 128 + 9}[what]] = bad
    state, ring = draw(len(lens) + 1, heads, vdim, 128) * 0.2, torch.zeros(len(lens) + 1, 4, channels, dtype=BF16, device=dev)
    results = []
    for in_chunks in (True, False):
        monkeypatch.setattr(ops, "_space_in_chunks", lambda *a, answer=in_chunks: answer)
        s = state.clone()
        results.append((ops.state_space(proj, 0, dt, shape, s, ring.clone(), rows, seq_lens), s))
    same_reach(*results)
