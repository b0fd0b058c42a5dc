"""The convolution and the selective scan of steps with several tokens, bfloat16, against the same in
64 bits: sizes at the edges of the kernels' stages, lanes and pieces."""

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
    seq_lens = torch.full((len(lens),), held, dtype=torch.int32, device=dev)
    rows = ops.step_rows(torch.tensor(cu, dtype=torch.int32, device=dev), torch.arange(len(lens), dtype=torch.int32, device=dev),
                         seq_lens, cu[-1], max(lens))
    return rows, seq_lens, cu


@pytest.mark.parametrize("channels,state,lens", [
    (5, 3, [2]), (33, 8, [15, 16, 17, 1]), (64, 9, [33]), (100, 16, [31, 48, 2]), (16, 16, [1, 1, 2]),
    (2400, 16, [18, 33]), (70, 17, [40]), (40, 32, [16, 5]), (40, 40, [16, 5])])
def test_scan_matches_64_bits(channels, state, lens, infinite=False):
    g = torch.Generator().manual_seed(channels * 31 + state)
    rows, _, cu = step(lens)
    total, dev = cu[-1], rows.slots.device
    draw = lambda *shape: torch.randn(*shape, generator=g)
    x, bc, gate = draw(total, channels).to(BF16), draw(total, 2 * state + 2).to(BF16), draw(total, channels + 3).to(BF16)
    dt, bias, d, start = draw(total, channels) * 2, draw(channels) * 0.1, draw(channels), draw(len(lens), channels, state)
    a = -torch.exp(draw(channels, state))
    if infinite:
        a[::2, state // 2] = -float("inf")
    held = start.to(dev)
    y = ops.selective_scan(x.to(dev), dt.to(dev), bias.to(dev), bc.to(dev), a.to(dev), d.to(dev), gate.to(dev), 3, held, rows)
    want, want_state = torch.zeros(total, channels, dtype=torch.float64), start.double()
    size = torch.nn.functional.softplus(dt.double() + bias.double())
    for i in range(len(lens)):
        for r in range(cu[i], cu[i + 1]):
            want_state[i] = torch.exp(size[r][:, None] * a.double()) * want_state[i] + (size[r] * x[r].double())[:, None] * bc[r, :state].double()
            want[r] = ((want_state[i] * bc[r, state:2 * state].double()).sum(-1) + d.double() * x[r].double()) \
                * torch.nn.functional.silu(gate[r, 3:].double())
    # a float32 recurrence of at most 48 tokens: each adds a few ulp of the state's size; y is rounded to bfloat16 once
    scale = want_state.abs().amax()
    assert (held.cpu().double() - want_state).abs().max() <= 48 * 4 * 2 ** -24 * scale
    assert ((y.cpu().double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -14 * want.abs().amax()).all()


@pytest.mark.parametrize("channels,state,lens", [(2400, 16, [3] + [1] * 40), (4096, 16, [2] + [1] * 8), (4100, 9, [17] + [1] * 20), (2400, 32, [2] * 30)])
def test_scan_of_a_few_tokens_among_single_ones(channels, state, lens):
    """Steps that are cheaper token by token."""
    test_scan_matches_64_bits(channels, state, lens)


@pytest.mark.parametrize("channels,state,lens", [(33, 8, [18, 16, 5]), (2400, 16, [18, 33]), (70, 17, [40]), (2400, 16, [3] + [1] * 40)])
def test_scan_with_decays_of_zero(channels, state, lens):
    """An infinite rate: a state that holds the last token alone, also where the tokens do not fill a stage."""
    test_scan_matches_64_bits(channels, state, lens, infinite=True)


@pytest.mark.parametrize("channels,offset,lens,held,bias", [
    (4, 0, [1], 0, True), (12, 4, [9, 2, 8], 0, True), (516, 8, [7, 17], 2, False), (64, 0, [1, 3, 24], 5, True),
    (6, 0, [9], 3, True), (64, 2, [9], 3, True)])
def test_conv_matches_64_bits(channels, offset, lens, held, bias):
    g = torch.Generator().manual_seed(channels + offset)
    rows, seq_lens, cu = step(lens, held)
    total, dev, taps = cu[-1], rows.slots.device, 4
    proj = torch.randn(total, offset + channels + 4, generator=g).to(BF16)
    ring = torch.randn(len(lens), taps, channels, generator=g).to(BF16)
    w, b = torch.randn(channels, taps, generator=g), torch.randn(channels, generator=g)
    got = ops.causal_conv(proj.to(dev), offset, channels, w.to(dev), b.to(dev) if bias else None, ring.to(dev), rows, seq_lens)
    want = torch.zeros(total, channels, dtype=torch.float64)
    for i in range(len(lens)):
        for r in range(cu[i], cu[i + 1]):
            acc = b.double() if bias else torch.zeros(channels, dtype=torch.float64)
            pos = held + r - cu[i]
            for back in range(min(taps - 1, pos) + 1):
                raw = proj[r - back, offset:offset + channels] if back <= r - cu[i] else ring[i, (pos - back) % taps]
                acc = acc + w[:, taps - 1 - back].double() * raw.double()
            want[r] = torch.nn.functional.silu(acc)
    # four products and a silu in float32 (2^-20 of the sums' size), one rounding to bfloat16
    assert ((got.cpu().double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -18 * 16).all()


@pytest.mark.parametrize("rows,heads,size,kind,own_gain", [
    (4096, 1, 128, "silu", False), (1025, 4, 64, "logistic", True), (683, 6, 128, "logistic", True), (2049, 2, 64, "silu", False)])
def test_gated_head_norm_of_many_pairs(rows, heads, size, kind, own_gain):
    g = torch.Generator().manual_seed(rows)
    dev = torch.device("cuda", 0)
    o, gate = torch.randn(rows, heads, size, generator=g), torch.randn(rows, heads * size + 8, generator=g).to(BF16)
    w = torch.randn(heads * size if own_gain else size, generator=g)
    got = ops.gated_head_norm(o.to(dev), gate.to(dev), 4, w.to(dev), 1e-6, heads, size, BF16, kind)
    x, z = o.double(), gate[:, 4:4 + heads * size].double().view(rows, heads, size)
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double().view(-1, size) * (torch.sigmoid(z) if kind == "logistic" else torch.nn.functional.silu(z))
    # float32 throughout and one rounding to bfloat16
    assert ((got.cpu().double().view(rows, heads, size) - want).abs() <= 2 ** -8 * want.abs() + 1e-7).all()


@pytest.mark.parametrize("rows,heads", [(12287, 1), (12288, 1), (768, 16), (1025, 12)])
def test_gated_head_norm_at_the_line_of_the_silu_gate(rows, heads):
    test_gated_head_norm_of_many_pairs(rows, heads, 128, "silu", False)


@pytest.mark.parametrize("gated", [True, False])
def test_linear_attention_of_one_step_and_of_two(gated):
    """Many rows are prepared four entries a thread, few an entry a thread, with the same bits."""
    heads, size, dev = 2, 64, torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(5)
    draw = lambda *s: torch.randn(*s, generator=g, device=dev)
    proj, gate, bias = draw(130, 3 * heads * size).to(BF16), draw(130, heads * size), draw(heads * size)
    results = []
    for cuts in ([0, 130], [0, 65, 130]):
        state, out = torch.zeros(1, heads, size, size, device=dev), []
        for a, b in zip(cuts, cuts[1:]):
            rows, _, _ = step([b - a])
            how = dict(gate=gate[a:b].contiguous(), gate_bias=bias, tau=16.0) if gated else dict(decay=torch.tensor([0.9, 0.99], device=dev), silu_inputs=True)
            out.append(ops.linear_attention(proj[a:b].contiguous(), (0, heads * size, 2 * heads * size), state, rows, heads, size, size, **how))
        results.append((torch.cat(out), state))
    assert all(torch.equal(x, y) for x, y in zip(*results))
