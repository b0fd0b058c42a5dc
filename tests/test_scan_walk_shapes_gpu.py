"""The selective scan's walk on prompts of 64 tokens and more (eight warps beside the four that walk) and on shorter ones (four), for states
of every size class and few and many channels, against the same in 64 bits."""

import pytest
import torch

from test_scan_kernels_gpu import BF16, step
from thing_htn_2026_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,state,lens", [
    (33, 8, [70, 64]), (40, 5, [129]), (33, 8, [30, 20]), (100, 16, [65]), (61, 9, [64, 97, 31]), (4800, 16, [64]), (2400, 12, [70, 80]), (2400, 16, [20, 18, 19]),
    (70, 17, [65]), (40, 32, [80, 64]), (70, 30, [20, 40])])
def test_matches_64_bits(channels, state, lens):
    g = torch.Generator(device="cuda").manual_seed(channels + state)
    rows, _, cu = step(lens)
    total = cu[-1]
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda")      # noqa: E731
    x, bc, gate = draw(total, channels).to(BF16), draw(total, 2 * state).to(BF16), draw(total, channels).to(BF16)
    dt, bias, d, start = draw(total, channels) * 2, draw(channels) * 0.1, draw(channels), draw(len(lens), channels, state)
    a, held = -torch.exp(draw(channels, state)), start.clone()
    y = ops.selective_scan(x, dt, bias, bc, a, d, gate, 0, held, rows)
    size, want, S = torch.nn.functional.softplus(dt.double() + bias.double()), torch.zeros(total, channels, dtype=torch.float64, device="cuda"), start.double()
    for i in range(len(lens)):
        for r in range(cu[i], cu[i + 1]):
            S[i] = torch.exp(size[r][:, None] * a.double()) * S[i] + (size[r] * x[r].double())[:, None] * bc[r, :state].double()
            want[r] = ((S[i] * bc[r, state:].double()).sum(-1) + d.double() * x[r].double()) * torch.nn.functional.silu(gate[r].double())
    # each token adds a few ulp of the state's size; y is rounded to bfloat16 once
    assert (held.double() - S).abs().max() <= max(lens) * 4 * 2 ** -24 * S.abs().amax()
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -14 * want.abs().amax()).all()
