"""Mixtures of experts as products of the chosen experts alone (csrc/moe_grouped.cu), against the same sums in 64 bits."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(shape, seed, std=1.0):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0, std, generator=torch.Generator(device=DEV).manual_seed(seed))


def plain(x, dense, w_up, w_down, ff, shared_ff, glu, gate):
    """All experts over all rows in 64 bits."""
    n = dense.shape[1]
    width = n * ff + shared_ff
    w = torch.cat([dense.double().repeat_interleave(ff, dim=1), torch.ones(x.shape[0], shared_ff, dtype=torch.float64, device=DEV)], dim=1)
    after = torch.ones_like(w)
    if gate is not None:
        after[:, n * ff:] = torch.sigmoid(gate.double())[:, None]
    up = x.double() @ w_up.double().t()
    if glu is None:
        act = 0.5 * up * (1 + torch.erf(up / math.sqrt(2.0))) * w * after
    else:
        limit, shared_limit, alpha, shift, at = glu
        lim = torch.full((width,), float(limit), dtype=torch.float64, device=DEV)
        lim[n * ff:] = shared_limit
        scale = w if at == "input" else torch.ones_like(w)
        g = torch.minimum(up[:, :width] * scale, lim)
        u = torch.maximum(torch.minimum(up[:, width:] * scale, lim), -lim)
        act = g * torch.sigmoid(alpha * g) * (u + shift) * after * (w if at == "output" else (w != 0))
    return act @ w_down.double().t()


SILU = (math.inf, math.inf, 1.0, 0.0, "output")
CLAMPED = (1.5, 2.0, 1.7, 1.0, "input")


def check(rows, hidden, experts, top, ff, shared_ff, glu, gated, logits=None):
    from thing_htn_2026_b200 import ops
    x = rand((rows, hidden), 1).bfloat16()
    width = experts * ff + shared_ff
    w_up = rand(((1 if glu is None else 2) * width, hidden), 2, hidden ** -0.5).bfloat16()
    w_down = rand((hidden, width), 3, ff ** -0.5).bfloat16()
    z = rand((rows, experts + 1), 4) if logits is None else logits
    routing = ops.moe_route(z, experts, 1, 1, top, 1.0, scoring="softmax_chosen")
    err = ops.new_error_word(torch.device(DEV))
    got = ops.grouped_experts(x, routing, w_up, w_down, ff, shared_ff, glu, z if gated else None, experts, err)
    again = ops.grouped_experts(x, routing, w_up, w_down, ff, shared_ff, glu, z if gated else None, experts, err)
    assert int(err.item()) == 0 and torch.equal(got, again)
    want = plain(x, routing.dense, w_up, w_down, ff, shared_ff, glu, z[:, experts] if gated else None)
    # the activations and the result are rounded to bfloat16 once each: 2^-9 / sqrt(3) = 1.1e-3 of either's size, together 1.6e-3
    difference = got.double() - want
    assert float(difference.norm() / want.norm()) < 4e-3
    assert float(difference.abs().max() / want.pow(2).mean().sqrt()) < 0.06
    return x, routing, got, (w_up, w_down, z)


@pytest.mark.parametrize("rows", [1, 2, 31, 33, 127, 128, 129, 255, 256, 257, 511, 513, 1000])
@pytest.mark.parametrize("form", ["silu", "clamped", "gelu"])
def test_rows_around_the_tiles_edges(rows, form):
    check(rows, 256, 8, 2, 128, 128, {"silu": SILU, "clamped": CLAMPED, "gelu": None}[form], form == "clamped")


@pytest.mark.parametrize("hidden, experts, top, ff, shared_ff", [(64, 2, 1, 64, 0), (192, 3, 1, 64, 192), (320, 64, 6, 192, 64),
                                                                 (1024, 5, 2, 320, 0), (2048, 8, 2, 1024, 1024), (128, 256, 8, 64, 64)])
@pytest.mark.parametrize("form", ["silu", "clamped", "gelu"])
def test_sizes(hidden, experts, top, ff, shared_ff, form):
    check(300, hidden, experts, top, ff, shared_ff, {"silu": SILU, "clamped": CLAMPED, "gelu": None}[form], form == "gelu" and shared_ff > 0)


def test_one_expert_takes_all_and_others_nothing():
    z = torch.full((600, 9), -3.0, device=DEV)
    z[:, 5], z[:300, 1], z[300:, 7] = 2.0, 1.0, 1.0
    check(600, 256, 8, 2, 128, 128, SILU, False, z)


def test_a_row_does_not_depend_on_the_others():
    from thing_htn_2026_b200 import ops
    x, routing, got, (w_up, w_down, z) = check(700, 256, 8, 2, 128, 128, SILU, True)
    pick = torch.tensor([699, 3, 256, 511, 17], device=DEV)
    fewer = ops.moe_route(z[pick].contiguous(), 8, 1, 1, 2, 1.0, scoring="softmax_chosen")
    alone = ops.grouped_experts(x[pick].contiguous(), fewer, w_up, w_down, 128, 128, SILU, z[pick].contiguous(), 8)
    assert torch.equal(alone, got[pick])


@pytest.mark.parametrize("form", ["clamped", "gelu"])
def test_a_step_in_pieces_gives_the_same(form, monkeypatch):
    """Scratch that would be larger than the dense form's is taken for some of the rows at a time."""
    from thing_htn_2026_b200 import ops
    glu, hidden, experts, top, ff, shared_ff = {"clamped": CLAMPED, "gelu": None}[form], 512, 8, 4, 64, 64
    x, z = rand((700, hidden), 1).bfloat16(), rand((700, experts + 1), 4)
    width = experts * ff + shared_ff
    w_up, w_down = rand(((2 if glu else 1) * width, hidden), 2, hidden ** -0.5).bfloat16(), rand((hidden, width), 3, ff ** -0.5).bfloat16()
    routing = ops.moe_route(z, experts, 1, 1, top, 1.0, scoring="softmax_chosen")
    whole = ops.grouped_experts(x, routing, w_up, w_down, ff, shared_ff, glu, z, experts)
    calls, inner = [], ops._call
    monkeypatch.setattr(ops, "GROUPED_SCRATCH", 0)
    monkeypatch.setattr(ops, "_call", lambda name, *a: calls.append(name) or inner(name, *a))
    pieces = ops.grouped_experts(x, routing, w_up, w_down, ff, shared_ff, glu, z, experts)
    assert len(calls) == (4 if glu else 6) and torch.equal(whole, pieces)


def test_a_row_that_is_not_a_number_stays_alone():
    from thing_htn_2026_b200 import ops
    x, routing, got, (w_up, w_down, z) = check(300, 256, 8, 2, 128, 0, SILU, False)
    bad, logits = x.clone(), z.clone()
    bad[7] = math.nan
    logits[9, :8] = math.nan
    logits[11, 2:8] = math.nan           # fewer numbers than choices: an expert stands twice
    logits[11, 0], logits[11, 1] = math.nan, 1.0
    r = ops.moe_route(logits, 8, 1, 1, 2, 1.0, scoring="softmax_chosen")
    y = ops.grouped_experts(bad, r, w_up, w_down, 128, 0, SILU)
    assert torch.isnan(y[7]).all() and torch.isnan(y[9]).all()
    dense = ops.linear(ops.routed_clamped_glu(ops.linear(bad, w_up), r, 128, 0, math.inf, math.inf, 1.0, None, 0, "output", 0.0), w_down)
    close = (y[11].double() - dense[11].double()).norm() <= 0.01 * dense[11].double().norm()
    assert bool(close) and torch.isfinite(y[11]).all()
    others = [i for i in range(300) if i not in (7, 9, 11)]
    assert torch.equal(y[others], got[others])


def test_sizes_and_operands_that_are_refused():
    from thing_htn_2026_b200 import ops
    for hidden, experts, ff, shared in ((96, 8, 128, 0), (128, 8, 96, 0), (128, 8, 128, 32), (128, 257, 64, 0)):
        assert not ops.lib().thn_moe_grouped_supported(hidden, experts, ff, shared)
    x = rand((8, 96), 1).bfloat16()
    routing = ops.moe_route(rand((8, 8), 2), 8, 1, 1, 2, 1.0, scoring="softmax_chosen")
    with pytest.raises(ops.KernelError):
        ops.grouped_experts(x, routing, rand((2048, 96), 3).bfloat16(), rand((96, 1024), 4).bfloat16(), 128, 0, SILU)
    with pytest.raises(ops.KernelError):
        ops.grouped_experts(x, routing, rand((2048, 96), 3).bfloat16(), rand((96, 1000), 4).bfloat16(), 128, 0, SILU)


@pytest.mark.parametrize("form, shared_ff", [("silu", 128), ("gelu", 0)])
def test_a_wait_that_runs_out_sets_its_bit_and_the_kernels_return(form, shared_ff, monkeypatch):
    """With no operand loaded every wait of the products ends after 20 ms, the bit is set, and the next launch is right again."""
    from thing_htn_2026_b200 import ops
    glu = {"silu": SILU, "gelu": None}[form]
    x, width = rand((300, 256), 1).bfloat16(), 8 * 128 + shared_ff
    w_up, w_down = rand(((2 if glu else 1) * width, 256), 2).bfloat16(), rand((256, width), 3).bfloat16()
    routing = ops.moe_route(rand((300, 8), 4), 8, 1, 1, 2, 1.0, scoring="softmax_chosen")
    err = ops.new_error_word(torch.device(DEV))
    with monkeypatch.context() as patch:
        patch.setattr(ops, "GROUPED_SKIP_LOADS", 1)
        ops.grouped_experts(x, routing, w_up, w_down, 128, shared_ff, glu, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == ops.ERR_WAIT_TIMEOUT
    check(300, 256, 8, 2, 128, shared_ff, glu, False)


def test_without_an_error_word_a_wait_that_runs_out_raises(monkeypatch):
    from thing_htn_2026_b200 import ops
    x, w_up, w_down = rand((300, 256), 1).bfloat16(), rand((2048, 256), 2).bfloat16(), rand((256, 1024), 3).bfloat16()
    routing = ops.moe_route(rand((300, 8), 4), 8, 1, 1, 2, 1.0, scoring="softmax_chosen")
    monkeypatch.setattr(ops, "GROUPED_SKIP_LOADS", 1)
    with pytest.raises(ops.KernelError, match="bounded wait"):
        ops.grouped_experts(x, routing, w_up, w_down, 128, 0, SILU)
