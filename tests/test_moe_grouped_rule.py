"""Which mixtures of experts are multiplied in groups (``ops.experts_in_groups``): a rule of sizes, type and alignment."""

import pytest
import torch


def test_rule():
    from thing_htn_2026_b200 import ops
    x = torch.empty(2048, 2048, dtype=torch.bfloat16)
    assert ops.experts_in_groups(x, 8, 2, 1024, 1024, True) and ops.experts_in_groups(x, 8, 2, 1024, 0, False)
    assert not ops.experts_in_groups(x[:512], 8, 2, 1024, 1024, True)             # 39e9 operations saved
    assert ops.experts_in_groups(x[:1024], 8, 2, 1024, 1024, True) and not ops.experts_in_groups(x[:1024], 8, 2, 1024, 1024, False)
    assert ops.experts_in_groups(x[:256], 64, 6, 512, 512, True) and not ops.experts_in_groups(x[:255], 64, 6, 512, 512, True)
    assert not ops.experts_in_groups(x, 8, 8, 1024, 1024, True)                   # nothing is left out
    assert not ops.experts_in_groups(x.float(), 8, 2, 1024, 1024, True)
    assert not ops.experts_in_groups(x.view(-1)[1:1 + 2047 * 2048].view(2047, 2048), 8, 2, 1024, 1024, True)      # 2-byte aligned
    for ff, shared in ((1000, 0), (1024, 1000), (1056, 1024)):
        assert not ops.experts_in_groups(x, 8, 2, ff, shared, True)
    assert not ops.experts_in_groups(torch.empty(2048, 2056, dtype=torch.bfloat16), 8, 2, 1024, 1024, True)
    assert not ops.experts_in_groups(x, 512, 2, 64, 0, True)


# sizes, gated, rows: us in the dense form, in groups (B200, cold weights)
MEASURED = [((2048, 8, 2, 1024, 1024), True, 640, 70, 77), ((2048, 8, 2, 1024, 1024), True, 896, 95, 76), ((2048, 8, 2, 1024, 1024), False, 1024, 73, 73),
            ((2048, 8, 2, 1024, 1024), False, 2048, 126, 104), ((4096, 8, 2, 2048, 2048), True, 288, 126, 145), ((4096, 8, 2, 2048, 2048), True, 384, 149, 153),
            ((4096, 8, 2, 2048, 2048), True, 448, 177, 150), ((4096, 8, 2, 2048, 2048), False, 512, 128, 131), ((4096, 8, 2, 2048, 2048), False, 768, 178, 159),
            ((2048, 64, 6, 512, 512), True, 192, 115, 126), ((2048, 64, 6, 512, 512), True, 256, 135, 125), ((2048, 64, 6, 512, 512), False, 288, 109, 113),
            ((2048, 16, 4, 1024, 0), True, 448, 98, 74), ((4096, 64, 8, 256, 0), True, 256, 119, 138), ((4096, 64, 8, 256, 0), True, 384, 140, 153),
            ((4096, 64, 8, 256, 0), True, 640, 210, 180), ((4096, 16, 1, 2048, 0), True, 256, 209, 181), ((2048, 128, 8, 256, 256), True, 288, 130, 144),
            ((2048, 128, 8, 256, 256), True, 448, 179, 153), ((7168, 32, 8, 512, 512), True, 352, 219, 267), ((7168, 32, 8, 512, 512), True, 576, 341, 273),
            ((4096, 8, 2, 2048, 0), True, 256, 112, 101), ((2048, 16, 4, 1024, 0), True, 416, 91, 71), ((7168, 32, 8, 512, 0), True, 320, 201, 222),
            ((4096, 16, 2, 1024, 1024), True, 288, 116, 125), ((4096, 16, 2, 1024, 1024), True, 352, 137, 120), ((4096, 16, 2, 2048, 0), False, 256, 145, 129)]


@pytest.mark.parametrize("sizes,gated,rows,dense,grouped", MEASURED)
def test_the_faster_form_is_taken(sizes, gated, rows, dense, grouped):
    from thing_htn_2026_b200 import ops
    hidden, n_experts, top, ff, shared_ff = sizes
    taken = grouped if ops.experts_in_groups(torch.empty(rows, hidden, dtype=torch.bfloat16), n_experts, top, ff, shared_ff, gated) else dense
    assert taken <= 1.03 * min(dense, grouped)          # (nearer, the grouped form is taken: it rounds less)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["routed_glu_experts", "routed_clamped_experts", "routed_experts"])
def test_a_part_gives_the_same_on_both_sides(kind, monkeypatch):
    from thing_htn_2026_b200 import ops, parts
    from thing_htn_2026_b200.config.base import PartSpec
    from types import SimpleNamespace
    hidden, n, ff = 512, 8, 256
    params = {"hidden_size": hidden, "n_experts": n, "expert_ff": ff, "top": 2, "shared_ff": 192}
    if kind == "routed_clamped_experts":
        params.update(limit=1.5, slope=1.7)
    g = torch.Generator(device="cuda").manual_seed(3)
    cls = parts.part_class("ffn", kind)
    names = ["router", "shared_gate_proj", "shared_up", "shared_down", "shared_gate"] + [f"{m}.{e}" for m in ("gate", "up", "down") for e in range(n)]
    spec = PartSpec(kind, params, {name: name for name in names})
    tensors = {t.name: torch.empty(t.shape, dtype=torch.bfloat16, device="cuda").normal_(0, t.shape[1] ** -0.5, generator=g)
               for t in cls.tensor_specs(spec)}
    part = cls(spec, parts.Runtime(torch.bfloat16, torch.device("cuda"), tensors))
    ctx = SimpleNamespace(err=ops.new_error_word(torch.device("cuda")))
    x = torch.empty(700, hidden, dtype=torch.bfloat16, device="cuda").normal_(0, 1, generator=g)
    with torch.inference_mode():
        dense = part.forward(x, ctx)
        monkeypatch.setattr(ops, "GROUPED_MIN_SAVED", {True: 0.0, False: 0.0})
        calls = []
        inner = ops.grouped_experts
        monkeypatch.setattr(ops, "grouped_experts", lambda *a, **k: calls.append(1) or inner(*a, **k))
        grouped = part.forward(x, ctx)
        assert len(calls) == 1
        part.forward(x, SimpleNamespace(err=None))          # no word for the kernels' waits: the dense form
        short = part.forward(x[:300], ctx)                   # the same rows in a step of fewer: the dense form
    assert len(calls) == 1 and int(ctx.err.item()) == 0
    # each side rounds the activations and the result (1.6e-3 from 64 bits), the dense one gates and ups too (1.6e-3 more)
    assert float((dense.double() - grouped.double()).norm() / dense.double().norm()) < 8e-3
    assert float((short.double() - grouped[:300].double()).norm() / short.double().norm()) < 8e-3
