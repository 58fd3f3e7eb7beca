"""Routed experts whose weights are streamed once, against 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts, width, inner, top, tokens", [(1, 256, 256, 1, 1), (3, 272, 256, 2, 33), (5, 1024, 264 + 8, 3, 9), (70, 256, 720, 6, 40), (4, 512, 256, 4, 100)])
@pytest.mark.parametrize("identity, limit, on_input", [(0, 0.0, False), (2, 0.0, False), (0, 1.5, True)])
def test_streamed_experts(experts, width, inner, top, tokens, identity, limit, on_input):
    """Depths of fewer and more chunks than warps, ragged ones, experts that nobody and that everybody chose (more pairs than one product holds), identity
    experts, a clamped gate, weights on the input."""
    torch.manual_seed(experts + width)
    gate_up = (torch.randn(experts, 2 * inner, width, device="cuda") * width ** -0.5).to(torch.bfloat16)
    down = (torch.randn(experts, width, inner, device="cuda") * inner ** -0.5).to(torch.bfloat16)
    hidden, weights = torch.randn(tokens, width, device="cuda").to(torch.bfloat16), torch.rand(tokens, top, device="cuda")
    chosen = torch.stack([torch.randperm(max(experts + identity, top), device="cuda")[:top] % (experts + identity) for _ in range(tokens)]).to(torch.int32)
    inner_out = torch.full((tokens, top, inner), 7.0, device="cuda", dtype=torch.bfloat16)
    rows, out = torch.full((tokens * top, width), float("nan"), device="cuda"), torch.empty(tokens, width, device="cuda")
    kernels.moe_stream(hidden, gate_up, down, chosen, inner_out, rows, weights if on_input else None, limit)
    kernels.moe_combine(rows, None, None if on_input else weights, None, None, out, **({"chosen": chosen, "hidden": hidden, "real_experts": experts} if identity else {}))
    again = torch.empty_like(inner_out)
    kernels.moe_gate_up(hidden, gate_up, chosen, again, 8, weights if on_input else None, limit)
    real = (chosen < experts)[:, :, None].expand_as(inner_out)
    assert bool((inner_out[~real] == 7.0).all())
    # The same sums in another order before the one rounding: a step of bfloat16 here and there.
    assert bool(((inner_out.float() - again.float()).abs()[real] <= 2.0 ** -7 * again.float().abs()[real] + 1e-6).all())
    x = inner_out.double()
    wanted = torch.zeros(tokens, width, device="cuda", dtype=torch.float64)
    for token in range(tokens):
        for place in range(top):
            expert, weight = int(chosen[token, place]), 1.0 if on_input else weights[token, place].double()
            wanted[token] += weight * (hidden[token].double() if expert >= experts else down[expert].double() @ x[token, place])
    assert float((out.double() - wanted).abs().max() / wanted.abs().max()) < 1e-5      # 32-bit sums


@pytest.mark.parametrize("limit", [0.0, 1.5])
def test_infinities_come_out_as_from_the_kernels_of_fewer_pairs(limit):
    """An infinite activation and infinite weights in the first, a middle and the last span of columns: infinite sums stay infinite (a clamped gate makes them finite)."""
    torch.manual_seed(3)
    experts, width, inner, tokens = 3, 640, 528, 40
    gate_up = (torch.randn(experts, 2 * inner, width, device="cuda") * width ** -0.5).to(torch.bfloat16)
    down = (torch.randn(experts, width, inner, device="cuda") * inner ** -0.5).to(torch.bfloat16)
    hidden = torch.randn(tokens, width, device="cuda").to(torch.bfloat16)
    chosen = (torch.arange(tokens, device="cuda") % experts).to(torch.int32)[:, None]
    hidden[4, 300] = float("inf")
    gate_up[0, 16 * 5 + 8, 2], gate_up[1, 16 * 20 + 9, 630], gate_up[2, 16 * 7 + 3, 200] = float("inf"), float("-inf"), float("inf")      # two up rows and a gate row
    found, wanted = (torch.empty(tokens, 1, inner, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    rows, out = torch.empty(tokens, width, device="cuda"), torch.empty(tokens, width, device="cuda")
    kernels.moe_stream(hidden, gate_up, down, chosen, found, rows, None, limit)
    kernels.moe_gate_up(hidden, gate_up, chosen, wanted, 8, None, limit)
    kernels.moe_down(found, down, chosen, torch.ones(tokens, 1, device="cuda"), None, None, out)
    assert bool(torch.isinf(found).any() if limit == 0.0 else torch.isfinite(found[:2]).all())
    for mine, theirs, tolerance in ((found, wanted, 2.0 ** -7), (rows, out, 1e-5)):      # one bfloat16 rounding; 32-bit sums
        finite = torch.isfinite(theirs)
        assert torch.equal(torch.nan_to_num(mine[~finite], nan=7.0).float(), torch.nan_to_num(theirs[~finite], nan=7.0).float())
        assert bool(((mine - theirs).float().abs()[finite] <= tolerance * theirs.float().abs()[finite] + 1e-5).all())
