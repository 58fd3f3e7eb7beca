"""One launch for the products of all experts against a product per group in 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, features, depth", [([1], 16, 8), ([0, 5, 0, 0, 300, 256, 257, 0], 272, 136), ([0] * 40 + [7] + [0] * 30, 64, 64), ([130] * 33, 528, 72), ([1000, 1, 1], 1024, 520)])
@pytest.mark.parametrize("gated, out_dtype", [(False, torch.float32), (False, torch.bfloat16), (True, torch.bfloat16)])
def test_groups_of_any_size(sizes, features, depth, gated, out_dtype):
    """Empty groups at the ends and in the middle, groups around a tile of 256 rows, features that cut a tile of 256, rows behind the last group."""
    torch.manual_seed(features)
    rows, groups = sum(sizes) + 9, len(sizes)
    x = torch.randn(rows, depth + 8, device="cuda").to(torch.bfloat16)[:, :depth]
    weights = (torch.randn(groups, features, depth, device="cuda") * depth ** -0.5).to(torch.bfloat16)
    bounds = [0] + torch.tensor(sizes).cumsum(0).tolist()
    out = torch.full((rows, features // 2 if gated else features), 7.0, device="cuda", dtype=out_dtype)
    kernels.gemm_tc_grouped(x, weights, out, torch.tensor(bounds, dtype=torch.int32).cuda(), gated=gated)
    assert bool((out[bounds[-1] :] == 7.0).all())      # rows of no group are left alone
    for group in [group for group in range(groups) if sizes[group]]:
        mine = x[bounds[group] : bounds[group + 1]].double()
        wanted = mine @ weights[group].double().T
        if gated:
            pairs = wanted.view(-1, features // 16, 2, 8)
            gate, up = (pairs[:, :, i].reshape(mine.shape[0], -1) for i in (0, 1))
            wanted = torch.nn.functional.silu(gate) * up
        found = out[bounds[group] : bounds[group + 1]].double()
        bound = 2.0 ** -6 if gated else 2.0 ** -8 if out_dtype == torch.bfloat16 else 1e-5      # two roundings before the activation and one behind it; one; 32-bit sums
        assert bool(((found - wanted).abs() <= bound * (wanted.abs() + 0.3)).all()), group
    assert kernels.gemm_tc_status() == 0


@pytest.mark.parametrize("sizes, features, depth", [([5, 0, 300, 256, 1, 0], 272, 136), ([0] * 520 + [9, 0, 17], 32, 16)])
@pytest.mark.parametrize("gated, out_dtype", [(False, torch.float32), (True, torch.bfloat16)])
def test_a_launch_for_each_group_on_streams_of_their_own(sizes, features, depth, gated, out_dtype):
    """What layers of more experts than one launch numbers run: bounds on the host, four streams between the caller's kernels."""
    torch.manual_seed(depth)
    rows, groups = sum(sizes) + 3, len(sizes)
    x = torch.randn(rows, depth, device="cuda").to(torch.bfloat16)
    weights = (torch.randn(groups, features, depth, device="cuda") * depth ** -0.5).to(torch.bfloat16)
    bounds = [0] + torch.tensor(sizes).cumsum(0).tolist()
    out = torch.full((rows, features // 2 if gated else features), 7.0, device="cuda", dtype=out_dtype)
    kernels.gemm_tc_groups(x, weights, out, bounds, gated=gated)
    found = out.clone()      # behind the products, on the caller's stream
    assert bool((found[bounds[-1] :] == 7.0).all())
    for group in [group for group in range(groups) if sizes[group]]:
        mine = x[bounds[group] : bounds[group + 1]].double()
        wanted = mine @ weights[group].double().T
        if gated:
            pairs = wanted.view(-1, features // 16, 2, 8)
            gate, up = (pairs[:, :, i].reshape(mine.shape[0], -1) for i in (0, 1))
            wanted = torch.nn.functional.silu(gate) * up
        bound = 2.0 ** -6 if gated else 1e-5      # as above
        assert bool(((found[bounds[group] : bounds[group + 1]].double() - wanted).abs() <= bound * (wanted.abs() + 0.3)).all()), group
    assert kernels.gemm_tc_status() == 0


def test_a_layer_of_more_experts_than_one_launch_numbers(monkeypatch):
    """513 experts through a prompt, grouped with a launch each, against the kernels of few tokens."""
    from types import SimpleNamespace

    from tau_rs_b200.config import RoutedExpertsSpec
    from tau_rs_b200.parts import routed_experts

    torch.manual_seed(5)
    experts, width, inner, tokens = kernels.GROUPED_MOST + 1, 32, 16, 300
    part = routed_experts.RoutedExperts(RoutedExpertsSpec(hidden=width, intermediate=inner, experts=experts, top=3), "m", torch.bfloat16, "cuda")
    for name, spec in part.tensor_specs().items():
        part.assign(name, (torch.randn(*spec.shape, device="cuda") * 0.3).to(torch.bfloat16 if spec.role == "matrix" else torch.float32))
    part.finalize_weights()
    hidden = torch.randn(tokens, width, device="cuda").to(torch.bfloat16)
    calls = []
    monkeypatch.setattr(kernels, "gemm_tc_groups", lambda *a, run=kernels.gemm_tc_groups, **k: calls.append(1) or run(*a, **k))
    assert tokens * 3 >= routed_experts.GROUPED_FROM
    grouped, streamed = (part.forward(hidden, SimpleNamespace(all_single=single)) for single in (False, True))
    assert len(calls) == 2 and float((grouped - streamed).norm() / streamed.norm()) < 1e-2      # roundings of the products and of their inner values to bfloat16
