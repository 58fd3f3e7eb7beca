"""The router of prompts against 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens, width, experts, top, groups, keep, softmax", [(200, 32, 7, 2, 1, 1, False), (208, 2048, 64, 6, 1, 1, False), (223, 288, 65, 1, 1, 1, True),
                                                                               (1001, 512, 160, 8, 8, 3, False)])
def test_router_of_prompts(dtype, tokens, width, experts, top, groups, keep, softmax, tile=-1):
    """Around 16 tokens and 64 experts of a block, fewer chunks of columns than warps, groups, both scores: the weights of what 64 bits choose."""
    torch.manual_seed(width)
    hidden = torch.randn(tokens, width, device="cuda").to(dtype)
    router, bias, correction, gate = torch.randn(experts, width, device="cuda") * width ** -0.5, torch.randn(experts, device="cuda") * 0.1, torch.randn(experts, device="cuda") * 0.1, torch.randn(width, device="cuda") * 0.1
    chosen, weights, shared = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda"), torch.empty(tokens, device="cuda")
    options = {} if groups == 1 else {"groups": groups, "keep": keep}
    kernels.moe_route(hidden, router, correction, gate, chosen, weights, shared, top, softmax, False, bias, tile=tile, **options)
    z = hidden.double() @ router.double().T + bias.double()
    scores = torch.softmax(z, 1) if softmax else torch.sigmoid(z)
    picked = scores.gather(1, chosen.long())
    assert float((weights.double() - picked).abs().max()) < 2e-6
    choice = scores + correction.double()
    if groups > 1:
        ranks = choice.view(tokens, groups, -1).topk(2, dim=2).values.sum(2)
        kept = torch.zeros_like(ranks, dtype=torch.bool).scatter_(1, ranks.topk(keep, dim=1).indices, True)
        choice = choice.masked_fill(~kept.repeat_interleave(experts // groups, 1), float("-inf"))
    best = choice.topk(top, dim=1).values
    mine = choice.gather(1, chosen.long()).sort(dim=1, descending=True).values
    assert float((best - mine).abs().max()) < 2e-6      # another expert only where the two are as good
    assert bool((chosen.sort(1).values.diff(dim=1) > 0).all()) and float((shared.double() - torch.sigmoid(hidden.double() @ gate.double())).abs().max()) < 2e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens, width, experts, top, groups, keep, softmax", [(200, 32, 7, 2, 1, 1, False), (208, 2048, 64, 6, 1, 1, False), (223, 288, 65, 1, 1, 1, True),
                                                                               (17, 512, 160, 8, 8, 3, False), (1, 96, 32, 3, 1, 1, False)])
@pytest.mark.parametrize("tile", [0, 1])
def test_both_kernels_of_prompts(dtype, tokens, width, experts, top, groups, keep, softmax, tile):
    """Whatever the rule between them picks: the tiles, and token by token."""
    test_router_of_prompts(dtype, tokens, width, experts, top, groups, keep, softmax, tile)


@pytest.mark.parametrize("tokens, experts, width, narrow, tiles", [(300, 8, 4096, True, False), (2048, 8, 4096, True, False), (296, 64, 2048, True, False), (297, 64, 1024, True, True),
                                                                  (591, 64, 2048, False, False), (592, 64, 2048, False, True), (999, 64, 1024, False, False), (999, 32, 2048, True, False),
                                                                  (1000, 32, 2048, True, True), (2048, 64, 256, True, False)])
def test_which_kernel_scores_a_router(tokens, experts, width, narrow, tiles):
    """At the border between them: the bits of the weights tell the tiles' sums from the others'."""
    torch.manual_seed(experts)
    hidden = torch.randn(tokens, width, device="cuda").to(torch.bfloat16 if narrow else torch.float32)
    router = torch.randn(experts, width, device="cuda") * width ** -0.5
    results = []
    for tile in (-1, 0, 1):
        chosen, weights = torch.empty(tokens, 2, dtype=torch.int32, device="cuda"), torch.empty(tokens, 2, device="cuda")
        kernels.moe_route(hidden, router, None, None, chosen, weights, None, 2, tile=tile)
        results.append(weights)
    assert not torch.equal(results[1], results[2]) and torch.equal(results[0], results[2 if tiles else 1])
