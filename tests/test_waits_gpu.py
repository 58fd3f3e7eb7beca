"""Waits for bulk copies that never come: the kernels end within the limit, say so, and leave the state as it was."""
import pytest
import torch

import test_delta_rule_gpu as delta
import test_recurrence_gpu as recurrence
from tau_rs_b200.csrc import build, kernels

pytestmark = pytest.mark.gpu

LOST = ("TAU_LOST_COPIES", "TAU_WAIT_LIMIT_NS=1000000ull")      # no copy is asked for; a wait gives up after a millisecond


@pytest.fixture
def lost_copies(monkeypatch):
    """Every library that is loaded meanwhile is the one whose copies are lost; only its own status is raised."""
    monkeypatch.setattr(build, "load_library", lambda source, defines=(), load=build.load_library: load(source, (*defines, *LOST)))


@pytest.mark.parametrize("silu", [False, True])
def test_matrix_memory(lost_copies, silu):
    sizes = dict(heads=2, dim=64, vdim=40, exponential=not silu, silu=silu)
    inputs = recurrence.case([300, 70], seed=4, **sizes)
    _, state = recurrence.walk(*inputs, **sizes, longest=300)
    assert kernels.recurrence_status(64) == 1 and torch.equal(state, inputs[3])


def test_delta_rule(lost_copies):
    sizes = dict(heads=2, key_heads=1, dim=64, vdim=40)
    inputs = delta.case([300, 70], seed=9, **sizes)
    _, state = delta.walk(*inputs, **sizes, longest=300)
    assert kernels.delta_rule_status(64) == 1 and torch.equal(state, inputs[3])


def test_prefill_from_swizzled_pages(lost_copies):
    pages = [torch.zeros(4, 2, 64, 192, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    queries, bounds = torch.zeros(200, 384, device="cuda", dtype=torch.bfloat16), torch.tensor([0, 200], dtype=torch.int32).cuda()
    out = torch.full_like(queries, 7.0)
    kernels.attention_prefill(queries, *pages, out, bounds, torch.zeros(1, dtype=torch.int32).cuda(), torch.arange(4, dtype=torch.int32).cuda()[None], 2, 2, 192,
                              192 ** -0.5, 0, swizzled=True)
    assert kernels.attention_prefill_status(192) == 1 and bool((out == 7.0).all())      # every block meets a whole page
