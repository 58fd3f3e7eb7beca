"""Waits for bulk copies and operands that never come: the kernels end within the limit, say so, and leave the state or the output as it was."""
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


@pytest.fixture
def lost_rank(monkeypatch):
    """Every library that is loaded meanwhile is one in which nothing arrives in the second block of each cluster."""
    monkeypatch.setattr(build, "load_library", lambda source, defines=(), load=build.load_library: load(source, (*defines, *LOST, "TAU_LOST_RANK=1")))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_whose_ranges_meet_in_a_cluster(lost_rank, dtype):
    """Four ranges of K, one of which gives up: no block of the cluster stores a sum that lacks it."""
    x, w = torch.ones(64, 2048, device="cuda", dtype=dtype), torch.ones(256, 2048, device="cuda", dtype=dtype)
    out = torch.full((64, 256), 7.0, device="cuda", dtype=dtype)
    single = dtype == torch.float32
    (kernels.gemm_f32_tc if single else kernels.gemm_tc)(x, w, None, out, splits=4)
    library = build.load_library("gemm_f32_tc.cu" if single else "gemm_tc.cu")
    assert (library.tau_gemm_f32_tc_status if single else library.tau_gemm_tc_status)() == 1 and bool((out == 7.0).all())


@pytest.mark.parametrize("head_dim", [64, 128])
def test_float32_attention_whose_ranges_meet_in_a_cluster(lost_rank, head_dim):
    """Both ranges see a page in every tile of queries."""
    pages = torch.zeros(5, 2, 64, head_dim, device="cuda")
    queries, bounds = torch.zeros(300, 2 * head_dim, device="cuda"), torch.tensor([0, 300], dtype=torch.int32).cuda()
    out = torch.full_like(queries, 7.0)
    kernels.attention_f32_tc(queries, pages, pages, out, bounds, torch.zeros(1, dtype=torch.int32).cuda(), torch.arange(5, dtype=torch.int32).cuda()[None], 2, 2, head_dim,
                             head_dim ** -0.5, 0, ranges=2)
    assert build.load_library("attention_f32_tc.cu").tau_attention_f32_tc_status() == 1 and bool((out == 7.0).all())


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
