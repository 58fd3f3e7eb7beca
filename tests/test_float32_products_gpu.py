"""The float32 product on the tensor cores against 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m, n, k", [(1, 1, 4), (64, 128, 64), (65, 129, 68), (127, 1000, 100), (300, 130, 260), (129, 257, 1028)])
@pytest.mark.parametrize("box", [64, 128])
def test_any_sizes(m, n, k, box):
    """Tiles and steps of 64 columns cut anywhere, operands inside wider rows, a bias, an output inside a wider one."""
    torch.manual_seed(k)
    values, weight = torch.randn(m, k + 4, device="cuda")[:, :k], torch.randn(n, k + 8, device="cuda")[:, :k]
    bias = torch.randn(n, device="cuda")
    out = torch.full((m, n + 3), 7.0, device="cuda")
    kernels.gemm_f32_tc(values, weight, bias, out[:, :n], box)
    wanted = values.double() @ weight.double().T + bias.double()
    magnitude = values.double().abs() @ weight.double().abs().T + bias.double().abs()
    # 24 additions of the tensor core to a step's accumulator, each cut off at 2^-23 of it, what the pieces leave out (2^-24), and a rounding for every step.
    assert bool(((out[:, :n].double() - wanted).abs() <= (24 * 2 + 1 + k / 64 + 2) * 2.0 ** -24 * magnitude).all()) and bool((out[:, n:] == 7.0).all())
    assert kernels.build.load_library("gemm_f32_tc.cu").tau_gemm_f32_tc_status() == 0


def test_values_that_have_no_pieces():
    """Infinities, a NaN, a number next to the largest, small ones: as the plain product has them."""
    torch.manual_seed(3)
    values, weight = torch.randn(70, 256, device="cuda"), torch.randn(130, 256, device="cuda") * 0.02
    values[0, 3], values[1, 5], values[2] = float("inf"), float("nan"), 1e-33
    values[4, 7] = 3.4e38
    weight[9, 200] = float("-inf")
    found, plain = torch.empty(70, 130, device="cuda"), torch.empty(70, 130, device="cuda")
    kernels.gemm_f32_tc(values, weight, None, found)
    kernels.gemm_simt(values, weight, None, plain)
    assert torch.equal(found.isnan(), plain.isnan()) and torch.equal(found.isinf(), plain.isinf()) and torch.equal(found[plain.isinf()] > 0, plain[plain.isinf()] > 0)
    finite = plain.isfinite()
    error = (found - plain).abs()[finite] / (values.abs().nan_to_num(0.0, 0.0, 0.0) @ weight.abs().nan_to_num(0.0, 0.0, 0.0).T)[finite]
    assert float(error.max()) < 300 * 2.0 ** -24


@pytest.mark.parametrize("m, n, k, splits", [(1, 1, 128, 2), (65, 129, 196, 3), (129, 257, 1028, 8), (127, 1000, 520, 7)])
@pytest.mark.parametrize("box", [64, 128])
def test_ranges_of_a_tile(m, n, k, splits, box):
    """Steps that do not share out evenly, tiles of fewer tokens than ranges, a value without pieces in one range."""
    torch.manual_seed(k)
    values, weight, bias = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda"), torch.randn(n, device="cuda")
    out = torch.full((m, n + 3), 7.0, device="cuda")
    kernels.gemm_f32_tc(values, weight, bias, out[:, :n], box, splits)
    wanted = values.double() @ weight.double().T + bias.double()
    magnitude = values.double().abs() @ weight.double().abs().T + bias.double().abs()
    # As above; a sum of ranges has fewer roundings than steps.
    assert bool(((out[:, :n].double() - wanted).abs() <= (24 * 2 + 1 + k / 64 + 2) * 2.0 ** -24 * magnitude).all()) and bool((out[:, n:] == 7.0).all())
    values[m - 1, k - 1] = 3.4e38
    kernels.gemm_f32_tc(values, weight, bias, out[:, :n], box, splits)
    plain = torch.empty(m, n, device="cuda")
    kernels.gemm_simt(values, weight, bias, plain)
    assert torch.equal(out[:, :n].isinf(), plain.isinf()) and bool(out[:, :n].isnan().eq(plain.isnan()).all())
    assert kernels.build.load_library("gemm_f32_tc.cu").tau_gemm_f32_tc_status() == 0
