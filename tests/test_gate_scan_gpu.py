"""The gates' scan over runs of more chunks than it has lanes, against 64-bit."""
import pytest
import torch

from test_recurrence_gpu import case, exact, off, walk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs, forget", [([2048], 3.0), ([2049, 64, 71], 3.0), ([100, 2200], -4.0)])
def test_lanes_with_several_chunks(runs, forget):
    """A chunk to each lane, one chunk more, lanes without one; gates that forget at once and hardly at all."""
    sizes = dict(heads=3, dim=16, vdim=15, exponential=True, silu=False)
    inputs = case(runs, seed=len(runs), forget=forget, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    found, found_state = walk(*inputs, **sizes, longest=max(runs), shortest=min(runs))
    assert off(found, wanted) < 2e-6 and off(found_state, wanted_state) < 2e-6      # 32-bit sums over a chunk and its pieces
