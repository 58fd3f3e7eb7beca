"""Runs last: no bounded wait of any library that the tests before used has run out."""
import pytest

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


def test_no_wait_ran_out():
    assert [name for name in kernels.waits_that_ran_out() if "TAU_LOST_COPIES" not in name] == []
