"""The limit of the kernels' waits, on barriers that nothing completes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_wait_on_several_barriers_has_the_limit_of_one(lib):
    """All wait at the same time.  A limit for each barrier, one after the other, made it two and three times as long."""
    from fa2_custom_mask import _lib
    report = torch.full((6,), -1, dtype=torch.int32, device="cuda")
    assert lib.bsa_selftest_wait_limits(_lib.ptr(report), _lib.stream_ptr(report.device)) == 0
    one, ms_one, two, ms_two, three, ms_three = report.cpu().tolist()
    assert one == two == three == 0
    assert 1000 <= ms_one <= 10000
    assert 0.7 * ms_one <= ms_two <= 1.4 * ms_one and 0.7 * ms_one <= ms_three <= 1.4 * ms_one
    assert lib.bsa_selftest_wait_limits(None, None) == -4
