"""The kernels' roles share out the registers that a block is launched with: a kernel that was built with another number
is refused on the host, since the wait for registers that are not there has no limit."""
import pytest

pytestmark = pytest.mark.gpu


def test_another_number_of_registers_is_refused(lib):
    assert lib.bsa_selftest_launch_registers(0) == 0
    for more in (-8, -1, 1, 8):
        assert lib.bsa_selftest_launch_registers(more) == -10
    assert lib.bsa_strerror(-10) not in (b"", b"unknown status")
