"""What a kernel does when one of its bounded waits gives up: no fault, no hang, on waits made to run out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_warp_gives_up_as_a_whole_and_an_items_wait_with_the_flag(lib):
    """Half of the lanes see their barrier complete, the others never do: none may go on alone.  The flag is
    raised after 20 ms and looked at every quarter of a second; the wait without it makes all of its tries
    (0.04 s: the hardware does not suspend a warp whose lanes have parted, and 2 s one that is together)."""
    from fa2_custom_mask import _lib
    report = torch.full((5,), -1, dtype=torch.int32, device="cuda")
    assert lib.bsa_selftest_give_up(_lib.ptr(report), _lib.stream_ptr(report.device)) == 0
    with_flag, ms_flag, alone, ms_alone, ended = report.cpu().tolist()
    assert with_flag == 0 and alone == 0 and ended == 1
    assert ms_flag < 1000 and ms_alone <= 10000
