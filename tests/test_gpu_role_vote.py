"""The warps of a role that meet at a named barrier go on together or leave together, whatever the others were told when
the wait of one of them ran out: an item with work, one without, or the end.  (On its own verdict, a warp that saw
the end left the others at a barrier that it never came to.)  The waits are made to run out by the test kernel."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu
WORK = (0, 2, 3, 6)  # of items 0..7; 7 is the end


def _expected(run_out):
    """Items with work before the first wait that runs out."""
    first = min([i for i in run_out if 0 <= i <= 7], default=8)
    return sum(i < first for i in WORK) + 100


def test_all_warps_leave_together(lib):
    from fa2_custom_mask import _lib
    one = [tuple(i if w == warp else -1 for w in range(4)) for warp in range(4) for i in range(8)]
    cases = [(-1,) * 4, (8,) * 4, *one, *itertools.product((1, 4, 7), (2, 5, 7), (-1, 6), (3, 7))]
    reports = torch.full((len(cases), 4), -1, dtype=torch.int32, device="cuda")
    for case, report in zip(cases, reports):
        assert lib.bsa_selftest_role_vote(*case, _lib.ptr(report), _lib.stream_ptr(report.device)) == 0
    for case, got in zip(cases, reports.cpu().tolist()):
        assert got == [_expected(case)] * 4, case
    assert lib.bsa_selftest_role_vote(0, 0, 0, 0, None, None) == -4
