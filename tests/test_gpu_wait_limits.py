"""The limit of the kernels' waits, on barriers that nothing completes, and the flag that ends one before its limit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _limits(lib):
    """{form of the wait: milliseconds}; all of them wait at the same time and none is satisfied."""
    from fa2_custom_mask import _lib
    report = torch.full((12,), -1, dtype=torch.int32, device="cuda")
    assert lib.bsa_selftest_wait_limits(_lib.ptr(report), _lib.stream_ptr(report.device)) == 0
    got = report.cpu().tolist()
    assert got[0::2] == [0] * 6
    return dict(zip(("one", "two", "three", "item", "item with the flag"), got[1::2]))


def test_a_wait_on_several_barriers_has_the_limit_of_one(lib):
    """A limit for each barrier, one after the other, made it two and three times as long."""
    ms = _limits(lib)
    assert 1000 <= ms["one"] <= 10000
    for form in ("two", "three", "item"):
        assert 0.7 * ms["one"] <= ms[form] <= 1.4 * ms["one"], form
    assert lib.bsa_selftest_wait_limits(None, None) == -4


def test_the_flag_ends_a_wait_for_an_item(lib):
    """Looked at eight times within the limit: 100 ms until it is raised, up to an eighth of the limit until it is seen."""
    ms = _limits(lib)
    assert ms["item with the flag"] <= 100 + 0.25 * ms["one"] < 0.5 * ms["one"]


def test_a_role_that_gives_up_releases_the_others(lib):
    """The second warp begins to wait a second after the first one, whose limit raises the flag: by its own limit it
    would leave a second after it."""
    from fa2_custom_mask import _lib
    limit = _limits(lib)["one"]
    report = torch.full((4,), -1, dtype=torch.int32, device="cuda")
    assert lib.bsa_selftest_bounded_wait(None, _lib.ptr(report), _lib.stream_ptr(report.device)) == 0
    satisfied, satisfied_too, ended, ms = report.cpu().tolist()
    assert (satisfied, satisfied_too, ended) == (0, 0, 1)
    assert ms <= limit + 700
