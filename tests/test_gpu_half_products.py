"""The product that the attention kernels accumulate with: 64 rows in each lane half of tensor memory, each half times a
tile of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = {torch.float16: 0, torch.bfloat16: 1}


def _product(lib, a, b):
    from fa2_custom_mask import _lib
    a_dev, b_dev = a.cuda(), b.cuda()
    out = torch.full((128, 64), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = _lib.stream_ptr(out.device)
    assert lib.bsa_selftest_half_products(_lib.ptr(a_dev), _lib.ptr(b_dev), _lib.ptr(out), DTYPES[a.dtype],
                                          _lib.ptr(status), stream) == 0
    assert lib.bsa_check_status(_lib.ptr(status), stream) == 0
    return out.cpu()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("seed", range(3))
def test_each_lane_half_has_rows_and_a_tile_of_its_own(lib, dtype, seed):
    """Whole numbers up to 8, so that sums are exact; one half of NaN leaves the other one as it is."""
    g = torch.Generator().manual_seed(seed)
    a = torch.randint(-8, 9, (128, 64), generator=g)
    b = torch.randint(-8, 9, (2, 64, 64), generator=g)
    want = torch.cat([a[:64] @ b[0], a[64:] @ b[1]]).float()
    swapped = torch.cat([a[:64] @ b[1], a[64:] @ b[0]]).float()
    same_rows = torch.cat([a[:64] @ b[0], a[:64] @ b[1]]).float()
    assert not torch.equal(want, swapped) and not torch.equal(want, same_rows)
    assert torch.equal(_product(lib, a.to(dtype), b.to(dtype)), want)
    for half in range(2):
        rows = slice(64 * half, 64 * half + 64)
        bad_a, bad_b = a.to(dtype), b.to(dtype)
        bad_a[64 * (1 - half):64 * (2 - half)] = float("nan")
        bad_b[1 - half] = float("nan")
        assert torch.equal(_product(lib, bad_a, b.to(dtype))[rows], want[rows])
        assert torch.equal(_product(lib, a.to(dtype), bad_b)[rows], want[rows])


def test_bad_arguments_are_refused(lib):
    from fa2_custom_mask import _lib
    t = torch.zeros(128 * 64, device="cuda")
    assert lib.bsa_selftest_half_products(None, _lib.ptr(t), _lib.ptr(t), 0, None, None) == -4
    assert lib.bsa_selftest_half_products(_lib.ptr(t), _lib.ptr(t), _lib.ptr(t), 7, None, None) == -2
