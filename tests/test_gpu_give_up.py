"""What a kernel does when one of its bounded waits gives up: no fault, no hang, on waits made to run out."""
import pytest
import torch

from oracle import oracle

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


@pytest.mark.parametrize("train", [False, True])
def test_a_long_kernel_ahead_that_lets_us_in_early_is_waited_for(lib, train):
    """5.5 s, more than any wait's own limit (2^33 cycles for the sleeping ones, 4.4 s at 1.965 GHz): results as
    without that kernel, and nothing is reported.  Training: ahead of the forward and of the backward."""
    from fa2_custom_mask import _lib, flash_attention_custom_mask
    q, k, v, do = (t.cuda() for t in oracle.make_qkv(1, 2, 640, 64, seed=61, dtype=torch.float16, n=4))
    mask = oracle.make_block_mask(1, 2, 10, 0.5, seed=61).cuda()
    qkv = [t.requires_grad_(train) for t in (q, k, v)]
    stream = _lib.stream_ptr(q.device)

    def run(ms):
        assert lib.bsa_selftest_early_kernel(ms, stream) == 0
        o = flash_attention_custom_mask(*qkv, mask, 0.125)
        if not train:
            return [o]
        assert lib.bsa_selftest_early_kernel(ms, stream) == 0
        return [o, *torch.autograd.grad(o, qkv, do)]

    want, got = run(0), run(5500)
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    assert all(torch.equal(g, w) for g, w in zip(run(0), want))  # (raises what was reported)
    torch.cuda.synchronize()
