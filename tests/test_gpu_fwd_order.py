"""The order in which the forward hands out its work items: whatever it is, every query block is done once."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


# one CTA per SM (148); up to 4 items each the first query blocks of all heads come first, an eighth of a head's
# at most 8: one, none (heads of 7), 8, those of a row range, the largest such grid and one above it
@pytest.mark.parametrize("B,H,nb,rows", [
    (1, 19, 8, None), (2, 37, 7, None), (1, 3, 64, None), (2, 2, 70, (3, 67)), (1, 74, 8, None), (1, 75, 8, None)])
@pytest.mark.parametrize("mode", ["lists", "mask"])
def test_every_block_is_done_whatever_the_order(lib, B, H, nb, rows, mode):
    """Against calls on one head each, which have one item per CTA and no order: bit-equal, and the rows outside
    the range keep what they held."""
    from fa2_custom_mask import attention_forward, attention_forward_masked, build_tile_lists
    q, k, v = (t.cuda() for t in oracle.make_qkv(B, H, 64 * nb, 64, seed=71, dtype=torch.float16))
    mask = oracle.make_block_mask(B, H, nb, 0.3, seed=71).cuda()
    mask[:, :, :2] = True
    mask[:, :, nb // 2] = False

    def run(b, h):
        args = [t[b, h].contiguous() for t in (q, k, v)]
        out = (torch.full_like(args[0], 7.0), torch.full(args[0].shape[:3], 7.0, device="cuda"))
        m = mask[b, h].contiguous()
        if mode == "lists":
            attention_forward(*args, build_tile_lists(m, want_csc=False), 0.125, rows=rows, out=out)
        else:
            attention_forward_masked(*args, m, 0.125, rows=rows, out=out)
        return out

    o, lse = run(slice(None), slice(None))
    for b in range(B):
        for h in range(H):
            want_o, want_lse = run(slice(b, b + 1), slice(h, h + 1))
            assert torch.equal(o[b:b + 1, h:h + 1], want_o)
            assert torch.equal(lse[b:b + 1, h:h + 1], want_lse)
