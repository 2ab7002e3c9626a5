"""The forward exponentiates against a reference maximum that it does not look up anew for every
superstep of four key blocks: rows whose logits jump at some later block must come out right whatever
the block's position in the list (either team's superstep, first or second tile of a lane), for every
remainder of the list length and every head dimension the kernel takes."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("dtype,tol", [(torch.float16, 2e-2), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("nb", [1, 2, 3, 5, 8, 11, 13, 18])
def test_logits_that_jump_at_one_block(lib, nb, dtype, tol, D):
    from fa2_custom_mask import attention_forward_masked
    for pos in sorted({0, nb - 1, nb // 2, min(4, nb - 1), min(7, nb - 1)}):
        q, k, v = (t.to(dtype) for t in oracle.make_qkv(1, 2, 64 * nb, D, seed=nb + pos))
        k[:, :, 64 * pos:64 * (pos + 1)] *= 12
        k[:, 1, 64 * pos + 32:] *= 2      # and again behind it, in the second head
        mask = torch.ones(1, 1, nb, nb, dtype=torch.bool)
        scale = D ** -0.5
        o, lse2, _ = attention_forward_masked(q.cuda(), k.cuda(), v.cuda(), mask.cuda(), scale)
        o_ref, lse_ref = oracle.attn_forward(q, k, v, mask.expand(1, 2, nb, nb), scale)
        assert (o.float().cpu() - o_ref).abs().max().item() <= tol, (nb, pos)
        err = (lse2.cpu() * 0.6931471805599453 - lse_ref).abs().max().item()
        assert err <= 2e-3 * max(1.0, lse_ref.abs().max().item() / 8), (nb, pos, err)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 9])
def test_logits_that_jump_inside_the_first_blocks(lib, nb, dtype):
    """The reference of a row comes from the first 32 keys of its first tile; here the keys behind
    them, or the row's second tile, have logits that would not go into 16 bit against it."""
    from fa2_custom_mask import attention_forward_masked
    for start in (32, 64, 128):
        if start >= 64 * nb:
            continue
        q, k, v = (t.to(dtype) for t in oracle.make_qkv(1, 2, 64 * nb, 64, seed=nb + start))
        k[:, :, :start] *= 0.01
        k[:, :, start:] *= 25
        mask = torch.ones(1, 1, nb, nb, dtype=torch.bool)
        o, lse2, rowmax = attention_forward_masked(q.cuda(), k.cuda(), v.cuda(), mask.cuda(), 0.125)
        o_ref, lse_ref = oracle.attn_forward(q, k, v, mask.expand(1, 2, nb, nb), 0.125)
        assert (o.float().cpu() - o_ref).abs().max().item() <= 2e-2, (nb, start)
        err = (lse2.cpu() * 0.6931471805599453 - lse_ref).abs().max().item()
        assert err <= 2e-3 * max(1.0, lse_ref.abs().max().item() / 8), (nb, start, err)
