"""The forward exponentiates against a reference maximum that it does not look up anew for every
superstep of four key blocks: rows whose logits jump at some later block must come out right whatever
the block's position in the list (either team's superstep, first or second tile of a lane), for every
remainder of the list length and every head dimension the kernel takes."""
import math

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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("element_mask", [False, True])
def test_a_superstep_that_is_done_again_moves_the_reference(lib, dtype, element_mask):
    """Logits that are too many above a row's reference for the sum test, and each too little above it for
    a rescale, must become the reference, or every later superstep of the row is done twice.  Seen from the
    outside: the first eight blocks have logits 0, all later ones z with 2^z half a step of the 16-bit
    grid above 64.  Against the moved reference their probabilities are 1, exactly; against the old one
    they are rounded down to 64, while the fp32 row sum has them whole.  Both results are worked out here,
    rounded to the output type: they differ in many columns, and O has to be the first one (but for columns
    where fp32 sums, good to 1e-6, may fall on the other side of a rounding step of 2^-10 or more)."""
    from fa2_custom_mask import attention_forward_masked
    nb, step = 40, 2.0 ** (-10 if dtype == torch.float16 else -7)
    N = 64 * nb
    q = torch.zeros(1, 1, N, 64)
    k = torch.zeros(1, 1, N, 64)
    q[..., 0] = 1
    k[:, :, 512:, 0] = 1
    v = torch.zeros(1, 1, N, 64)
    v[:, :, 512:] = torch.linspace(1.0, 2.0, 64)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    scale = math.log(64 * (1 + 0.499 * step))              # base 2 logits: log2(64 * (1 + step / 2))
    block = torch.ones(1, 1, nb, nb, dtype=torch.uint8)
    dense = None
    if element_mask:                                       # a block of marked ones whose elements are all kept
        block[..., 3] = 2
        dense = torch.ones(1, 1, N, N, dtype=torch.bool).cuda()
    o, _, _ = attention_forward_masked(q.cuda(), k.cuda(), v.cuda(), block.cuda(), scale, dense=dense)
    e = math.exp(scale)
    total = (N - 512) * e + 512
    moved, kept = (((N - 512) * p * v[0, 0, -1].double() / total).to(dtype) for p in (e, 64.0))
    assert (moved != kept).double().mean().item() >= 0.25
    assert (o[0, 0].cpu() == moved).double().mean().item() >= 0.95
