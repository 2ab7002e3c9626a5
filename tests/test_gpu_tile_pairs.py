"""Products of two tiles at once: a list that ends with half a pair must not see what the other half's place holds.

Every second head is made of NaN, so that the SMs that work on the others have NaN left in their buffers, in
shared and in tensor memory; lists are 1 to 9 tiles long.  The sound heads must be what they are without the
others, bit for bit, and right."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
NB, HEADS = 9, 66  # 594 query blocks: four or five on every one of 148 SMs


def _run(q, k, v, do, mask, train):
    from fa2_custom_mask import flash_attention_custom_mask
    ts = [t.detach().requires_grad_(train) for t in (q, k, v)]
    o = flash_attention_custom_mask(*ts, mask, q.shape[-1] ** -0.5)
    return [o.detach(), *torch.autograd.grad(o, ts, do)] if train else [o]


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 64), (torch.float16, 32), (torch.bfloat16, 16)])
def test_half_pairs_see_zeros(lib, train, dtype, D):
    q, k, v, do = (t.cuda() for t in oracle.make_qkv(1, HEADS, 64 * NB, D, seed=D, dtype=dtype, n=4))
    mask = torch.ones(NB, NB, dtype=torch.bool).tril().cuda()
    want = _run(q, k, v, do, mask, train)
    for t in (q, k, v, do):
        t[:, 1::2] = float("nan")
    for _ in range(3):
        got = _run(q, k, v, do, mask, train)
        for g, w in zip(got, want):
            assert torch.equal(g[:, ::2], w[:, ::2])
    args = [t[:, :1].cpu() for t in (q, k, v)]
    block = mask.cpu().expand(1, 1, NB, NB)
    if train:
        o, _, dq, dk, dv = oracle.attn_forward_backward(*args, block, D ** -0.5, do[:, :1].cpu())
        refs = [o, dq, dk, dv]
    else:
        refs = [oracle.attn_forward(*args, block, D ** -0.5)[0]]
    for g, r, tol in zip(got, refs, (2e-2, 5e-2, 5e-2, 5e-2)):
        assert (g[:, :1].float().cpu() - r).abs().max() <= tol
