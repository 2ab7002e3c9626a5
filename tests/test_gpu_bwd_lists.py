"""The backward's lists: their first 32 entries come with the block, the others 32 at a time, and a block of the next
head may be set up while this one's is still at work."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
NB = 70


def _mask():
    """Rows and columns of 0, 1, 2, 31..34, 63..66 and 70 tiles, empty ones and single tiles between them."""
    m = torch.zeros(2, NB, NB, dtype=torch.bool)
    for h in range(2):
        for i, n in enumerate([1, 0, 31, 1, 32, 2, 33, 0, 34, 1, 63, 1, 64, 65, 1, 66, 70]):
            line = torch.randperm(NB, generator=torch.Generator().manual_seed(100 * h + i))[:n]
            at = 4 * i % NB
            if h == 0:
                m[h, at, line] = True
            else:
                m[h, line, at] = True
        m[h] |= torch.eye(NB, dtype=torch.bool) & (torch.arange(NB) % 3 != 0)[:, None]
    return m[None]


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 32)])
def test_lists_of_every_length(lib, dtype, D):
    """Against autograd through the fp32 oracle, and bit for bit against the same heads among 40 others."""
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v, do = oracle.make_qkv(1, 2, 64 * NB, D, seed=5, dtype=dtype, n=4)
    mask = _mask()

    def run(reps):
        ts = [t.cuda().repeat(1, reps, 1, 1).requires_grad_(True) for t in (q, k, v)]
        o = flash_attention_custom_mask(*ts, mask.cuda().repeat(1, reps, 1, 1), D ** -0.5)
        return [g.detach() for g in torch.autograd.grad(o, ts, do.cuda().repeat(1, reps, 1, 1))]

    got = run(1)
    many = run(20)
    for g, m in zip(got, many):
        assert torch.equal(m, g.repeat(1, 20, 1, 1))
    refs = oracle.attn_forward_backward(q, k, v, mask, D ** -0.5, do)[2:]
    for g, r in zip(got, refs):
        assert (g.float().cpu() - r).abs().max() <= 5e-2
