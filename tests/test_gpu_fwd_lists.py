"""The forward's lists: an item may be set up, and its Q loaded, while the one before the previous one is still being
written out.  Runs of empty rows, of single tiles and of long rows in one CTA's sequence of items."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
NB = 40


def _mask(pattern):
    """Row i keeps the first pattern[i % len] entries of a permutation of its own."""
    m = torch.zeros(NB, NB, dtype=torch.bool)
    for i in range(NB):
        m[i, torch.randperm(NB, generator=torch.Generator().manual_seed(i))[:pattern[i % len(pattern)]]] = True
    return m[None, None]


@pytest.mark.parametrize("pattern", [(0, 0, 0, 1), (1,), (1, 1, 40), (0, 5, 1, 0, 4, 8, 9, 2, 12, 13, 3), (40, 0, 1, 2)],
                         ids=lambda p: "-".join(map(str, p)))
@pytest.mark.parametrize("dtype,D,elements", [(torch.float16, 64, False), (torch.bfloat16, 32, False),
                                              (torch.bfloat16, 64, True)])
def test_runs_of_short_and_empty_rows(lib, pattern, dtype, D, elements):
    """Against the fp32 oracle; the same heads among 30 others (27 items a CTA) and one after the other bit for bit."""
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v = oracle.make_qkv(1, 3, 64 * NB, D, seed=7, dtype=dtype)
    block = _mask(pattern)
    mask = block.cuda()
    if elements:
        mask = mask.repeat_interleave(64, -2).repeat_interleave(64, -1)

    def run(ts):
        return flash_attention_custom_mask(*(t.cuda() for t in ts), mask, D ** -0.5)

    got = run((q, k, v))
    for _ in range(3):
        assert torch.equal(run([t.repeat(1, 33, 1, 1) for t in (q, k, v)]), got.repeat(1, 33, 1, 1))
    for h in range(3):
        assert torch.equal(run([t[:, h:h + 1] for t in (q, k, v)]), got[:, h:h + 1])
    ref = oracle.attn_forward(q, k, v, block.expand(1, 3, NB, NB), D ** -0.5)[0]
    # P and O are rounded to the inputs' type: half a unit in the last place of values up to 4 or so, twice
    assert (got.float().cpu() - ref).abs().max() <= (4e-3 if dtype == torch.float16 else 3e-2)
