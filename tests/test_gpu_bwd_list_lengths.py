"""The backward's lists at the lengths where something changes: a half pair, the first 32 entries that come with the block, the
batches of 32 behind them; and how much of a gradient one entry is."""
import functools

import pytest
import torch

from oracle import oracle

NB = 70
LENGTHS = (0, 1, 2, 31, 32, 33, 34, 63, 64, 65, 66, 70)
# Largest error of a block of 64 rows over its largest value.  P and dS are rounded to 16 bits (half a unit: 2^-9 of a
# term in bf16, 2^-12 in fp16) and so are O, from which delta is, and the result; the errors of 64 to 4,480 terms of
# either sign add up like the terms do.  Four such roundings: 8e-3 and 1e-3, and a little more for delta.  (The same roundings
# emulated on the CPU: up to 7e-3 in bf16, 7.5e-4 in fp16.)
BOUND = {torch.bfloat16: 1e-2, torch.float16: 2e-3}
CASES = pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 64), (torch.bfloat16, 32)])


def _mask():
    """[1, 2, NB, NB]: rows of head 0 and columns of head 1 with every one of LENGTHS, single tiles and random lengths between."""
    m = torch.zeros(2, NB, NB, dtype=torch.bool)
    for h in range(2):
        g = torch.Generator().manual_seed(h)
        for i in range(NB):
            n = LENGTHS[i // 2] if i % 2 == 0 and i // 2 < len(LENGTHS) else (1 if i % 3 else int(torch.randint(0, NB + 1, (1,), generator=g)))
            line = torch.randperm(NB, generator=g)[:n]
            if h == 0:
                m[0, i, line] = True
            else:
                m[1, line, i] = True
    return m[None]


@functools.lru_cache(maxsize=1)
def _inputs(dtype, D):
    return oracle.make_qkv(1, 2, 64 * NB, D, seed=11, dtype=dtype, n=4)


def _largest(x):
    """[.., nb, rows..] -> largest magnitude of each block of 64 rows of [1, 2, N, D]."""
    return x.reshape(2, NB, -1).abs().amax(-1)


def test_the_lists_have_these_lengths():
    m = _mask()[0]
    assert set(LENGTHS) <= set(m[0].sum(1).tolist()) and set(LENGTHS) <= set(m[1].sum(0).tolist())


@CASES
def test_one_entry_more_or_less_exceeds_the_bound(dtype, D):
    """dQ of head 0 and dK, dV of head 1, tile by tile on the CPU: what a lost or repeated entry of any list changes."""
    q, k, v, do = (t[0].float() for t in _inputs(dtype, D))
    mask = _mask()[0]
    for h in range(2):
        s = (q[h] @ k[h].T * D ** -0.5).masked_fill(~oracle.expand_block_mask(mask[h]), float("-inf"))
        p = torch.nan_to_num(torch.softmax(s, -1), nan=0.0)
        dp = do[h] @ v[h].T
        ds = p * (dp - (p * dp).sum(-1, keepdim=True)) * D ** -0.5
        p, ds = (x.reshape(NB, 64, NB, 64) for x in (p, ds))
        q4, k4, do4 = (x[h].reshape(NB, 64, D) for x in (q, k, do))
        if h == 0:
            parts = [torch.einsum("aibj,bjd->abid", ds, k4)]
        else:
            parts = [torch.einsum("aibj,aid->bajd", x, y) for x, y in ((ds, q4), (p, do4))]
        for part in parts:
            one = part.abs().amax((-1, -2))
            whole = part.sum(1).abs().amax((-1, -2))
            listed = mask[0] if h == 0 else mask[1].T
            assert (one / whole.clamp_min(1e-30)[:, None])[listed].min() > 2 * BOUND[dtype]


@pytest.mark.gpu
@CASES
def test_gradients_of_every_list(lib, dtype, D):
    """Against autograd through the fp32 oracle, block by block."""
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v, do = _inputs(dtype, D)
    mask = _mask()
    ts = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    o = flash_attention_custom_mask(*ts, mask.cuda(), D ** -0.5)
    got = torch.autograd.grad(o, ts, do.cuda())
    refs = oracle.attn_forward_backward(q, k, v, mask, D ** -0.5, do)[2:]
    for g, r in zip(got, refs):
        error, size = _largest(g.float().cpu() - r), _largest(r)
        assert (error <= BOUND[dtype] * size).all(), (error / size.clamp_min(1e-30)).max()
