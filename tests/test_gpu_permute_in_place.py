"""The one-launch in-place token reorder against the oracle's view permutation: every axis order, both
directions, grids that take one CTA, a cluster of 16 and one column chunk or several, odd extents, text
tokens in front, and the tensors and plans that go through the two-pass form instead."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 128), (torch.float32, 16),
                                     (torch.float16, 24), (torch.float16, 20), (torch.uint8, 16)])
@pytest.mark.parametrize("F,H,W,text", [(1, 1, 1, 0), (2, 1, 3, 1), (3, 4, 5, 7), (13, 30, 45, 226),
                                        (16, 33, 47, 0), (5, 7, 131, 3)])
def test_both_directions(lib, dtype, D, F, H, W, text):
    from fa2_custom_mask import inv_permute_attn_triton, permute_qkv_triton
    B, heads = 2, 7
    g = torch.Generator().manual_seed(F + D)
    x = [(torch.randn(B, heads, text + F * H * W, D, generator=g) * 50).to(dtype) for _ in range(3)]
    idx = torch.tensor([[0, 1, 2, 3, 4, 5, 2]])
    orders = oracle.PERMUTATIONS[idx[0].numpy()]
    plan = {"permute": idx.cuda()}
    dev = [t.cuda() for t in x]
    out = permute_qkv_triton(*dev, plan, 0, F=F, H=H, W=W, n_text_tokens=text)
    for t, o, d in zip(x, out, dev):
        assert o.data_ptr() == d.data_ptr()
        want = t.clone()
        want[:, :, text:] = oracle.reorder_by_view(t[:, :, text:], orders, F, H, W)
        assert torch.equal(o.cpu(), want)
        back = inv_permute_attn_triton(o, {"permute": idx.int().cuda()}, 0, F=F, H=H, W=W, n_text_tokens=text)
        assert torch.equal(back.cpu(), t)


def test_views_shared_storage_and_plans(lib):
    from fa2_custom_mask import permute_qkv_triton
    F, H, W, heads, text = 3, 5, 4, 6, 2
    T = text + F * H * W
    fused = torch.randn(2, T, 3, heads, 64, device="cuda").half()
    q, k, v = (fused[:, :, i].transpose(1, 2) for i in range(3))      # one storage
    want = [t.clone() for t in (q, k, v)]
    for w in want:
        w[:, :, text:] = oracle.reorder_by_view(w[:, :, text:].cpu(), oracle.PERMUTATIONS, F, H, W).cuda()
    for plan in (torch.arange(6).cuda()[None], torch.arange(6)[None].cuda().int(),
                 torch.arange(-6, 0).cuda()[None]):                    # (-6 is order 0 again)
        before = fused.clone()
        permute_qkv_triton(q, k, v, {"permute": plan}, 0, F=F, H=H, W=W, n_text_tokens=text)
        for t, w in zip((q, k, v), want):
            assert torch.equal(t, w)
        fused.copy_(before)
    one = torch.randn(1, heads, T, 64, device="cuda").half()
    same = one.clone()
    permute_qkv_triton(one, one, one, {"permute": torch.ones(1, heads, dtype=torch.long).cuda()}, 0, F=F, H=H,
                       W=W, n_text_tokens=text)                        # three times the same tensor
    for _ in range(3):
        same[:, :, text:] = oracle.reorder_by_view(same[:, :, text:].cpu(), oracle.PERMUTATIONS[[1] * heads],
                                                   F, H, W).cuda()
    assert torch.equal(one, same)
