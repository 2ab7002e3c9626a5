"""Backward with operands that do not share their strides (q, k, v as slices of one fused projection or
as [B,N,H,D] storage, dO in another layout), every head dimension, list lengths around the two-tile
supersteps and lists of a single tile, against autograd through the fp32 oracle."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _laid_out(t, layout, others=()):
    B, H, N, D = t.shape
    if layout == "bnhd":
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if layout == "qkv":
        fused = torch.stack([x.transpose(1, 2) for x in (t, *others)], 2).contiguous()
        return [fused[:, :, i].transpose(1, 2) for i in range(1 + len(others))]
    return t


@pytest.mark.parametrize("layout", ["bhnd", "bnhd", "qkv"])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("nb,density", [(1, 1.0), (3, 0.4), (9, 0.25), (21, 0.3)])
def test_gradients_of_differently_strided_operands(lib, layout, D, nb, density):
    from fa2_custom_mask import flash_attention_custom_mask
    B, H, N, scale = 2, 3, 64 * nb, D ** -0.5
    q, k, v, do = (t.to(torch.float16) for t in oracle.make_qkv(B, H, N, D, seed=nb + D, n=4))
    mask = oracle.make_block_mask(B, H, nb, density, seed=nb, causal=nb == 9)
    ref = oracle.attn_forward_backward(q, k, v, mask, scale, do)
    qc, kc, vc = (t.cuda() for t in (q, k, v))
    if layout == "qkv":
        qc, kc, vc = _laid_out(qc, layout, (kc, vc))
    else:
        qc, kc, vc = (_laid_out(t, layout) for t in (qc, kc, vc))
    qc, kc, vc = (t.detach().requires_grad_(True) for t in (qc, kc, vc))
    o = flash_attention_custom_mask(qc, kc, vc, mask.cuda(), scale)
    assert o.is_contiguous()
    for dout in (do.cuda(), _laid_out(do.cuda(), "bnhd")):
        grads = torch.autograd.grad(o, (qc, kc, vc), dout, retain_graph=True)
        for got, want, t in zip(grads, ref[2:], (qc, kc, vc)):
            assert got.stride() == t.stride()
            assert (got.float().cpu() - want).abs().max().item() <= 5e-2
    assert (o.detach().float().cpu() - ref[0]).abs().max().item() <= 2e-2


@pytest.mark.parametrize("Bm,Hm,nb", [(1, 1, 1), (2, 3, 31), (1, 4, 65), (2, 1, 130)])
def test_lists_in_places_equal_the_compact_ones(lib, Bm, Hm, nb):
    from fa2_custom_mask import _lib, build_tile_lists
    mask = oracle.make_block_mask(Bm, Hm, nb, 0.3, seed=nb, diagonal=False).cuda()
    tl = build_tile_lists(mask)
    rows = Bm * Hm * nb
    cnt = [torch.full((rows,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    ent = [torch.full((rows, nb), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    m = mask.view(torch.uint8)
    assert lib.bsa_tile_lists_places(_lib.ptr(m), _lib.strides4(m), Bm, Hm, nb, _lib.ptr(cnt[0]),
                                     _lib.ptr(ent[0]), _lib.ptr(cnt[1]), _lib.ptr(ent[1]),
                                     _lib.stream_ptr(m.device)) == 0
    for c, e, ptr, idx in zip(cnt, ent, (tl.row_ptr, tl.col_ptr), (tl.col_idx, tl.row_idx)):
        assert torch.equal(c, ptr[1:] - ptr[:-1])
        keep = torch.arange(nb, device="cuda") < c[:, None]
        assert torch.equal(e[keep], idx[: int(ptr[-1])]) and bool((e[~keep] == -1).all())
