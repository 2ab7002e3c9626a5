"""What a kernel reports through its stream's status word reaches the caller: named, once, from whichever
entry point looks first, and without touching another stream's report.  The word is set by the host here,
as a kernel would leave it; no kernel gives up."""
import ctypes

import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _word(stream):
    """The stream's status word in pinned host memory, as something that can be read and assigned."""
    from fa2_custom_mask import _lib
    _, status = _lib.native().state_tensors(stream.device_index, stream.cuda_stream)
    return ctypes.c_int32.from_address(status.data_ptr())


def _problem(seed, grad=False):
    q, k, v, do = (t.cuda() for t in oracle.make_qkv(1, 2, 512, 64, seed=seed, dtype=torch.float16, n=4))
    mask = oracle.make_block_mask(1, 2, 8, 0.5, seed=seed).cuda()
    return [t.requires_grad_(grad) for t in (q, k, v)], mask, do


def test_backward_names_the_role_and_takes_only_its_own_report(lib):
    from fa2_custom_mask import _lib, flash_attention_custom_mask
    from fa2_custom_mask import fa2_custom_mask as host
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(other):
        word2 = _word(other)
        host._stream_state(torch.device("cuda", other.device_index), other.cuda_stream)
    with torch.cuda.stream(s):
        qkv, mask, do = _problem(41, grad=True)
        o = flash_attention_custom_mask(*qkv, mask, 0.125)
        word = _word(s)
        s.synchronize()
        word.value, word2.value = 3, 2
        try:
            with pytest.raises(_lib.BsaError, match="role 3") as err:
                torch.autograd.grad(o, qkv, do, retain_graph=True)
            assert err.value.status == -9
            assert (word.value, word2.value) == (0, 2)
            got = torch.autograd.grad(o, qkv, do)             # the report was consumed
            s.synchronize()
        finally:
            word.value = word2.value = 0
    want = oracle.attn_forward_backward(*(t.detach().cpu() for t in qkv), mask.cpu(), 0.125, do.cpu())[2:]
    for g, w in zip(got, want):
        assert (g.float().cpu() - w).abs().max().item() <= 5e-2


def test_an_axis_order_that_is_none_is_reported(lib):
    """Its head is left as it is, the others are reordered; the first call after the kernel raises, the one
    after that works.  The same through the next reorder and through the attention op."""
    from fa2_custom_mask import flash_attention_custom_mask, inv_permute_attn_triton, permute_qkv_triton
    grid = dict(F=3, H=4, W=5, n_text_tokens=2)
    x = torch.randn(1, 6, 62, 64).half()
    good = torch.arange(6)[None]
    orders = oracle.PERMUTATIONS.copy()
    orders[[2, 4]] = 0, 1, 2
    want = x.clone()
    want[:, :, 2:] = oracle.reorder_by_view(x[:, :, 2:], orders, 3, 4, 5)
    qkv, mask, _ = _problem(43)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s), torch.no_grad():
        ts = [x.cuda() for _ in range(3)]
        permute_qkv_triton(*[t.clone() for t in ts], {"permute": good.cuda()}, 0, **grid)
        for low, high in ((-7, 6), (-2 ** 31, 2 ** 31 - 1)):
            bad = good.clone()
            bad[0, 2], bad[0, 4] = low, high
            for again in (lambda: permute_qkv_triton(*ts, {"permute": good.cuda()}, 0, **grid),
                          lambda: inv_permute_attn_triton(ts[0], {"permute": good.cuda().int()}, 0, **grid),
                          lambda: flash_attention_custom_mask(*qkv, mask, 0.125)):
                for plan in (bad.cuda(), bad.cuda().int()):
                    ts = [x.cuda() for _ in range(3)]
                    permute_qkv_triton(*ts, {"permute": plan}, 0, **grid)
                    s.synchronize()
                    assert all(torch.equal(t.cpu(), want) for t in ts)
                    with pytest.raises(IndexError, match="axis-order"):
                        again()
                    assert all(torch.equal(t.cpu(), want) for t in ts)
                    again()
                    s.synchronize()


def test_an_axis_order_that_is_none_in_a_plan_on_the_host(lib):
    from fa2_custom_mask import inv_permute_attn_triton, permute_qkv_triton
    grid = dict(F=3, H=4, W=5, n_text_tokens=2)
    x = torch.randn(1, 6, 62, 64).half()
    for bad in (-7, 6):
        for plan in (torch.tensor([[0, 1, bad, 3, 4, 5]]), [[0, 1, bad, 3, 4, 5]]):
            ts = [x.cuda() for _ in range(3)]
            with pytest.raises(IndexError):
                permute_qkv_triton(*ts, {"permute": plan}, 0, **grid)
            with pytest.raises(IndexError):
                inv_permute_attn_triton(ts[0], {"permute": plan}, 0, **grid)
            assert all(torch.equal(t.cpu(), x) for t in ts)


def test_report_on_a_stream_first_used_in_inference_mode(lib):
    """The stream's word belongs to no mode: a report is raised and taken outside inference mode too."""
    from fa2_custom_mask import _lib, flash_attention_custom_mask
    s = torch.cuda.Stream(priority=-1)
    with torch.cuda.stream(s), torch.no_grad():
        qkv, mask, _ = _problem(42)
        with torch.inference_mode():
            want = flash_attention_custom_mask(*qkv, mask, 0.125).clone()
        word = _word(s)
        s.synchronize()
        word.value = 4
        try:
            with pytest.raises(_lib.BsaError, match="role 4"):
                flash_attention_custom_mask(*qkv, mask, 0.125)
            assert word.value == 0
            assert torch.equal(flash_attention_custom_mask(*qkv, mask, 0.125), want)
        finally:
            word.value = 0
