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
