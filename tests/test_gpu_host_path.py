"""What the native host path of the public op takes, and what it has to leave to the general one."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _problem(dtype=torch.float16, N=512, D=64, seed=51):
    q, k, v, do = (t.to(dtype).cuda() for t in oracle.make_qkv(1, 2, N, D, seed=seed, n=4))
    return q, k, v, do, oracle.make_block_mask(1, 2, N // 64, 0.5, seed=seed).cuda()


def test_forward_mode_tangents_are_refused(lib):
    """The op has no forward derivative; an input with a tangent is refused instead of losing it."""
    import torch.autograd.forward_ad as fwd
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v, _, mask = _problem()
    with fwd.dual_level():
        for i in range(3):
            args = [fwd.make_dual(t, torch.ones_like(t)) if i == j else t for j, t in enumerate((q, k, v))]
            for grad in (True, False):
                with torch.set_grad_enabled(grad), pytest.raises(NotImplementedError):
                    flash_attention_custom_mask(*args, mask, 0.125)


@pytest.mark.parametrize("byte_mask", [False, True])
def test_transforms_that_the_op_does_not_have_are_refused(lib, byte_mask):
    """Tracing, vmap and the functional derivatives: no result rather than one without the kernels."""
    import torch.func as F
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v, _, mask = _problem()
    if byte_mask:
        mask = mask.view(torch.uint8)

    def op(q, mask):
        return flash_attention_custom_mask(q, k, v, mask, 0.125)

    for call in (lambda: torch.jit.trace(op, (q, mask), check_trace=False),
                 lambda: torch.jit.trace(op, (q.clone().requires_grad_(True), mask), check_trace=False),
                 lambda: F.vmap(op, (0, None))(torch.stack([q, q]), mask),
                 lambda: F.vmap(op, (None, 0))(q, torch.stack([mask, mask])),
                 lambda: F.grad(lambda q: op(q, mask).sum())(q),
                 lambda: F.jvp(lambda q: op(q, mask), (q,), (q,))):
        with pytest.raises((RuntimeError, AssertionError, NotImplementedError)):
            call()


def test_saved_tensor_hooks_see_what_the_backward_keeps(lib):
    """Everything that the op makes for its backward goes through the saved-tensor hooks (offloading,
    checkpointing): q, k, v, O, the log-sum-exp and the tile lists."""
    from fa2_custom_mask import flash_attention_custom_mask
    q, k, v, do, mask = _problem()
    for t in (q, k, v):
        t.requires_grad_(True)
    want = torch.autograd.grad(flash_attention_custom_mask(q, k, v, mask, 0.125), (q, k, v), do)
    packed = []

    def pack(t):
        packed.append(t.dtype)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        o = flash_attention_custom_mask(q, k, v, mask, 0.125)
    assert sorted(map(str, packed)) == ["torch.float16"] * 4 + ["torch.float32", "torch.int32"]
    for g, w in zip(torch.autograd.grad(o, (q, k, v), do), want):
        assert torch.equal(g, w)


def test_inference_tensors_are_reordered_outside_inference_mode(lib):
    from fa2_custom_mask import inv_permute_attn_triton, permute_qkv_triton
    grid = dict(F=3, H=4, W=5, n_text_tokens=2)
    x = torch.randn(1, 6, 62, 64).half()
    plan = {"permute": torch.arange(6, device="cuda")[None]}
    with torch.inference_mode():
        ts = [x.cuda() for _ in range(3)]
    want = x.clone()
    want[:, :, 2:] = oracle.reorder_by_view(x[:, :, 2:], oracle.PERMUTATIONS, 3, 4, 5)
    for t in permute_qkv_triton(*ts, plan, 0, **grid):
        assert t.is_inference() and torch.equal(t.cpu(), want)
        assert torch.equal(inv_permute_attn_triton(t, plan, 0, **grid).cpu(), x)


@pytest.mark.parametrize("native", [True, False])
def test_a_captured_call_does_not_draw_from_its_streams_counter(lib, native):
    """A graph may be replayed on any stream, beside calls on the one it was captured on.  Seen here with a
    counter that says that everything has been handed out, and in replays beside such calls."""
    from fa2_custom_mask import _lib, flash_attention_custom_mask
    from fa2_custom_mask import fa2_custom_mask as host
    op = flash_attention_custom_mask if native else host._attention.apply
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    q, k, v, do = (t.cuda() for t in oracle.make_qkv(1, 4, 4096, 64, seed=52, dtype=torch.float16, n=4))
    mask = oracle.make_block_mask(1, 4, 64, 0.2, seed=52, causal=True).cuda()   # 256 rows of blocks
    for t in (q, k, v):
        t.requires_grad_(True)

    def step():
        o = op(q, k, v, mask, 0.125)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]

    with torch.cuda.stream(s):
        want = step()
        counter, _ = _lib.native().state_tensors(s.device_index, s.cuda_stream)
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            got = step()
        for t in got:
            t.zero_()
        counter.fill_(1 << 20)
        graph.replay()
        s.synchronize()
        assert int(counter.item()) == 1 << 20
        counter.zero_()
        s.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    eager = []
    for _ in range(8):
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(s):
            eager.append(step())
    torch.cuda.synchronize()
    for res in (got, *eager):
        assert all(torch.equal(g, w) for g, w in zip(res, want))
    assert int(counter.item()) == 0
