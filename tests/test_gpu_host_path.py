"""What the native host path of the public op takes, and what it has to leave to the general one."""
import ctypes

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


def test_a_captured_step_zeroes_its_counters_once_for_each_direction(lib):
    """With more blocks than SMs a graph has two nodes more than with fewer: one for the forward's work counter
    and one for both of the backward's."""
    from fa2_custom_mask import flash_attention_custom_mask as op

    def nodes(H):
        q, k, v, do = (t.cuda() for t in oracle.make_qkv(1, H, 4096, 64, seed=53, dtype=torch.float16, n=4))
        mask = oracle.make_block_mask(1, H, 64, 0.2, seed=53).cuda()
        for t in (q, k, v):
            t.requires_grad_(True)

        def step():
            o = op(q, k, v, mask, 0.125)
            return [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]

        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            step()
            s.synchronize()
            graph = torch.cuda.CUDAGraph(keep_graph=True)
            with torch.cuda.graph(graph, stream=s):
                step()
        n = ctypes.c_size_t()
        assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None,
                                                           ctypes.byref(n)) == 0
        return n.value

    assert nodes(4) == nodes(2) + 2      # 256 and 128 blocks for 148 CTAs


def _layouts(dtype, N, D):
    """Name -> q, k, v as programs hold them: contiguous, projections, slices of a fused projection, and
    rows that the copy engine cannot read in place (copied first)."""
    B, H = 2, 3
    fused = torch.randn(B, N, 3, H, D, device="cuda", dtype=dtype)
    return {
        "bhnd": [torch.randn(B, H, N, D, device="cuda", dtype=dtype) for _ in range(3)],
        "bnhd": [torch.randn(B, N, H, D, device="cuda", dtype=dtype).transpose(1, 2) for _ in range(3)],
        "qkv": [fused[:, :, i].transpose(1, 2) for i in range(3)],
        "odd rows": [torch.randn(B, H, N, D + 1, device="cuda", dtype=dtype)[..., :D] for _ in range(3)],
    }


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
def test_ordinary_calls_take_the_native_path(lib, monkeypatch, dtype, D):
    """Whatever the native path refuses goes through the Python layer without a word and costs six times
    the host time; here that layer is taken away."""
    from fa2_custom_mask import flash_attention_custom_mask
    from fa2_custom_mask import fa2_custom_mask as host
    monkeypatch.setattr(host, "_attention", None)
    N, nb = 192, 3
    block = torch.rand(2, 3, nb, nb, device="cuda") < 0.5
    dense = torch.rand(N, N, device="cuda") < 0.5
    masks = [block, block[:1], block[:, :1], block[:1, :1], block[0], block[0, 0], block.view(torch.uint8),
             block.transpose(2, 3), dense, dense.view(torch.uint8), dense.expand(2, 3, N, N), dense.t()]
    for name, qkv in _layouts(dtype, N, D).items():
        for mask in masks if name == "bhnd" else [block, dense]:
            with torch.no_grad():
                assert flash_attention_custom_mask(*qkv, mask, 0.125).shape == (2, 3, N, D)
            for needs in ((True, True, True), (False, True, False)):
                leaves = [t.detach().requires_grad_(n) for t, n in zip(qkv, needs)]
                o = flash_attention_custom_mask(*leaves, mask, 0.125)
                assert o.grad_fn.name() == "AttentionBackward"
                wanted = [t for t in leaves if t.requires_grad]
                for g, t in zip(torch.autograd.grad(o, wanted, torch.ones_like(o)), wanted):
                    assert g.shape == t.shape
    with pytest.raises(AttributeError):      # what it does not take: no mask
        flash_attention_custom_mask(*qkv, None, 0.125)


def test_reorders_that_take_one_launch(lib, monkeypatch):
    """Up to 18,432 tokens of rows that split into 64-byte chunks go in one launch, whatever the layout;
    more, tensors of one storage and plans on the host go through the two-pass form."""
    from fa2_custom_mask import functional, inv_permute_attn_triton, permute_qkv_triton

    class TwoPass(Exception):
        pass

    def two_pass(*args):
        raise TwoPass

    monkeypatch.setattr(functional, "apply_head_wise_reorder", two_pass)
    monkeypatch.setattr(functional, "apply_inv_reorder", two_pass)
    plan = {"permute": torch.arange(1, 4, device="cuda")[None]}

    def call(ts, F, H, W, text=0, plan=plan):
        grid = dict(F=F, H=H, W=W, n_text_tokens=text)
        permute_qkv_triton(*ts, plan, 0, **grid)
        inv_permute_attn_triton(ts[0], plan, 0, **grid)

    def tensors(T, D=64, dtype=torch.float16):
        return [torch.zeros(1, 3, T, D, device="cuda", dtype=dtype) for _ in range(3)]

    call(tensors(226 + 13 * 30 * 45), 13, 30, 45, 226)
    call(tensors(60, 128, torch.bfloat16), 3, 4, 5)
    call([t.transpose(1, 2).contiguous().transpose(1, 2) for t in tensors(60)], 3, 4, 5)
    for D in (64, 128):
        call(tensors(18432, D), 2, 96, 96)
        with pytest.raises(TwoPass):
            call(tensors(18434, D), 2, 13, 709)
    call(tensors(24576, 24), 4, 64, 96)               # 48-byte rows: one chunk
    fused = torch.zeros(1, 60, 3, 3, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(TwoPass):
        call([fused[:, :, i].transpose(1, 2) for i in range(3)], 3, 4, 5)
    with pytest.raises(TwoPass):
        call(tensors(60), 3, 4, 5, plan={"permute": torch.arange(1, 4)[None]})
