"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call (or one forward and backward) of the public entry points: the block-sparse
attention op `flash_attention_custom_mask` and the head-wise token reorder around it.  `listed()`
names the cases, `draw()` gives more of the same ranges, `prepare()` makes what a program holds before
the call, `run()` is the call, `work()` and `tolerance()` say what it needs and how exact it is.

Fields of an attention case: op ("forward" or "train"), dtype, B, H, N, D; layout of q, k, v (and dO)
in memory ("bhnd": contiguous [B,H,N,D]; "bnhd": what a projection of [B,N,H*D] leaves; "qkv":
slices of one fused [B,N,3,H,D] projection); mask ("block": a 64x64 block mask for every head,
"shared": one block mask for all heads, "dense": a shared [N,N] mask made of whole blocks,
"token-causal": such a block mask cut along the diagonal element by element, shared); density of the
blocks; diagonal (diagonal blocks forced on); causal (blocks above the diagonal off).
Fields of a reorder case: op "reorder", dtype, B, H (heads), F, Y, X (the token grid), text (tokens
before it that stay), D.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "customize-block-sparse-attention-with-triton_b200"))

from fa2_custom_mask import (  # noqa: E402
    flash_attention_custom_mask, inv_permute_attn_triton, permute_qkv_triton)

BLOCK = 64
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _attention(name, op, dtype, B, H, N, D=64, layout="bhnd", mask="block", density=0.1,
               diagonal=True, causal=False):
    case = dict(op=op, dtype=dtype, B=B, H=H, N=N, D=D, layout=layout, mask=mask, density=density,
                diagonal=diagonal, causal=causal)
    return dict(case, name=name) if name else case


def _reorder(name, dtype, B, H, F, Y, X, text, D=64):
    case = dict(op="reorder", dtype=dtype, B=B, H=H, F=F, Y=Y, X=X, text=text, D=D)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: one short head, where launches and the host path are all there is
        _attention("forward_1k", "forward", "fp16", 1, 1, 1024),
        # a caller that holds an ordinary dense boolean mask and no block mask
        _attention("forward_6k_dense_mask", "forward", "fp16", 1, 1, 6400, mask="dense"),
        # the headline: one head of a long sequence at a tenth of the blocks
        _attention("forward_17k", "forward", "fp16", 1, 1, 17536),
        # the same head with nothing masked out: long lists, all tiles
        _attention("forward_17k_full", "forward", "fp16", 1, 1, 17536, density=1.0),
        # a layer of the reference's own check: eight heads with masks of their own, rows may be empty
        _attention("forward_17k_8_heads", "forward", "fp16", 1, 8, 17536, diagonal=False),
        # the largest inference call: a whole layer over a very long sequence
        _attention("forward_32k_32_heads", "forward", "bf16", 1, 32, 32000),
        # a small model with narrow heads, an odd number of blocks and one mask for all heads
        _attention("forward_4k_narrow_heads", "forward", "fp16", 2, 12, 4160, D=32, mask="shared",
                   density=0.25),
        # one training step of a short sequence: launches and autograd
        _attention("train_1k", "train", "bf16", 1, 2, 1024),
        # a training step on q, k, v as a projection leaves them, block-causal, one mask for all heads
        _attention("train_4k_projected", "train", "bf16", 2, 8, 4160, layout="bnhd", mask="shared",
                   density=0.25, causal=True),
        # a training step with a mask whose diagonal blocks are cut element by element
        _attention("train_6k_token_causal", "train", "fp16", 1, 4, 6400, mask="token-causal",
                   density=0.25, causal=True),
        # the largest training step: two sequences, sixteen heads, block-causal masks of their own
        _attention("train_16k_16_heads", "train", "bf16", 2, 16, 16384, density=0.25, causal=True),
        # the reorder around an attention layer of a video model: 13 x 30 x 45 tokens behind 226 of text
        _reorder("reorder_video_48_heads", "fp16", 2, 48, 13, 30, 45, 226),
    ]


# At most this much work in a drawn case: listed 64x64 tiles times matrix products over them (2 in a
# forward, 7 in a training step), and bytes of one tensor of a reorder.  The largest listed cases have
# 1.9 million of the one and 218 MB of the other.
_MOST_PRODUCTS = 1.5e6
_MOST_REORDER_BYTES = 2.0e8


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    if rng.random() < 0.12:
        while True:
            case = _reorder(None, rng.choice(["fp16", "bf16"]), rng.choice([1, 2]),
                            _log_int(rng, 2, 48), rng.randint(2, 17), rng.randint(6, 48),
                            rng.randint(6, 64), rng.choice([0, rng.randint(1, 300)]),
                            rng.choice([64, 64, 128]))
            if _elements(case) * 2 <= _MOST_REORDER_BYTES:
                return case
    while True:
        mask = rng.choice(["block", "block", "block", "shared", "dense", "token-causal"])
        elements = mask in ("dense", "token-causal")
        case = _attention(
            None, rng.choice(["forward", "train"]), rng.choice(["fp16", "bf16"]),
            rng.choice([1, 1, 2]), _log_int(rng, 1, 8 if elements else 32),
            BLOCK * _log_int(rng, 8, 274 if elements else 500), rng.choice([64] * 8 + [32, 16]),
            rng.choice(["bhnd", "bhnd", "bnhd", "qkv"]), mask,
            rng.choice([1.0] + [round(math.exp(rng.uniform(math.log(0.05), 0.0)), 3)] * 5),
            rng.random() < 0.8, mask == "token-causal" or rng.random() < 0.4)
        # a forward without a diagonal may leave rows empty, as the reference's check does; a training
        # step on such a mask is no use to anybody
        case["diagonal"] = case["diagonal"] or case["op"] == "train" or case["causal"]
        if _tiles(case) * (2 if case["op"] == "forward" else 7) <= _MOST_PRODUCTS:
            return case


def _elements(case):
    """Elements of one of the case's tensors (for a reorder those that move)."""
    tokens = case["F"] * case["Y"] * case["X"] if case["op"] == "reorder" else case["N"]
    return case["B"] * case["H"] * tokens * case["D"]


def _tiles(case):
    """How many 64x64 blocks all heads list, on average."""
    nb, p = case["N"] // BLOCK, case["density"]
    off = nb * (nb - 1) * p * (0.5 if case["causal"] else 1.0)
    return case["B"] * case["H"] * (off + nb * (1.0 if case["diagonal"] else p))


def _block_mask(case, g):
    nb = case["N"] // BLOCK
    heads = (case["B"], case["H"]) if case["mask"] == "block" else (1, 1)
    m = torch.rand(*heads, nb, nb, device="cuda", generator=g) < case["density"]
    if case["diagonal"]:
        m |= torch.eye(nb, dtype=torch.bool, device="cuda")
    return torch.tril(m) if case["causal"] else m


def _tensors(case, n, g):
    """n tensors [B,H,N,D] of standard normal values in the case's layout."""
    B, H, N, D, dtype = case["B"], case["H"], case["N"], case["D"], DTYPES[case["dtype"]]
    if case["layout"] == "bhnd":
        return [torch.randn(B, H, N, D, device="cuda", generator=g, dtype=dtype) for _ in range(n)]
    got = []
    if case["layout"] == "qkv":
        fused = torch.randn(B, N, 3, H, D, device="cuda", generator=g, dtype=dtype)
        got = [fused[:, :, i].transpose(1, 2) for i in range(3)]
    return got + [torch.randn(B, N, H, D, device="cuda", generator=g, dtype=dtype).transpose(1, 2)
                  for _ in range(n - len(got))]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["op"] == "reorder":
        tokens = case["text"] + case["F"] * case["Y"] * case["X"]
        q, k, v, o = (torch.randn(case["B"], case["H"], tokens, case["D"], device="cuda",
                                  generator=g, dtype=DTYPES[case["dtype"]]) for _ in range(4))
        # one axis order of six for every head, as a plan made beforehand says
        plan = {"permute": torch.randint(0, 6, (1, case["H"]), device="cuda", generator=g)}
        grid = dict(F=case["F"], H=case["Y"], W=case["X"], n_text_tokens=case["text"])
        return {"op": "reorder", "qkv": (q, k, v), "o": o, "plan": plan, "grid": grid}
    train = case["op"] == "train"
    ts = _tensors(case, 4 if train else 3, g)
    mask = _block_mask(case, g)
    if case["mask"] in ("dense", "token-causal"):
        mask = mask.repeat_interleave(BLOCK, -2).repeat_interleave(BLOCK, -1)
    if case["mask"] == "token-causal":
        mask = torch.tril(mask)
    qkv = tuple(t.detach().requires_grad_(train) for t in ts[:3])
    return {"op": case["op"], "qkv": qkv, "mask": mask, "scale": case["D"] ** -0.5,
            "dout": ts[3] if train else None}


def run(state):
    if state["op"] == "reorder":
        q, k, v = permute_qkv_triton(*state["qkv"], state["plan"], 0, **state["grid"])
        return [q, k, v, inv_permute_attn_triton(state["o"], state["plan"], 0, **state["grid"])]
    q, k, v = state["qkv"]
    o = flash_attention_custom_mask(q, k, v, state["mask"], state["scale"])
    if state["op"] == "forward":
        return o
    return [o, *torch.autograd.grad(o, (q, k, v), state["dout"])]


def work(case):
    if case["op"] == "reorder":
        return {"bytes": 4 * 2 * 2 * _elements(case), "flops": 0}  # q, k, v and the output, there and back
    train, nb = case["op"] == "train", case["N"] // BLOCK
    masks = case["B"] * case["H"] if case["mask"] == "block" else 1
    mask_bytes = masks * (case["N"] ** 2 if case["mask"] in ("dense", "token-causal") else nb * nb)
    kept = _tiles(case) * BLOCK * BLOCK
    if case["mask"] == "token-causal":  # of a diagonal block only the lower triangle is kept
        kept -= case["B"] * case["H"] * nb * BLOCK * (BLOCK - 1) / 2
    # forward: q, k, v in, o out; training: dO in and dq, dk, dv out as well.  A forward has two matrix
    # products over the kept elements, the backward five more.
    return {"bytes": (8 if train else 4) * 2 * _elements(case) + mask_bytes,
            "flops": (14 if train else 4) * case["D"] * kept}


def tolerance(case):
    if case["op"] == "reorder":
        return "exact"
    # probabilities (and, backward, dS) are rounded to the tensors' type before the second product
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
