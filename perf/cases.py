"""What the framework's users have it do, as cases that can be timed: attention forward + backward of
a training step, attention forward of inference, the batched embedding of images, and the attention
step on host buffers, over the sizes of the repository's configurations and tests.

``listed()`` are the cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` makes
what a user's program has in hand before the call, ``run(state)`` is one pass through the public
entry points, ``work(case)`` what a pass cannot do without and ``tolerance(case)`` how far two correct
implementations at the same precision may differ.

A case is one of

* ``dense``: ``sdpa`` on ``batch`` x ``heads`` sequences of ``seqlen`` tokens, the drop-in for
  ``F.scaled_dot_product_attention``. ``memory`` is ``blhd`` (views of the projections' outputs, what
  ``modules.Attention`` hands over) or ``bhld`` (contiguous logical order);
* ``packed``: ``sdpa_varlen`` on ``batch`` sequences whose lengths are spread evenly over
  [``len_lo``, ``len_hi``], plus ``extra`` sequences of ``extra_len`` tokens (the seed decides their order);
* ``embed``: ``ViTMAE3D.embed_packed`` on ``batch`` images of a 128^3 volume's patch grid whose in-mask
  patch counts are spread evenly over [``len_lo``, ``len_hi``];
* ``host``: ``HostPipeline`` on pinned host tensors, lengths as for ``packed``.

``train`` cases run forward and backward, the others the forward under ``torch.inference_mode``.
"""

import math
import random

import torch

from nanobrain_b200 import HostPipeline, sdpa, sdpa_varlen
from nanobrain_b200.model import ViTMAE3D

HEAD_DIM = 64
DEV = "cuda"
GRID = (128, 128, 128)  # the embed cases' volume: 16^3 patches of 8^3 voxels
PATCHES, PATCH_DIM = 4096, 512
EMBED_DIM, DEPTH = 768, 12  # the ViT-B encoder (ViTMAE3D's defaults)


def _dense(batch, heads, seqlen, train=True, memory="blhd"):
    return {"kind": "dense", "batch": batch, "heads": heads, "seqlen": seqlen, "train": train, "memory": memory}


def _packed(batch, heads, len_lo, len_hi, train=True, extra=0, extra_len=0):
    return {"kind": "packed", "batch": batch, "heads": heads, "len_lo": len_lo, "len_hi": len_hi, "train": train,
            "extra": extra, "extra_len": extra_len}


def listed():
    named = {
        # The decoder of the tests' tiny model (6 sequences of a class token and 32 patches, 2 heads):
        # a call whose time is launches and host work.
        "tiny_dense_train": _dense(6, 2, 33),
        # Three short packed sequences, the smoke test's size: the same for the packed entry point.
        "tiny_packed_train": _packed(3, 2, 64, 150),
        # The CPU-checkable parity configuration (B=2, H=12, L=820) with contiguous [B, H, L, 64] memory.
        "check_dense_train": _dense(2, 12, 820, memory="bhld"),
        # One image per forward, the reference's evaluation loop: all in-mask patches and the class token.
        "image_dense_infer": _dense(1, 12, 3476, train=False),
        # ViT-B encoder attention of one training step: 32 volumes, about 80 % of 4096 patches masked.
        "encoder_packed_train": _packed(32, 12, 720, 920),
        # The same with the scaling configuration's global batch on one GPU.
        "encoder_b256_packed_train": _packed(256, 12, 720, 920),
        # Decoder attention over the full 4096-patch grid: the longest-running call.
        "decoder_dense_train": _dense(32, 8, 4096),
        # ViT-L-style encoder on the 20 x 24 x 20 grid.
        "vitl_packed_train": _packed(16, 16, 1700, 2140),
        # Sequences of very different lengths in one step: one long volume among thirty small ones.
        "skewed_packed_train": _packed(30, 12, 200, 200, extra=1, extra_len=2000),
        # Attention of a batched evaluation: eight images from one in-mask patch to 3475.
        "eval_packed_infer": _packed(8, 12, 1, 3475, train=False),
        # The whole batched evaluation: eight images through the ViT-B encoder in one packed pass.
        "embed_images": {"kind": "embed", "batch": 8, "len_lo": 1, "len_hi": 3475, "train": False},
        # Encoder attention for a caller whose tensors live in pinned host memory.
        "host_encoder_train": {"kind": "host", "batch": 32, "heads": 12, "len_lo": 720, "len_hi": 920, "train": True,
                               "extra": 0, "extra_len": 0},
    }
    return [dict(case, name=name) for name, case in named.items()]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random):
    """One more case: kinds weighted as listed, sizes over the logarithm of their range, heads as the
    encoder, decoder, ViT-L-style and test configurations have them. A drawn case stays below the
    largest listed ones in operations and in tokens."""
    most_flops, most_rows = work(_dense(32, 8, 4096))["flops"], 256 * 12 * 820
    while True:
        kind = rng.choices(("dense", "packed", "embed", "host"), (4, 6, 1, 1))[0]
        heads = rng.choice((2, 8, 12, 12, 16))
        if kind == "dense":
            case = _dense(_log_int(rng, 1, 32), heads, _log_int(rng, 13, 4500), rng.random() < 0.75,
                          rng.choice(("blhd", "blhd", "bhld")))
        elif kind == "packed":
            hi = _log_int(rng, 40, 3600)
            lo = _log_int(rng, 1, hi)
            extra = rng.choice((0, 0, 1, 2))
            case = _packed(_log_int(rng, 1, 256), heads, lo, hi, rng.random() < 0.75, extra,
                           _log_int(rng, 500, 4000) if extra else 0)
        elif kind == "embed":
            hi = _log_int(rng, 100, 4000)
            case = {"kind": "embed", "batch": _log_int(rng, 1, 8), "len_lo": _log_int(rng, 1, hi), "len_hi": hi,
                    "train": False}
        else:
            hi = _log_int(rng, 200, 1500)
            case = {"kind": "host", "batch": _log_int(rng, 2, 32), "heads": rng.choice((8, 12, 16)),
                    "len_lo": _log_int(rng, 100, hi), "len_hi": hi, "train": True, "extra": 0, "extra_len": 0}
        rows = case.get("heads", 12) * sum(_lengths(case))
        if rows <= most_rows / (1 if kind in ("dense", "packed") else 8) and work(case)["flops"] <= most_flops:
            return case


def _lengths(case):
    """Tokens of every sequence of a case, the same for every seed."""
    if case["kind"] == "dense":
        return [case["seqlen"]] * case["batch"]
    n, lo, hi = case["batch"], case["len_lo"], case["len_hi"]
    spread = [hi if n == 1 else lo + round(i * (hi - lo) / (n - 1)) for i in range(n)]
    return spread + [case["extra_len"]] * case.get("extra", 0) if case.get("extra") else spread


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).to(torch.bfloat16)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    lengths = _lengths(case)
    random.Random(seed).shuffle(lengths)
    train = case["train"]
    if case["kind"] == "embed":
        # The model that such a program keeps (random weights) and its images: patches and in-mask flags.
        with torch.random.fork_rng(devices=[torch.cuda.current_device()]), torch.device(DEV):
            torch.manual_seed(seed)
            model = ViTMAE3D(grid_size=GRID, patch_size=8).eval()
        samples = []
        for n in lengths:
            in_mask = torch.zeros(PATCHES, dtype=torch.bool, device=DEV)
            in_mask[torch.randperm(PATCHES, generator=gen, device=DEV)[:n]] = True
            samples.append((torch.randn(PATCHES, PATCH_DIM, generator=gen, device=DEV), in_mask))
        return {"kind": "embed", "model": model, "samples": samples}
    heads, total = case["heads"], sum(lengths)
    if case["kind"] == "host":
        ins = [_normal(gen, total, heads, HEAD_DIM).cpu().pin_memory() for _ in range(4)]
        outs = [torch.empty(total, heads, HEAD_DIM, dtype=torch.bfloat16, pin_memory=True) for _ in range(4)]
        return {"kind": "host", "pipe": HostPipeline(lengths, heads, torch.device(DEV, torch.cuda.current_device())),
                "ins": ins, "outs": outs}
    if case["kind"] == "dense":
        b, l = case["batch"], case["seqlen"]
        if case["memory"] == "blhd":
            q, k, v, g = (_normal(gen, b, l, heads, HEAD_DIM).transpose(1, 2) for _ in range(4))
        else:
            q, k, v, g = (_normal(gen, b, heads, l, HEAD_DIM) for _ in range(4))
        state = {"kind": "dense", "train": train}
    else:
        q, k, v, g = (_normal(gen, total, heads, HEAD_DIM) for _ in range(4))
        cu = torch.tensor([0] + lengths, device=DEV).cumsum(0).to(torch.int32)
        state = {"kind": "packed", "train": train, "cu": cu, "max_len": max(lengths)}
    if train:
        q, k, v = (t.requires_grad_(True) for t in (q, k, v))
        state["g"] = g
    state["qkv"] = (q, k, v)
    return state


def _attention(state):
    q, k, v = state["qkv"]
    if state["kind"] == "dense":
        return sdpa(q, k, v)
    cu, n = state["cu"], state["max_len"]
    return sdpa_varlen(q, k, v, cu, cu, n, n)


def run(state):
    if state["kind"] == "embed":
        return state["model"].embed_packed(state["samples"], return_dense=True)
    if state["kind"] == "host":
        state["pipe"].run(*state["ins"], *state["outs"])
        state["pipe"].wait()
        return state["outs"]
    if not state["train"]:
        with torch.inference_mode():
            return _attention(state)
    out = _attention(state)
    return (out, *torch.autograd.grad(out, state["qkv"], state["g"]))


def work(case):
    lengths = _lengths(case)
    if case["kind"] == "embed":
        # Every image's sequence starts with a class token. Weights and the in-mask patches are read
        # once, the dense grids (fp32) and the means are written once.
        tokens, pairs = sum(n + 1 for n in lengths), sum((n + 1) ** 2 for n in lengths)
        weights = DEPTH * 12 * EMBED_DIM ** 2 + PATCH_DIM * EMBED_DIM
        flops = 2 * weights * tokens + 4 * DEPTH * EMBED_DIM * pairs
        return {"bytes": 4 * (weights + PATCH_DIM * sum(lengths) + EMBED_DIM * (PATCHES + 1) * len(lengths)), "flops": flops}
    pairs = case["heads"] * sum(n * n for n in lengths)
    rows = case["heads"] * sum(lengths)
    # forward: Q, K, V in, O out, two products; training: dO in and dQ, dK, dV out too, seven products
    tensors, products = (8, 7) if case["train"] else (4, 2)
    return {"bytes": tensors * rows * HEAD_DIM * 2, "flops": 2 * products * HEAD_DIM * pairs}


def tolerance(case):
    # bf16 results of bf16 products with fp32 accumulation: a few roundings of 2^-9 each. The embedding
    # has twelve blocks of them in a row.
    return {"rel": 2e-2 if case["kind"] == "embed" else 1e-2}
