"""The native inference encoder behind ``embed_packed`` against the module-by-module path of the same
model (``forward_encoder`` per image under bf16 autocast), at row widths and patch counts where its
kernels have remainders, and the cases it has to leave to the modules."""

import pytest
import torch

from nanobrain_b200 import model as M
from nanobrain_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def build(heads, class_tokens, bias=True, grid=(24, 16, 20), patch=4, depth=2):
    torch.manual_seed(heads)
    model = M.ViTMAE3D(grid_size=grid, patch_size=patch, depth=depth, embed_dim=64 * heads, num_heads=heads,
                       decoder_depth=0, decoder_embed_dim=64, decoder_num_heads=1, qkv_bias=bias, proj_bias=bias,
                       class_tokens=class_tokens)
    for p in model.parameters():
        if p.dim() == 1:
            torch.nn.init.normal_(p, std=0.1)
    return model.to(DEV).eval()


def images(model, counts, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    p, d = model.coord_grid.shape[1], model.patch_embed.in_features
    out = []
    for n in counts:
        m = torch.zeros(p, dtype=torch.bool, device=DEV)
        m[torch.randperm(p, generator=g, device=DEV)[:n]] = True
        out.append((torch.randn(p, d, generator=g, device=DEV), m))
    return out


@pytest.mark.parametrize("heads,class_tokens,bias", [(1, 1, True), (2, 0, True), (3, 2, False), (11, 1, True), (16, 4, True)])
def test_native_encoder_matches_the_modules(heads, class_tokens, bias):
    model = build(heads, class_tokens, bias)
    samples = images(model, [1, 120, 63, 65, 7])
    assert model._native_encoder(samples) is not None
    outs = model.embed_packed(samples, return_dense=True)
    plain = model.embed_packed(samples)
    ops.check_status()
    for (patches, mask), out, short in zip(samples, outs, plain):
        with torch.inference_mode(), torch.autocast("cuda", dtype=torch.bfloat16):
            tokens = model.forward_encoder(patches[mask][None], model.coord_grid[:, mask])[0, class_tokens:].float()
        dense = out["dense_embedding"].reshape(-1, model.embed_dim)
        scale = tokens.abs().max()
        assert (dense[mask] - tokens).abs().max() <= 3e-2 * scale
        assert (dense[mask] - tokens).norm() <= 1e-2 * tokens.norm()
        assert bool((dense[~mask] == 0).all()) and torch.equal(out["dense_mask"].reshape(-1), mask)
        assert (out["global_embedding"] - dense[mask].mean(dim=0)).abs().max() <= 1e-4 * scale
        assert torch.equal(short["global_embedding"], out["global_embedding"]) and short["dense_embedding"] is None


def test_many_images_and_an_empty_one():
    model = build(1, 1, grid=(8, 8, 8))
    samples = images(model, [1 + i % 8 for i in range(70)])      # more than one call's worth of images
    outs = model.embed_packed(samples)
    for i in (0, 63, 64, 69):
        alone = model.embed_packed([samples[i]])[0]["global_embedding"]
        assert (alone - outs[i]["global_embedding"]).abs().max() <= 2e-2 * alone.abs().max()
    with pytest.raises(ValueError, match="in-mask"):
        model.embed_packed(samples[:2] + images(model, [0]))


def test_what_the_native_encoder_leaves_to_the_modules():
    model = build(2, 1)
    samples = images(model, [30, 40])
    want = [o["global_embedding"] for o in model.embed_packed(samples)]
    seen = []
    handle = model.blocks[0].attn.register_forward_hook(lambda *a: seen.append(1))
    assert model._native_encoder(samples) is None
    got = [o["global_embedding"] for o in model.embed_packed(samples)]
    handle.remove()
    assert seen and all((a - b).abs().max() <= 2e-2 * b.abs().max() for a, b in zip(got, want))
    assert model._native_encoder([(p.half(), m) for p, m in samples]) is None
    assert model.double()._native_encoder(samples) is None


@pytest.mark.parametrize("copies", [1, 65])
def test_gelu_of_every_bf16_value(copies):
    # all 65536 codes, by the formula and (many values) through the table: torch's bits
    import ctypes as C

    from nanobrain_b200 import _lib

    lib = _lib.load()
    lib.nb_enc_gelu.argtypes = [C.c_void_p, C.c_int64, C.c_void_p]
    v = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).to(DEV).repeat(copies)
    got = v.clone()
    assert lib.nb_enc_gelu(got.data_ptr(), got.numel(), torch.cuda.current_stream().cuda_stream) == 0
    want = torch.nn.functional.gelu(v)
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(got), nan) and torch.equal(got[~nan], want[~nan])


def alone(model, samples):
    """The reference's loop: one dense forward of the modules per image."""
    out = []
    for patches, mask in samples:
        with torch.inference_mode(), torch.autocast("cuda", dtype=torch.bfloat16):
            tokens = model.forward_encoder(patches[mask][None], model.coord_grid[:, mask])[0, model.class_tokens:].float()
        out.append(tokens.mean(0))
    return out


def flat_parameters(model, offset):
    """Every parameter a view of one buffer, `offset` elements past a 16-byte boundary."""
    params = [p for p in model.parameters()]
    flat = torch.empty(sum((p.numel() + 3) // 4 * 4 for p in params) + 4, device=DEV)
    at = offset
    for p in params:
        view = flat[at:at + p.numel()].view_as(p)
        view.copy_(p.data)
        p.data = view
        at += (p.numel() + 3) // 4 * 4


def without(model, names):
    for name in names:
        model.blocks[1].get_submodule(name.rsplit(".", 1)[0]).register_parameter(name.rsplit(".", 1)[1], None)


@pytest.mark.parametrize("change,native", [
    (lambda m: None, True),
    (lambda m: flat_parameters(m, 0), True),
    (lambda m: flat_parameters(m, 1), False),
    (lambda m: without(m, ["norm1.weight", "norm1.bias"]), False),
    (lambda m: without(m, ["norm2.bias"]), False),
    (lambda m: without(m, ["attn.k.bias"]), False),
    (lambda m: setattr(m.blocks[0], "mlp", M.Mlp(128, mlp_ratio=2.7, bias=True).to(DEV)), False),  # 345 columns
])
@pytest.mark.parametrize("counts", [[31, 40], [30, 41, 1]])
def test_parameters_that_the_kernels_do_not_take(change, native, counts):
    model = build(2, 1)
    change(model)
    samples = images(model, counts)
    assert (model._native_encoder(samples) is not None) == native
    got = model.embed_packed(samples)
    ops.check_status()
    for a, b in zip(got, alone(model, samples)):
        assert (a["global_embedding"] - b).abs().max() <= 3e-2 * b.abs().max()


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_patches_that_start_anywhere(offset):
    model = build(2, 1)
    samples = images(model, [31, 40])
    want = model.embed_packed(samples)
    moved = [(torch.empty(p.numel() + offset, device=DEV)[offset:].view_as(p).copy_(p), m) for p, m in samples]
    for a, b in zip(model.embed_packed(moved), want):
        assert torch.equal(a["global_embedding"], b["global_embedding"])


class Halved(torch.nn.Module):
    def forward(self, x):
        return x * 0.5


class Subclass(M.ViTMAE3D):
    def forward_encoder_packed(self, *args, **kwargs):
        x, *rest = super().forward_encoder_packed(*args, **kwargs)
        return (x * 0.5, *rest)


def replaced_forward(module):
    original = module.forward
    module.forward = lambda *args, **kwargs: original(*args, **kwargs) * 0.5


@pytest.mark.parametrize("change", [
    lambda m: replaced_forward(m.blocks[1].attn),
    lambda m: replaced_forward(m.blocks[1].mlp.fc2),
    lambda m: replaced_forward(m.norm),
    lambda m: setattr(m.blocks[0], "drop_path2", Halved()),
    lambda m: setattr(m, "__class__", Subclass),
], ids=["attn.forward", "fc2.forward", "norm.forward", "drop_path2", "subclass"])
def test_changed_modules_are_run(change):
    model = build(2, 1)
    samples = images(model, [31, 40])
    before = model.embed_packed(samples)
    change(model)
    assert model._native_encoder(samples) is None
    got = [o["global_embedding"] for o in model.embed_packed(samples)]
    # (alone() goes through forward_encoder, which the subclass does not change)
    want = [o["global_embedding"] * 0.5 for o in before] if type(model) is Subclass else alone(model, samples)
    for a, b, c in zip(got, want, before):
        assert (a - b).abs().max() <= 3e-2 * b.abs().max()
        assert (a - c["global_embedding"]).norm() > 0.05 * a.norm()


def test_compiled_and_watched_blocks_are_run():
    model = build(2, 1)
    samples = images(model, [31, 40])
    ran = []
    model.blocks[0].compile(backend=lambda graph, inputs: lambda *args: ran.append(1) or graph(*args))
    assert model._native_encoder(samples) is None
    model.embed_packed(samples)
    assert ran
    model = build(2, 1)
    handle = model.blocks[1].drop_path1.register_forward_hook(lambda *args: ran.append(2))
    model.embed_packed(samples)
    handle.remove()
    assert 2 in ran and model._native_encoder(samples) is not None
    drops = M.ViTMAE3D(grid_size=(24, 16, 20), patch_size=4, depth=2, embed_dim=128, num_heads=2, decoder_depth=0,
                       decoder_embed_dim=64, decoder_num_heads=1, drop_path_rate=0.5).to(DEV)
    assert drops.train()._native_encoder(samples) is None and drops.eval()._native_encoder(samples) is not None


def test_modes_see_the_operations():
    from torch.overrides import TorchFunctionMode
    from torch.utils.flop_counter import FlopCounterMode

    model = build(2, 1)
    samples = images(model, [31, 40])
    with FlopCounterMode(display=False) as counter:
        model.embed_packed(samples)
    rows, pairs = 31 + 40 + 2, 32 ** 2 + 41 ** 2
    assert counter.get_total_flops() == 2 * 71 * 64 * 128 + 2 * (2 * rows * 12 * 128 ** 2 + 4 * 128 * pairs)
    seen = []

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Mode():
        model.embed_packed(samples)
    assert torch.nn.functional.layer_norm in seen
    with torch.device(DEV):  # only places new tensors
        assert model._native_encoder(samples) is not None


def test_refused_parameters_leave_no_write_behind():
    # A refusal comes before anything is launched: the pinned words for the patch counts go back to their
    # allocator, and the next owner must not see a kernel write to them.
    model = build(2, 1)
    samples = images(model, [31, 40, 5])
    head, blocks, eps, heads = model._native_encoder(samples)
    coord = model.coord_grid[0].contiguous()
    patches, masks = [p for p, _ in samples], [m for _, m in samples]
    blocks = list(blocks)
    blocks[-6] = None  # norm2.weight of the last block
    torch.cuda._sleep(20_000_000)  # about 10 ms: what is launched now runs later
    with torch.inference_mode(), pytest.raises(RuntimeError, match="LayerNorm"):
        ops._load_native().encode_images(patches, masks, coord, head, blocks, eps, heads, False)
    words = [torch.full((3,), -7, dtype=torch.int32).pin_memory() for _ in range(4)]
    torch.cuda.synchronize()
    assert all(w.tolist() == [-7] * 3 for w in words)
