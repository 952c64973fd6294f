"""GPU: the sampler's kernel shapes against each other and the oracle, bit for bit.  An image whose rows start on no 16-byte boundary takes the
general kernel, the same image in its own memory the strip kernel in the shape its size calls for: every form has to give the same bits."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


# tall strips (large planar batches: the coarse visiting orders) with one tensor copy per strip, with row copies (rows of 2048 bytes), with a short last
# strip, with windowed columns (rows of 8 KB); low strips with the tensor copy (large batches) and without (small ones); every dtype, mode, padding, layout
@pytest.mark.parametrize("dtype,H,W,B,F,mode,pad,layout", [
    ("f32", 256, 64, 340, 3, "bilinear", "zeros", "BFCN"), ("f32", 250, 64, 360, 1, "nearest", "zeros", "BFCN"), ("bf16", 300, 72, 400, 2, "bilinear", "border", "FBCN"),
    ("u8", 512, 48, 200, 2, "bilinear", "zeros", "BFCN"), ("f32", 128, 512, 110, 2, "bilinear", "zeros", "BFCN"), ("f32", 40, 2048, 3, 2, "bilinear", "zeros", "BFCN"),
    ("f32", 96, 128, 100, 2, "bilinear", "zeros", "PAIRS"), ("bf16", 97, 136, 130, 17, "nearest", "border", "BFNC"), ("u8", 64, 64, 2, 4, "bilinear", "zeros", "PAIRS"),
    ("f32", 33, 68, 1, 1, "bilinear", "border", "BFCN")])
def test_every_shape_gives_the_same_bits(golden, dtype, H, W, B, F, mode, pad, layout):
    from fovi_b200 import ops
    grid = golden("sensor_a1.npz")["sampling_grid"]
    plan = ops.SamplerPlan(grid)
    gen = torch.Generator(device="cuda").manual_seed(H * W)
    tdt = {"f32": torch.float32, "bf16": torch.bfloat16, "u8": torch.uint8}[dtype]
    img = torch.randint(0, 256, (B, 3, H, W), generator=gen, device="cuda").to(tdt) if dtype == "u8" else \
        torch.randn((B, 3, H, W), generator=gen, device="cuda").to(tdt)
    odd = torch.zeros((B, 3, H, W + 1), dtype=tdt, device="cuda")
    odd[..., :W] = img
    fix = -0.2 + 1.4 * torch.rand((B, F, 2), generator=gen, device="cuda")          # some fixations look past the image
    hw = min(H, W) * (0.5 + torch.rand((B, F, 2), generator=gen, device="cuda"))
    kw = dict(mode=ops.BILINEAR if mode == "bilinear" else ops.NEAREST, pad=ops.PAD_ZEROS if pad == "zeros" else ops.PAD_BORDER)
    if layout == "PAIRS":
        shape = ((B * F + 127) // 128, (plan.n_points + 1) // 2, 128, 8)
        a, b = (torch.zeros(shape, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        ops.sample(plan, img, fix, hw, layout=ops.OUT_FB_PAIRS, out=a, **kw)
        ops.sample(plan, odd[..., :W], fix, hw, layout=ops.OUT_FB_PAIRS, out=b, **kw)
    else:
        out_dtype = torch.bfloat16 if layout == "BFNC" else torch.float32
        code = {"BFCN": ops.OUT_BFCN, "FBCN": ops.OUT_FBCN, "BFNC": ops.OUT_BFNC}[layout]
        a = ops.sample(plan, img, fix, hw, out_dtype=out_dtype, layout=code, **kw)
        b = ops.sample(plan, odd[..., :W], fix, hw, out_dtype=out_dtype, layout=code, **kw)
    plan.check()
    assert torch.equal(a, b)
    if layout == "BFCN":
        some = sorted({0, B // 2, B - 1})
        ref = oracle.retinal_sample(img[some].float().cpu().numpy(), grid, fix[some].cpu().numpy(), hw[some].cpu().numpy(), mode=mode, padding=pad)
        assert np.array_equal(a[some].cpu().numpy(), ref)
