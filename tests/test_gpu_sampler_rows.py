"""GPU: the general sampler's forms for many rows (one CTA per row, staged; points-major rows in 16-byte pieces) against the form that few rows take:
the same images in one call and in slices of a few give the same bits.  Slices are compared with the oracle elsewhere (test_gpu_sampler.py); one row is here too."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu
DT = {"f32": torch.float32, "bf16": torch.bfloat16, "u8": torch.uint8}


# (in, out, channels, height, width, images, fixations, mode, pad, layout, channel stride): rows from the first count that takes the new form; images at an odd
# width, so that no strip kernel applies; odd point counts; rows of the result that start on no 16-byte boundary
@pytest.mark.parametrize("sensor,din,dout,C,H,W,B,F,mode,pad,layout,cp", [
    ("a1", "f32", "f32", 3, 151, 199, 370, 2, "bilinear", "zeros", "BFCN", None), ("a2p78", "f32", "f32", 3, 151, 199, 247, 3, "bilinear", "border", "FBCN", None),
    ("a2p78", "bf16", "bf16", 3, 331, 335, 186, 4, "bilinear", "zeros", "BFCN", None), ("a1", "u8", "f32", 3, 231, 235, 371, 4, "bilinear", "zeros", "BFCN", None),
    ("a1", "f32", "bf16", 4, 151, 199, 740, 1, "bilinear", "border", "BFCN", None), ("a1", "f32", "f32", 2, 351, 399, 185, 4, "bilinear", "zeros", "BFCN", None),
    ("a1", "bf16", "bf16", 8, 71, 73, 241, 4, "bilinear", "zeros", "BFCN", None), ("a1", "f32", "f32", 3, 291, 299, 185, 8, "nearest", "border", "BFCN", None),
    ("a1", "f32", "f32", 3, 251, 239, 370, 2, "bilinear", "zeros", "CL", None), ("a2p78", "f32", "bf16", 3, 401, 451, 185, 8, "bilinear", "zeros", "PAIRS", None),
    ("a2p78", "f32", "bf16", 4, 401, 451, 185, 8, "nearest", "border", "PAIRS", None), ("a2p78", "bf16", "bf16", 9, 61, 63, 111, 2, "bilinear", "zeros", "BFNC", 11),
    ("a1", "f32", "f32", 3, 61, 63, 370, 4, "bilinear", "zeros", "FBNC", 3), ("a1", "bf16", "bf16", 3, 61, 63, 370, 4, "nearest", "zeros", "BFNC", 5),
    # 16-byte pieces: one and several per point, channels that fill them, do not, and end on a multiple of four
    ("a2p78", "bf16", "bf16", 1, 61, 63, 33, 1, "bilinear", "zeros", "BFNC", 8), ("a1", "f32", "f32", 3, 61, 63, 17, 2, "bilinear", "border", "FBNC", 8),
    ("a1", "u8", "bf16", 3, 61, 63, 17, 2, "nearest", "zeros", "BFNC", 8), ("a2p78", "f32", "bf16", 21, 31, 33, 17, 2, "bilinear", "zeros", "BFNC", 24),
    ("a1", "bf16", "f32", 12, 31, 33, 17, 2, "nearest", "border", "BFNC", 12), ("a1", "f32", "f32", 64, 31, 33, 40, 1, "bilinear", "zeros", "BFNC", 64)])
def test_one_call_equals_its_slices(golden, sensor, din, dout, C, H, W, B, F, mode, pad, layout, cp):
    from fovi_b200 import ops
    grid = golden(f"sensor_{sensor}.npz")["sampling_grid"]
    plan = ops.SamplerPlan(grid)
    gen = torch.Generator(device="cuda").manual_seed(H * W)
    shape = (B, H, W, C) if layout == "CL" else (B, C, H, W)
    img = torch.randint(0, 256, shape, generator=gen, device="cuda").to(DT[din]) if din == "u8" else torch.randn(shape, generator=gen, device="cuda").to(DT[din])
    if layout == "CL":
        img = img.permute(0, 3, 1, 2)
    fix = -0.2 + 1.4 * torch.rand((B, F, 2), generator=gen, device="cuda")          # some fixations look past the image
    hw = min(H, W) * (0.5 + torch.rand((B, F, 2), generator=gen, device="cuda"))
    kw = dict(mode=ops.BILINEAR if mode == "bilinear" else ops.NEAREST, pad=ops.PAD_ZEROS if pad == "zeros" else ops.PAD_BORDER)
    few = max(1, 16 // F)                                                            # images per slice
    if layout == "PAIRS":
        n_pairs = (plan.n_points + 1) // 2
        out = torch.zeros(((B * F + 127) // 128, n_pairs, 128, 8), dtype=torch.bfloat16, device="cuda")
        ops.sample(plan, img, fix, hw, layout=ops.OUT_BF_PAIRS, out=out, **kw)
        rows = out.permute(0, 2, 1, 3).reshape(-1, n_pairs, 8)
        for lo in range(0, B, few):
            hi = min(B, lo + few)
            part = torch.zeros((1, n_pairs, 128, 8), dtype=torch.bfloat16, device="cuda")
            ops.sample(plan, img[lo:hi], fix[lo:hi], hw[lo:hi], layout=ops.OUT_BF_PAIRS, out=part, **kw)
            assert torch.equal(rows[lo * F:hi * F], part[0].permute(1, 0, 2)[:(hi - lo) * F])
        assert not rows[B * F:].any()
        return
    code = {"BFCN": ops.OUT_BFCN, "CL": ops.OUT_BFCN, "FBCN": ops.OUT_FBCN, "BFNC": ops.OUT_BFNC, "FBNC": ops.OUT_FBNC}[layout]
    if cp is not None:
        kw["channel_stride"] = cp
    out = ops.sample(plan, img, fix, hw, out_dtype=DT[dout], layout=code, **kw)
    for lo in range(0, B, few):
        hi = min(B, lo + few)
        part = ops.sample(plan, img[lo:hi], fix[lo:hi], hw[lo:hi], out_dtype=DT[dout], layout=code, **kw)
        assert torch.equal(out[:, lo:hi] if layout.startswith("F") else out[lo:hi], part)
    if layout in ("BFCN", "CL") and dout == "f32":
        ref = oracle.retinal_sample(img[B - 1:].float().cpu().numpy(), grid, fix[B - 1:].cpu().numpy(), hw[B - 1:].cpu().numpy(), mode=mode, padding=pad)
        assert np.array_equal(out[B - 1:].cpu().numpy(), ref)
