"""GPU: the exact float32 kernel with four points per warp (layers of at most 4 channels, more than two images) where its warps take several quads of points, and on
both sides of the rule that chooses it.  A run two images at a time takes the kernel with a point per warp, whose sums are the same bit for bit; that one is compared with
the oracle in test_gpu_knnconv_f32_few.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def layer(cin, cout, K, side, n_out, n_in=400, seed=0):
    from fovi_b200 import ops
    rs = np.random.RandomState(seed + n_out + cout)
    idx = rs.randint(0, n_in, (K, n_out)).astype(np.int32)
    idx[rs.rand(K, n_out) < 0.1] = n_in                                # lists of different lengths in one warp
    idx[:, n_out // 2] = n_in
    plan = ops.KnnConvPlan(idx, rs.randint(0, side * side, (n_out, K)).astype(np.uint16), n_in, side * side, cin, cout, group=1)
    return plan, plan.pack_weights(torch.from_numpy(rs.standard_normal((cout, cin * side * side)).astype(np.float32)).cuda(), dtype=torch.float32)


def kernels(call):
    """Names of the kernels that a call launches; None where no profiler is to be had."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return " ".join(e.key for e in p.key_averages()) or None


def compare(plan, wt, x, relu=False):
    from fovi_b200 import ops
    bias = torch.randn(plan.c_out, device="cuda")
    for xl in (ops.ACT_BCN, ops.ACT_BNC):
        xin = x if xl == ops.ACT_BCN else x.transpose(1, 2).contiguous()
        for yl in (ops.ACT_BCN, ops.ACT_BNC):
            got = plan.forward_f32(xin, wt, bias, relu=relu, x_layout=xl, y_layout=yl)
            want = torch.cat([plan.forward_f32(xin[b:b + 2], wt, bias, relu=relu, x_layout=xl, y_layout=yl) for b in range(0, len(x), 2)])
            assert torch.equal(got, want), (xl, yl)


# More quads than the chip has warps (148 SMs x 12 or 16), the last tile of images with one image, last quads of one, two and three points; lists of one pass and
# of one neighbour more or less; channel tiles of 32, 64 and 96, and several of them
@pytest.mark.parametrize("cin,cout,K,n_out,B,dtype", [
    (3, 32, 7, 2001, 41, torch.float32), (3, 64, 8, 2002, 41, torch.float32), (3, 96, 15, 2003, 41, torch.float32), (4, 64, 9, 2003, 41, torch.bfloat16),
    (4, 96, 16, 2001, 41, torch.float32), (1, 64, 25, 3002, 41, torch.float32), (2, 33, 9, 3001, 41, torch.bfloat16), (4, 160, 7, 1001, 25, torch.float32),
    (3, 64, 9, 12003, 4, torch.float32), (3, 96, 8, 12002, 3, torch.float32), (1, 32, 9, 14001, 3, torch.float32)])
def test_many_quads_equal_the_other_kernel(cin, cout, K, n_out, B, dtype):
    plan, wt = layer(cin, cout, K, 5, n_out)
    x = torch.randn((B, cin, 400), device="cuda").to(dtype)
    tiles = {32: 1, 33: 1, 64: 1, 96: 1, 160: 5}[cout]                 # (33 channels take a tile of 64)
    assert (n_out + 3) // 4 * -(-B // (8 if B > 4 else 4)) * tiles > 148 * 16
    compare(plan, wt, x, relu=cout == 64)
    ran = kernels(lambda: plan.forward_f32(x, wt))
    assert ran is None or "f32_quad" in ran


# tiles of eight points per SM of a 148-SM chip, on both sides of 1 (4 channels; 96 values gathered; 48 for a tile of 32 channels), 2 (3 channels; 96-channel tiles;
# 2 -> 32) and 3 (the rest), and behind the second round of the quad kernel's warps; long lists
# of 4 channels; two images and a large filter
@pytest.mark.parametrize("cin,cout,K,side,n_out,B,quad", [
    (3, 64, 25, 5, 1184, 8, False), (3, 64, 25, 5, 1185, 8, True), (4, 64, 9, 3, 1184, 8, False), (4, 64, 9, 3, 1185, 8, True), (3, 32, 9, 3, 1185, 8, True),
    (2, 32, 25, 5, 1185, 8, True), (3, 64, 9, 3, 2368, 8, False), (3, 64, 9, 3, 2369, 8, True), (3, 96, 9, 3, 964, 8, False), (2, 96, 9, 3, 2368, 4, False),
    (2, 96, 9, 3, 2369, 4, True), (2, 32, 9, 3, 2368, 4, False), (2, 32, 9, 3, 2369, 4, True), (1, 64, 9, 3, 3552, 8, False), (1, 64, 9, 3, 3553, 8, True),
    (1, 64, 9, 3, 3700, 16, False), (1, 64, 9, 3, 4200, 16, True), (3, 64, 49, 7, 7, 3, False), (4, 160, 49, 7, 7, 8, True), (4, 160, 41, 7, 30, 4, False),
    (3, 64, 25, 5, 9000, 2, False), (3, 96, 25, 9, 4000, 8, False)])
def test_both_sides_of_the_rule(cin, cout, K, side, n_out, B, quad):
    plan, wt = layer(cin, cout, K, side, n_out)
    x = torch.randn((B, cin, 400), device="cuda")
    compare(plan, wt, x)
    ran = kernels(lambda: plan.forward_f32(x, wt))
    if ran is not None and torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert ("f32_quad" in ran) == quad, ran
