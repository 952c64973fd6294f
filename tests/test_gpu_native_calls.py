"""GPU: the native launch path (csrc/bind.cpp) is the one that takes a call in its plain form, and only that; and what test_gpu_native_path.py leaves out: a training
block's two halves on both paths."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]


@pytest.fixture
def taken(monkeypatch):
    """took(call): the native functions that answered during the call, and those that left it to the Python path."""
    from fovi_b200 import ops
    real = ops._native
    assert real is not None
    log = []

    class Counting:
        def __getattr__(self, name):
            def call(*args):
                got = getattr(real, name)(*args)
                log.append((name, got is not None))
                return got
            return call
    monkeypatch.setattr(ops, "_native", Counting())

    def took(call):
        log.clear()
        call()
        return [n for n, yes in log if yes], [n for n, yes in log if not yes]
    return took


def tables(n_in, n_out, K, V, seed=0):
    rs = np.random.RandomState(seed)
    return rs.randint(0, n_in + 1, (K, n_out)).astype(np.int32), rs.randint(0, V, (n_out, K)).astype(np.uint16)


def test_sampler(taken, golden):
    from fovi_b200 import ops
    plan = ops.SamplerPlan(golden("sensor_a1.npz")["sampling_grid"])
    rc, hw = torch.rand((4, 3, 2), device="cuda"), torch.full((4, 3, 2), 48.0, device="cuda")
    for dtype in (torch.float32, torch.bfloat16, torch.uint8):
        img = torch.randint(0, 255, (4, 3, 48, 60), device="cuda").to(dtype)
        for layout in range(6):
            for out in (None, torch.float32, torch.bfloat16):
                for i in (img, img[:, :, 3:, 1:], img.to(memory_format=torch.channels_last)):
                    assert taken(lambda: ops.sample(plan, i, rc, hw, out_dtype=out, layout=layout)) == (["sample"], [])
    assert taken(lambda: ops.sample(plan, img, rc.double(), hw)) == ([], ["sample"])
    assert taken(lambda: ops.sample(plan, img, rc, hw.transpose(0, 1).contiguous().transpose(0, 1))) == ([], ["sample"])
    assert taken(lambda: ops.sample(plan, img, rc, hw, out=torch.empty((4, 3, 3, plan.n_points), device="cuda"))) == ([], [])


@pytest.mark.parametrize("c_in,c_out,B", [(3, 64, 130), (16, 32, 7), (64, 64, 200)])
def test_layers(taken, c_in, c_out, B):
    from fovi_b200 import grad, ops
    n_in, n_out, V = 90, 24, 16
    idx, tap = tables(n_in, n_out, 9, V)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, c_in, c_out)
    x, w, b = torch.randn((B, c_in, n_in), device="cuda"), torch.randn((c_out, c_in * V), device="cuda"), torch.randn(c_out, device="cuda")
    pairs = plan.x_layout == ops.X_PAIRS
    for dt in (torch.float32, torch.bfloat16):
        assert taken(lambda: ops.pack_points(x.to(dt), plan)) == (["pack_points"], [])
        assert taken(lambda: plan.pack_weights(w.to(dt))) == (([], []) if pairs else (["pack_slabs"], []))       # (the pair layout's filter: the Python path)
        wt32 = plan.pack_weights(w, dtype=torch.float32)
        assert taken(lambda: plan.forward_f32(x.to(dt), wt32, b)) == (["conv_forward_f32"], [])
        xp, wt = ops.pack_points(x, plan), plan.pack_weights(w)
        for bias in (None, b):
            assert taken(lambda: plan.forward(xp, wt, bias, relu=True, out_dtype=dt, batch=B)) == (["conv_forward"], [])
    assert taken(lambda: plan.forward(xp, wt, b.double(), batch=B)) == ([], ["conv_forward"])
    assert taken(lambda: plan.forward(xp, wt, b.repeat_interleave(2)[::2], batch=B)) == ([], ["conv_forward"])
    assert taken(lambda: plan.forward_f32(x.permute(0, 2, 1).contiguous().permute(0, 2, 1), wt32, b)) == ([], ["conv_forward_f32"])
    assert taken(lambda: ops.pack_points(x.permute(0, 2, 1).contiguous().permute(0, 2, 1), plan)) == ([], ["pack_points"])
    assert taken(lambda: plan.forward(xp, wt, batch=B, out=torch.empty((B, n_out, c_out), device="cuda", dtype=torch.bfloat16))) == ([], [])
    if not pairs:
        g = grad.KnnConvGrad(idx, tap, n_in, V, c_in, c_out, torch.device("cuda"))
        gy = torch.randn((B, n_out, c_out), device="cuda").to(torch.bfloat16)
        assert taken(lambda: g.input_grad(gy, w)) == (["pack_slabs", "conv_forward"], [])
        assert taken(lambda: g.weight_grad(gy, xp, plan)) == (["weight_grad"], [])
        assert taken(lambda: g.weight_grad(gy, xp, plan, torch.bfloat16)) == (["weight_grad"], [])


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("pooled", [True, False])
@pytest.mark.parametrize("B,N,C", [(7, 50, 32), (40, 61, 144)])
def test_block_halves_on_both_paths(taken, monkeypatch, B, N, C, pooled, relu):
    from fovi_b200 import ops
    from fovi_b200.norm import KNNBatchNorm
    gen = torch.Generator(device="cuda").manual_seed(B)
    y = torch.randn((B, N, C), generator=gen, device="cuda")
    pool = ops.KnnPoolPlan(tables(N, 12, 5, 1)[0], N, device="cuda") if pooled else None
    n_out = 12 if pooled else N
    g = torch.randn((B, n_out, C), generator=gen, device="cuda")
    results = []

    def run():
        norm = KNNBatchNorm(N, C).train()
        with torch.no_grad():
            norm.weight.copy_(torch.linspace(0.5, 1.5, C))
            norm.bias.copy_(torch.linspace(-1, 1, C))
            mean, rstd, out, arg = ops.block_forward(y, norm, relu, pool)
            act = out if relu and not pooled else None
            results.append([mean, rstd, out] + ([arg] if pooled else []) + list(norm.buffers()) + list(ops.norm_block_backward(y, mean, rstd, norm.weight, act, g, pool, arg)))
        assert (arg is not None) == pooled
    assert taken(run) == (["block_forward", "block_backward"], [])
    monkeypatch.setattr(ops, "_native", None)
    assert taken(run) == ([], [])
    for a, b in zip(*results, strict=True):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)


# three layers; where the masked kernel runs only the top layer's gradient is masked and summed on its own
@pytest.mark.parametrize("rows,separate", [(200, 1), (40, 3), (129, 1)])
def test_stack_masks_in_the_kernel(monkeypatch, rows, separate):
    from fovi_b200 import grad, ops
    from fovi_b200.coords import get_in_out_coords
    from fovi_b200.knn import KNNConvLayer, KNNConvStack
    ic, oc, _ = get_in_out_coords(20, 16, 1.0, 2, auto_match_cart_resources=0)
    stack = KNNConvStack([KNNConvLayer(3, 64, 9, ic, oc, device="cuda", ref_frame_side_length=3, bias=True),
                          KNNConvLayer(64, 96, 9, oc, oc, device="cuda", ref_frame_side_length=3, bias=True),
                          KNNConvLayer(96, 32, 9, oc, oc, device="cuda", ref_frame_side_length=3, bias=True)], final_relu=True)
    calls, kernel = [], []
    mask, masked = ops.relu_mask_colsum, grad.KnnConvGrad.input_grad_masked
    monkeypatch.setattr(ops, "relu_mask_colsum", lambda *a: calls.append(1) or mask(*a))

    def count(*a):
        got = masked(*a)
        kernel.append(got is not None)
        return got
    monkeypatch.setattr(grad.KnnConvGrad, "input_grad_masked", count)
    stack(torch.randn((rows, 3, len(ic)), device="cuda").to(torch.bfloat16)).square().mean().backward()
    assert len(calls) == separate and kernel == [separate == 1] * 2
