"""GPU: the native launch path (csrc/bind.cpp) and the Python path it stands in for give the same tensors for every form the native one accepts, and what the
Python path refuses is refused."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def both(monkeypatch):
    from fovi_b200 import ops
    assert ops._native is not None

    def run(call):
        got = call(ops)
        with monkeypatch.context() as m:
            m.setattr(ops, "_native", None)
            want = call(ops)
        flat = lambda t: list(t) if isinstance(t, tuple) else [t]      # noqa: E731
        for a, b in zip(flat(got), flat(want), strict=True):
            assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and a.device == b.device and torch.equal(a, b)
    return run


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.uint8])
def test_sample(both, golden, dtype):
    from fovi_b200 import ops
    plan = ops.SamplerPlan(golden("sensor_a1.npz")["sampling_grid"])
    img = torch.randint(0, 255, (4, 3, 48, 60), device="cuda").to(dtype)
    rc, hw = torch.rand((4, 3, 2), device="cuda"), torch.full((4, 3, 2), 48.0, device="cuda")
    for layout in range(6):
        for out in (None, torch.float32, torch.bfloat16):
            for stride in (None, 8):
                rows = slice(12 if layout >= 4 else None)               # the pair layout's rows past the batch are left unwritten
                for i in (img, img[:, :, 3:, 1:], img.to(memory_format=torch.channels_last)):
                    both(lambda o: o.sample(plan, i, rc, hw, mode=o.NEAREST, out_dtype=out, layout=layout, channel_stride=stride)[:, :, rows])
    both(lambda o: o.sample(plan, img, rc.double(), hw.transpose(0, 1).contiguous().transpose(0, 1)))
    for bad, error in ((dict(img=img.cpu()), ValueError), (dict(img=img.half()), TypeError), (dict(rc=rc[:2]), AssertionError), (dict(img=img[0]), ValueError)):
        a = dict(img=img, rc=rc, hw=hw) | bad
        with pytest.raises(error):
            ops.sample(plan, a["img"], a["rc"], a["hw"])


@pytest.mark.parametrize("c_in,c_out,B", [(3, 64, 130), (3, 48, 5), (16, 32, 7), (64, 64, 200)])
def test_layers(both, c_in, c_out, B):
    from fovi_b200 import grad, ops
    rs = np.random.RandomState(c_in)
    n_in, n_out, K, V = 90, 24, 9, 16
    idx = rs.randint(0, n_in + 1, (K, n_out)).astype(np.int32)
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, c_in, c_out)
    x, w, b = torch.randn((B, c_in, n_in), device="cuda"), torch.randn((c_out, c_in * V), device="cuda"), torch.randn(c_out, device="cuda")
    for dt in (torch.float32, torch.bfloat16):
        both(lambda o: o.pack_points(x.to(dt), plan))
        both(lambda o: plan.pack_weights(w.to(dt)))
        both(lambda o: plan.pack_weights(w, dtype=torch.float32))
        both(lambda o: plan.forward_f32(x.to(dt), plan.pack_weights(w, dtype=torch.float32), b))
        for bias in (None, b, b.double(), b.repeat_interleave(2)[::2]):
            both(lambda o: plan.forward(o.pack_points(x, plan), plan.pack_weights(w), bias, relu=True, out_dtype=dt, batch=B))
    if plan.x_layout != ops.X_PAIRS:
        g = grad.KnnConvGrad(idx, tap, n_in, V, c_in, c_out, torch.device("cuda"))
        gy = torch.randn((B, n_out, c_out), device="cuda").to(torch.bfloat16)
        both(lambda o: g.input_grad(gy, w))
        ones = torch.ones((B, n_in, plan.cin_packed), device="cuda", dtype=torch.bfloat16)          # whole numbers: the same in any order of adding
        both(lambda o: g.weight_grad(gy.round(), ones, plan))
    xp, wt = ops.pack_points(x, plan), plan.pack_weights(w)
    with pytest.raises(AssertionError):
        plan.forward(xp[:, :-1], wt, batch=B)
    with pytest.raises(ValueError):
        plan.forward(xp, wt.cpu(), batch=B)
    with pytest.raises(TypeError):
        plan.forward(xp, wt, batch=B, out_dtype=torch.float16)
