"""Fixations that need a conversion on their way to the C calls (another dtype, strided views): the pointers handed over must name the converted
values while the call runs.  On the CPU the library is replaced by one that reads what the pointers name; on the GPU the results are compared."""
import ctypes

import numpy as np
import pytest
import torch

FORMS = ["float64", "strided", "float64 strided"]


def _form(t, form):
    if "float64" in form:
        t = t.double()
    if "strided" in form:
        t = torch.stack([t, -t], -1)[..., 0]
    assert t.dtype != torch.float32 or not t.is_contiguous()
    return t


def _read(ptr, shape):
    n = int(np.prod(shape))
    return np.ctypeslib.as_array(ctypes.cast(ctypes.c_void_p(ptr), ctypes.POINTER(ctypes.c_float)), (n,)).reshape(shape).copy()


class _Plan:
    _h = _h_tc = None
    n_points, n_out, c_out = 5, 4, 16


@pytest.fixture
def ops(monkeypatch):
    from fovi_b200 import ops
    monkeypatch.setattr(ops, "_need_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_on", lambda device: ops._HERE)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return ops


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("call", ["backward", "fused"])
def test_pointers_name_the_converted_fixations(ops, monkeypatch, call, form):
    B, F = 64, 16                  # 8 KB each: a freed copy's block is what the next copy of that size gets
    rc, hw = torch.rand(B, F, 2), 100 * torch.rand(B, F, 2)
    seen = {}

    class Lib:
        @staticmethod
        def fovi_sample_backward(*a):
            seen.update(rc=_read(a[8], (B, F, 2)), hw=_read(a[9], (B, F, 2)))
            return 0

        @staticmethod
        def fovi_sample_knnconv_fused(*a):
            seen.update(rc=_read(a[9], (B, F, 2)), hw=_read(a[10], (B, F, 2)))
            return 0

        @staticmethod
        def fovi_fused_intermediate_bytes(*a):
            return 64
    with monkeypatch.context() as m:
        m.setattr(ops, "lib", Lib)
        if call == "backward":
            ops.sample_backward(_Plan, torch.zeros(B, F, 1, 5), (B, 1, 8, 8), _form(rc, form), _form(hw, form))
        else:
            ops.sample_knnconv_fused(_Plan, _Plan, torch.zeros(B, 1, 8, 8), _form(rc, form), _form(hw, form), torch.zeros(1))
    assert np.array_equal(seen["rc"], rc.numpy()) and np.array_equal(seen["hw"], hw.numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
def test_results_do_not_depend_on_the_form(golden, form):
    from fovi_b200 import ops
    B, F = 6, 3
    plan = ops.SamplerPlan(golden("sensor_a1.npz")["sampling_grid"])
    gen = torch.Generator(device="cuda").manual_seed(1)
    img = torch.rand((B, 3, 64, 64), generator=gen, device="cuda")
    rc, hw = torch.rand((B, F, 2), generator=gen, device="cuda"), 32 + 32 * torch.rand((B, F, 2), generator=gen, device="cuda")
    gout = torch.randint(-4, 5, (B, F, 3, plan.n_points), generator=gen, device="cuda").float()
    want = ops.sample_backward(plan, gout, img.shape, rc, hw, mode=ops.NEAREST)           # whole numbers: the same in any order of adding
    assert torch.equal(ops.sample_backward(plan, gout, img.shape, _form(rc, form), _form(hw, form), mode=ops.NEAREST), want)

    rs = np.random.RandomState(0)
    K, V, n_out = 9, 9, 12
    idx = rs.randint(0, plan.n_points, (K, n_out)).astype(np.int32)
    conv = ops.KnnConvPlan(idx, rs.randint(0, V, (n_out, K)).astype(np.uint16), plan.n_points, V, 3, 32)
    wt = conv.pack_weights(torch.randn((32, 3 * V), generator=gen, device="cuda"))
    want, _ = ops.sample_knnconv_fused(plan, conv, img, rc, hw, wt)
    got, _ = ops.sample_knnconv_fused(plan, conv, img, _form(rc, form), _form(hw, form), wt)
    assert torch.equal(got, want)
