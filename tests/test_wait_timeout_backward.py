"""The failure path of the backward pass: a launch that gave up on a wait leaves an incomplete gradient, and the layer's check has to say so."""
import numpy as np
import pytest
import torch

FOVI_ERR_DEVICE_TIMEOUT = 6   # include/fovi_b200.h


class _Pts:
    def __init__(self, n):
        self.shape, self.dtype = (n, 2), torch.float32


def test_every_derived_plan_is_asked():
    from fovi_b200.grad import KnnConvGrad
    asked = []

    class Plan:
        def __init__(self, name):
            self.name = name

        def check(self):
            asked.append(self.name)
    g = KnnConvGrad(np.zeros((1, 2), np.int64), np.zeros((2, 1), np.int64), 3, 1, 16, 16, torch.device("cpu"))
    g.check()
    assert asked == []
    g._dx_plan = Plan("dx")
    g._dw_plans = {"dw": (Plan("dw"), np.zeros(1)), ("f32", 4): (Plan("dx32"), Plan("dw32"), torch.zeros(1))}
    g.check()
    assert sorted(asked) == ["dw", "dw32", "dx", "dx32"]


# weight gradient on one CTA, on CTA pairs, of the pair layout
@pytest.mark.gpu
@pytest.mark.autograd
@pytest.mark.parametrize("cin,cout,B", [(16, 64, 5), (256, 256, 70), (3, 64, 70)])
def test_a_gradient_that_gave_up_is_reported(cin, cout, B):
    from fovi_b200 import ops
    from fovi_b200._lib import FoviError
    from fovi_b200.knn import KNNConvLayer
    rs = np.random.RandomState(cin)
    n_in, n_out, K, V = 40, 30, 9, 9
    idx = np.stack([rs.permutation(n_in)[:K] for _ in range(n_out)], 1).astype(np.int64)
    layer = KNNConvLayer(cin, cout, K, _Pts(n_in), _Pts(n_out), device="cuda",
                         tables_override=dict(knn_indices=idx, tap=rs.randint(0, V, (n_out, K)), V=V))
    torch.manual_seed(0)
    x = torch.randn(B, cin, n_in, device="cuda").to(torch.bfloat16).requires_grad_(cin > 4)
    gy = torch.randn(B, n_out, cout, device="cuda").to(torch.bfloat16)

    def gradient():
        layer.weight.grad = None
        layer(x).backward(gy.permute(0, 2, 1))
        layer.check()
        return layer.weight.grad.clone()
    want = gradient()

    def gave_up():
        for check in (layer.check, layer.plan.check):
            with pytest.raises(FoviError) as e:
                run()
                check()
            assert e.value.status == FOVI_ERR_DEVICE_TIMEOUT and "wait site" in str(e.value)
            layer.check()                            # the status word was cleared by the failing check
    g, xp = layer.grad_plans, ops.pack_points(x.detach(), layer.plan)
    if cin <= 4:
        run = lambda: layer.plan.weight_grad_pairs(gy, xp, selftest=True)                                      # noqa: E731
    else:
        run = lambda: g.dw_plan()[0].run(*((xp, gy) if g.dw_swapped else (gy, xp)), selftest=True)             # noqa: E731
    gave_up()
    if cin > 4:
        dx = g.dx_plan()
        run = lambda: dx.selftest_wait_timeout(gy, dx.pack_weights_transposed(layer.weight))                   # noqa: E731
        gave_up()
    err = (gradient() - want).abs().max().item()
    assert err <= 1e-5 * want.abs().max().item()      # the same products, added in any order
