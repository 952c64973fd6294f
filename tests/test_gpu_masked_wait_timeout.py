"""GPU: the failure path of the masked input gradient.  Its epilogue warps meet at a barrier of their own behind the loop, which each of them has to reach after a wait
that ran out; the wait is made to run out by a launch that issues no loads and whose wait limit is a few thousand attempts."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]
FOVI_ERR_DEVICE_TIMEOUT = 6   # include/fovi_b200.h


# one pair of CTAs with work, several items per pair, two column tiles
@pytest.mark.parametrize("B,c_in,c_out,n_in,n_out,K", [(129, 32, 64, 1, 9, 5), (700, 64, 192, 120, 60, 9), (260, 512, 64, 20, 11, 3)])
def test_a_masked_gradient_that_gave_up_is_reported(B, c_in, c_out, n_in, n_out, K):
    from fovi_b200 import grad
    from fovi_b200._lib import FoviError
    rs = np.random.RandomState(B)
    g = grad.KnnConvGrad(rs.randint(0, n_in, (K, n_out)), rs.randint(0, 9, (n_out, K)), n_in, 9, c_in, c_out, torch.device("cuda"))
    gen = torch.Generator(device="cuda").manual_seed(B)
    gy = torch.randn((B, n_out, c_out), generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn((c_out, c_in * 9), generator=gen, device="cuda") / 8
    act = torch.relu(torch.randn((B, n_in, c_in), generator=gen, device="cuda")).to(torch.bfloat16)
    want, _ = g.input_grad_masked(gy, w, act)
    g.check()
    plan = g.dx_plan()
    for _ in range(2):
        plan.input_grad_masked(gy, plan.pack_weights_transposed(w), act, selftest=True)
        with pytest.raises(FoviError) as e:
            g.check()
        assert e.value.status == FOVI_ERR_DEVICE_TIMEOUT and "wait site" in str(e.value)
        g.check()                                    # the status word was cleared by the failing check
        got, sums = g.input_grad_masked(gy, w, act)
        g.check()
        assert torch.equal(got, want) and torch.isfinite(sums).all()
