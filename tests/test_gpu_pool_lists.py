"""GPU: channels-last bf16 pooling fetches three neighbours at a time; lists of every remainder against the scalar kernel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["max", "avg", "sum"])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 8, 10, 16])
def test_lists_of_every_remainder(mode, K):
    from fovi_b200 import ops
    rs = np.random.RandomState(K)
    B, C, n_in, n_out = 5, 40, 37, 23
    x = torch.from_numpy(rs.standard_normal((B, n_in, C)).astype(np.float32)).to(torch.bfloat16)
    x[1, 3, 5] = float("nan")
    x[2, :, 7] = float("nan")
    x[3, 4, :3] = torch.tensor([float("inf"), float("-inf"), torch.finfo(torch.bfloat16).min])
    idx = rs.randint(0, n_in + 1, (K, n_out)).astype(np.int32)
    idx[:, 0] = n_in                                                        # no neighbour
    idx[K // 2:, 1] = n_in                                                  # pads at the end of a list
    idx[-1, 2] = n_in - 1                                                   # the last point in the last place
    plan = ops.KnnPoolPlan(idx, n_in)
    y = plan.forward(x.cuda(), mode, ops.ACT_BNC)
    want = plan.forward(x.float().cuda(), mode, ops.ACT_BNC).to(torch.bfloat16)         # one neighbour at a time, float32 in and out
    assert y.dtype == torch.bfloat16 and torch.equal(torch.isnan(y), torch.isnan(want))
    assert torch.equal(y.float().nan_to_num(0.0, 1e30, -1e30), want.float().nan_to_num(0.0, 1e30, -1e30))
