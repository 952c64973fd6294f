"""GPU: the exact float32 kernel of layers with at most 4 input channels, at the edges of its tiles, against the oracle.

Both sides add K * c_in products per output, the oracle in float64: float32 sums of n terms differ from it by at most
n * 2^-24 of the sum of the terms' magnitudes."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# images at the edges of the 2 / 4 / 8 tiles; channels at the edges of the 32 / 64 / 96 tiles; points at the edges of the CTA's eight;
# neighbours at the edges of a 16-neighbour pass (16 and 17 of them without a gap, one pass and one more); a filter that fits shared memory and one that does not
@pytest.mark.parametrize("B,cin,cout,K,side,n_out,dtype", [
    (1, 3, 64, 9, 3, 7, torch.float32), (2, 3, 32, 32, 6, 8, torch.float32), (3, 3, 33, 33, 6, 9, torch.bfloat16),
    (5, 1, 96, 49, 7, 41, torch.float32), (8, 4, 97, 31, 5, 16, torch.float32), (9, 3, 160, 25, 5, 65, torch.float32),
    (17, 2, 5, 65, 9, 24, torch.bfloat16), (4, 3, 96, 121, 22, 33, torch.float32),
    (8, 3, 64, 16, 5, 24, torch.float32), (6, 4, 64, 17, 5, 24, torch.float32), (2, 2, 32, 16, 4, 9, torch.bfloat16), (3, 3, 96, 17, 4, 9, torch.float32)])
def test_few_channel_f32_against_oracle(B, cin, cout, K, side, n_out, dtype):
    from fovi_b200 import ops
    rs = np.random.RandomState(B * 1000 + cout)
    n_in, V = 200, side * side
    idx = np.stack([rs.permutation(n_in)[:K] for _ in range(n_out)], 1).astype(np.int32)
    if K not in (16, 17):                                       # lists of exactly one pass and of one neighbour more keep all of theirs
        idx[rs.rand(K, n_out) < 0.2] = n_in
    idx[:, n_out // 2] = n_in                                   # a point without any neighbour
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    w = rs.standard_normal((cout, cin * V)).astype(np.float32)
    bias = rs.standard_normal(cout).astype(np.float32)
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(dtype)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout)
    wt = plan.pack_weights(dev(w), dtype=torch.float32)
    ref = oracle.knnconv_forward_closed_form(x.float().numpy(), idx, tap.astype(np.int64), V, w, bias, relu=True)
    size = oracle.knnconv_forward_closed_form(np.abs(x.float().numpy()), idx, tap.astype(np.int64), V, np.abs(w), np.abs(bias))
    bound = (K * cin + 2) * 2.0 ** -24 * size + 1e-30
    got = {}
    for xl in (ops.ACT_BCN, ops.ACT_BNC):
        xin = (x if xl == ops.ACT_BCN else x.transpose(1, 2)).contiguous().cuda()
        for yl in (ops.ACT_BCN, ops.ACT_BNC):
            y = plan.forward_f32(xin, wt, dev(bias), relu=True, x_layout=xl, y_layout=yl)
            y = (y if yl == ops.ACT_BCN else y.permute(0, 2, 1)).cpu().numpy()
            assert np.all(np.abs(y - ref) <= bound), (xl, yl, float(np.abs(y - ref).max()))
            got[xl, yl] = y
    assert all(np.array_equal(v, got[ops.ACT_BCN, ops.ACT_BCN]) for v in got.values())       # a layout changes no sum
