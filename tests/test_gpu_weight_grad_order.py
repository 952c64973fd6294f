"""GPU: the weight gradient of a first layer (pair layout) adds its sums in a fixed order: repeated runs give the same bits.  Also with a workspace
that holds one output point, a few of them, all but one and all, against the oracle on bf16-rounded operands (both sides sum the same products, the oracle in
float64: 1e-4 of the largest entry covers the float32 sums of a few thousand terms in any order)."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


# lists within one 32-slot tile and over several, an odd number of points, one and two channel tiles, taps with one entry and with thousands
@pytest.mark.parametrize("B,cin,cout,K,n_in,n_out,V", [
    (1, 3, 16, 4, 11, 6, 24), (70, 3, 64, 30, 200, 213, 49), (65, 3, 96, 121, 401, 9, 2), (200, 4, 144, 20, 33, 300, 1), (129, 1, 48, 60, 301, 17, 9)])
def test_same_bits_every_time(B, cin, cout, K, n_in, n_out, V):
    from fovi_b200 import ops
    from fovi_b200._lib import FoviError, lib
    rs = np.random.RandomState(B + cout)
    idx = rs.randint(0, n_in, (K, n_out)).astype(np.int32)          # a point may list a neighbour twice
    idx[rs.rand(K, n_out) < 0.2] = n_in
    idx[:, n_out // 2] = n_in                                       # a point without neighbours
    tap = rs.randint(0, max(1, V - 1), (n_out, K)).astype(np.uint16)   # the last tap is never used
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(torch.bfloat16)
    gy = torch.from_numpy(rs.standard_normal((B, cout, n_out)).astype(np.float32)).to(torch.bfloat16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout)
    g, xp = gy.permute(0, 2, 1).contiguous().cuda(), ops.pack_points(x.cuda(), plan)
    whole = lib.fovi_knnconv_weight_grad_workspace_bytes(plan._h)
    one = whole // n_out
    assert whole % n_out == 0 and one % 256 == 0
    _, want, _ = oracle.knnconv_backward(x.float().numpy(), idx, tap.astype(np.int64), V, np.zeros((cout, cin * V), np.float32), gy.float().numpy())
    for work in (None, whole, one, 3 * one + 16, whole - 1):
        got = plan.weight_grad_pairs(g, xp, work_bytes=work)
        torch.empty(whole, dtype=torch.uint8, device="cuda").fill_(0xFF)     # NaN in memory that the next call's workspace may get
        for _ in range(3):
            assert torch.equal(plan.weight_grad_pairs(g, xp, work_bytes=work), got)
        plan.check()
        dw = ops.weight_grad_unpack(got, cout, cin).cpu().numpy()
        assert np.abs(dw - want).max() < 1e-4 * np.abs(want).max()
    with pytest.raises(FoviError):
        plan.weight_grad_pairs(g, xp, work_bytes=one - 1)
