"""GPU: layers so wide that the bias table leaves the ring of operand stages only two or three slots (the four producer warps must not run ahead
of it), in every tensor-core kernel that has such a ring, against the oracle on bf16-rounded operands.  Both sides sum the same products, the oracle in
float64: 1e-4 of the largest output covers float32 sums of up to 640 terms in any order, 2^-8 the rounding of bf16 results."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# one CTA per tile: three and two slots; CTA pairs: three and two slots; pair layout on CTA pairs with tensor stores: three slots
@pytest.mark.parametrize("B,cin,cout,K,n_in,n_out,f32", [
    (64, 16, 6656, 40, 50, 24, True), (64, 16, 8192, 40, 50, 24, True), (5, 16, 20480, 25, 50, 12, True), (130, 16, 23552, 40, 50, 4, True),
    (300, 16, 31488, 20, 40, 3, True), (200, 3, 16128, 55, 70, 6, False)])
def test_rings_of_few_slots(B, cin, cout, K, n_in, n_out, f32):
    from fovi_b200 import ops
    rs = np.random.RandomState(cout)
    V = 9
    # pair layout: neighbours from a window of 60 points, so that the lists hold at most 32 pairs and the results leave as tensor copies
    idx = np.stack([rs.permutation(min(n_in, 60))[:K] for _ in range(n_out)], 1).astype(np.int32)
    idx[rs.rand(K, n_out) < 0.1] = n_in
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    w = (rs.standard_normal((cout, cin * V)) / np.sqrt(cin * K)).astype(np.float32)
    bias = rs.standard_normal(cout).astype(np.float32)
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(torch.bfloat16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout, group=1)
    assert plan.tc_supported
    y = plan.forward(ops.pack_points(x.cuda(), plan), plan.pack_weights(dev(w)), dev(bias), batch=B, out_dtype=torch.float32 if f32 else torch.bfloat16)
    plan.check()
    rows = np.unique(np.r_[0, B // 2, B - 1])
    ref = oracle.knnconv_forward_closed_form(x[rows].float().numpy(), idx, tap.astype(np.int64), V,
                                             torch.from_numpy(w).to(torch.bfloat16).float().numpy(), bias)
    got = y[torch.from_numpy(rows).cuda()].float().permute(0, 2, 1).cpu().numpy()
    assert np.abs(got - ref).max() < (1e-4 if f32 else 2.0 ** -8) * np.abs(ref).max()
    if f32:      # whatever was not compared with the oracle: rows of the batch do not depend on each other
        again = plan.forward(ops.pack_points(x[B // 2:].cuda(), plan), plan.pack_weights(dev(w)), dev(bias), batch=B - B // 2, out_dtype=torch.float32)
        assert (y[B // 2:] - again).abs().max().item() < 1e-4 * np.abs(ref).max()
