"""GPU: 64-channel layers on small batches (several output points per tile, split contraction), at the edges of its tiles, against the oracle on
bf16-rounded operands (both sides sum the same products: 1e-4 of the largest output covers float32 sums of up to some thousand terms in any order)."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# batches at the edges of the 8 / 16 / 32 / 64 row slots; channels at the edges of the 64-channel chunks and of one c_out tile; point counts around a
# group, a single point; one split and many; taps that collide, points and a whole group without
# neighbours; one row more than the kernel takes
@pytest.mark.parametrize("B,cin,cout,K,V,n_in,n_out,f32", [
    (1, 16, 32, 3, 9, 20, 1, True), (4, 192, 384, 9, 36, 60, 33, True), (8, 64, 192, 25, 100, 80, 70, False), (9, 96, 64, 9, 4, 30, 17, True),
    (16, 384, 256, 9, 36, 40, 40, True), (15, 72, 96, 5, 5, 25, 15, False), (13, 256, 512, 2, 9, 12, 16, True), (2, 64, 64, 9, 36, 500, 330, False),
    (16, 128, 256, 9, 36, 225, 2000, True), (4, 256, 256, 9, 1, 30, 31, True), (17, 64, 64, 9, 9, 40, 33, True)])
def test_small_batches_against_oracle(B, cin, cout, K, V, n_in, n_out, f32):
    from fovi_b200 import ops
    rs = np.random.RandomState(B + cin)
    idx = rs.randint(0, n_in, (K, n_out)).astype(np.int32)
    idx[rs.rand(K, n_out) < 0.2] = n_in
    idx[:, n_out // 2] = n_in
    if n_out > 300:
        idx[:, 64:96] = n_in                                     # a whole group of points
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    w = (rs.standard_normal((cout, cin * V)) / np.sqrt(cin * K)).astype(np.float32)
    bias = rs.standard_normal(cout).astype(np.float32)
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(torch.bfloat16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout)
    xp, wt = ops.pack_points(x.cuda(), plan), plan.pack_weights(dev(w))
    out_dtype = torch.float32 if f32 else torch.bfloat16
    y = plan.forward(xp, wt, dev(bias), relu=True, out_dtype=out_dtype)
    plan.check()
    again = plan.forward(xp, wt, dev(bias), relu=True, out_dtype=out_dtype)
    assert torch.equal(y, again)                                 # the splits are added in order
    ref = oracle.knnconv_forward_closed_form(x.float().numpy(), idx, tap.astype(np.int64), V,
                                             torch.from_numpy(w).to(torch.bfloat16).float().numpy(), bias, relu=True)
    got = y.float().permute(0, 2, 1).cpu().numpy()
    assert np.abs(got - ref).max() < (1e-4 if f32 else 2.0 ** -8) * np.abs(ref).max()
    # a larger batch of the same rows runs on the kernels that fill a tile with the batch
    big = plan.forward(torch.cat([xp, xp[:1].expand(65, -1, -1)]).contiguous(), wt, dev(bias), relu=True, out_dtype=torch.float32)[:B]
    assert (big - y.float()).abs().max().item() < (1e-4 if f32 else 2.0 ** -8) * np.abs(ref).max()
