"""GPU: the weight-gradient kernel (contraction over the batch, operands read as the forward pass left them) against the oracle's backward on
bf16-rounded operands: both sides sum the same products, the oracle in float64, so what differs is float32 summation (1e-4 of the largest
entry covers the few thousand terms of these sums in any order)."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]


def _run(B, cin, cout, K, n_in, n_out, V, seed):
    from fovi_b200 import ops
    from fovi_b200.grad import KnnConvGrad
    rs = np.random.RandomState(seed)
    idx = rs.randint(0, n_in, (K, n_out)).astype(np.int32)          # a point may list a neighbour twice
    idx[rs.rand(K, n_out) < 0.2] = n_in
    idx[:, n_out // 2] = n_in                                       # a point without neighbours
    tap = rs.randint(0, max(1, V - 1), (n_out, K)).astype(np.uint16)   # the last tap is never used
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(torch.bfloat16)
    gy = torch.from_numpy(rs.standard_normal((B, cout, n_out)).astype(np.float32)).to(torch.bfloat16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout)
    grad = KnnConvGrad(idx, tap, n_in, V, cin, cout, torch.device("cuda"))
    got = grad.weight_grad(gy.permute(0, 2, 1).contiguous().cuda(), ops.pack_points(x.cuda(), plan), plan)
    plan.check()
    if "dw" in grad._dw_plans:
        grad.dw_plan()[0].check()
    w = np.zeros((cout, cin * V), np.float32)
    _, want, _ = oracle.knnconv_backward(x.float().numpy(), idx, tap.astype(np.int64), V, w, gy.float().numpy())
    assert got.shape == want.shape and got.dtype == torch.float32
    got = got.cpu().numpy()
    assert np.abs(got - want).max() < 1e-4 * np.abs(want).max()


# batches at the edges of the 64-row stages; channels at the edges of the 64-channel boxes, the 128 / 256 row tiles and the 256-column tiles;
# one CTA (rows up to 128 channels) and CTA pairs, either operand as the rows
@pytest.mark.parametrize("B,cin,cout,K,n_in,n_out,V", [
    (1, 16, 16, 3, 20, 9, 4), (63, 64, 64, 9, 40, 30, 9), (65, 64, 192, 5, 50, 40, 9), (128, 72, 144, 4, 30, 25, 4),
    (70, 24, 48, 9, 60, 50, 16), (130, 192, 384, 3, 20, 16, 5), (64, 384, 256, 2, 12, 10, 4), (40, 520, 272, 2, 9, 7, 3), (96, 136, 128, 3, 15, 12, 1)])
def test_channels_last_operands(B, cin, cout, K, n_in, n_out, V):
    _run(B, cin, cout, K, n_in, n_out, V, seed=B + cin)


# slot lists shorter than a tile, just past one tile of 32 and of several tiles; odd point counts; channels past one row tile; rows past a 128-row tile
@pytest.mark.parametrize("B,cin,cout,K,n_in,n_out,V", [
    (1, 3, 16, 4, 11, 6, 4), (64, 3, 64, 30, 200, 12, 49), (65, 3, 96, 60, 401, 9, 25), (129, 4, 64, 121, 1001, 7, 121), (200, 1, 144, 20, 33, 10, 9),
    (257, 2, 272, 9, 77, 5, 16)])
def test_pair_layout_operands(B, cin, cout, K, n_in, n_out, V):
    _run(B, cin, cout, K, n_in, n_out, V, seed=B + cout)


@pytest.mark.parametrize("rows,C", [(1, 8), (1000, 64), (777, 192), (333, 384), (50, 2048)])
def test_relu_mask_and_channel_sums(rows, C):
    from fovi_b200 import ops
    torch.manual_seed(rows)
    g = torch.randn(rows, C, device="cuda").to(torch.bfloat16)
    y = torch.relu(torch.randn(rows, C, device="cuda")).to(torch.bfloat16)
    y[0, 0] = float("nan")
    masked, sums = ops.relu_mask_colsum(g, y)
    want = torch.where(y > 0, g, torch.zeros_like(g))
    assert torch.equal(masked, want)
    err = (sums.double() - want.double().sum(0)).abs()
    assert (err <= rows * 2.0 ** -24 * want.double().abs().sum(0) + 1e-30).all()
    assert ops.relu_mask_colsum(g[:, :4].contiguous(), y[:, :4].contiguous()) is None
