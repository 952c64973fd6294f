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


# channel counts around the 64 x 64 tiles, padded channels, taps past one tile
@pytest.mark.parametrize("cin,cout,V,dtype", [(16, 48, 9, torch.float32), (72, 64, 36, torch.bfloat16), (100, 32, 130, torch.float32), (192, 384, 64, torch.float32),
                                              (65, 16, 65, torch.float32)])
def test_filter_layout_changes(cin, cout, V, dtype):
    from fovi_b200 import ops
    torch.manual_seed(cin)
    w = torch.randn(cout, cin * V, device="cuda").to(dtype)
    w3 = w.view(cout, cin, V)
    one = lambda a, b: ops.KnnConvPlan(np.zeros((1, 2), np.int32), np.zeros((2, 1), np.uint16), 3, V, a, b)   # noqa: E731
    plan = one(cin, cout)
    for t in (torch.bfloat16, torch.float32):
        got = plan.pack_weights(w, t)
        assert torch.equal(got[:, :, :cin], w3.permute(2, 0, 1).to(t)) and not got[:, :, cin:].any()
    got = one(cout, cin).pack_weights_transposed(w)
    assert torch.equal(got[:, :, :cout], w3.permute(2, 1, 0).to(torch.bfloat16)) and not got[:, :, cout:].any()
    g = torch.randn(V, cout + 8, cin + 8, device="cuda")
    assert torch.equal(ops.weight_grad_unpack(g, cout, cin, dtype=dtype), g[:, :cout, :cin].permute(1, 2, 0).reshape(cout, cin * V).to(dtype))
    gs = torch.randn(V, cin + 8, cout, device="cuda")
    assert torch.equal(ops.weight_grad_unpack(gs, cout, cin, swapped=True, dtype=dtype), gs[:, :cin].permute(2, 1, 0).reshape(cout, cin * V).to(dtype))


@pytest.mark.parametrize("cin,cout,V,n_out,group", [(3, 64, 484, 12, 3), (4, 48, 25, 8, 4), (1, 96, 9, 6, 2), (3, 16, 801, 4, 4)])
def test_grouped_weights_equal_the_ungrouped_ones(cin, cout, V, n_out, group):
    """Every member's rows of a group's packed weights are the filter rows its own taps name (801 taps: past the shared-memory kernel)."""
    from fovi_b200 import ops
    rs = np.random.RandomState(V)
    n_in, K = 60, 9
    idx = np.stack([rs.permutation(n_in)[:K] for _ in range(n_out)], 1).astype(np.int32)
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout, group=group)
    assert plan.group == group
    w = torch.randn(cout, cin * V, device="cuda")
    x = torch.randn(3, cin, n_in, device="cuda").to(torch.bfloat16)
    xp = ops.pack_points(x, plan)
    got = plan.forward(xp, plan.pack_weights(w), batch=3, out_dtype=torch.float32)
    flat = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout, group=1)
    want = flat.forward(xp, flat.pack_weights(w), batch=3, out_dtype=torch.float32)
    assert (got - want).abs().max().item() < 1e-5 * want.abs().max().item()
