"""GPU: pair-layout layers of more than one 128-row tile (CTA pairs), at the edges of its tiles and splits,
against the oracle on bf16-rounded operands (both sides sum the same products: 1e-4 of the largest output covers float32 sums of up
to 1000 terms in any order)."""
import numpy as np
import pytest
import torch

from oracle import fovi_oracle as oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).float().numpy()


# rows just past one tile, one CTA pair exactly, an odd last tile, many units per pair; few and many slabs; one and several channel
# tiles; grouped points; lists shorter than the activation ring and long ones; a large point count
@pytest.mark.parametrize("B,cin,cout,K,n_in,n_out,group,f32", [
    (129, 3, 64, 9, 300, 5, 1, True), (256, 3, 192, 40, 300, 7, 1, False), (300, 3, 64, 60, 401, 12, 4, False),
    (385, 3, 64, 121, 1001, 9, 3, True), (640, 1, 512, 25, 77, 3, 1, False), (700, 4, 32, 3, 50, 200, 1, True),
    (1024, 3, 256, 100, 400, 4, 1, False), (900, 3, 96, 30, 13001, 11, 1, False)])
def test_pair_layout_cta_pairs_against_oracle(B, cin, cout, K, n_in, n_out, group, f32):
    from fovi_b200 import ops
    rs = np.random.RandomState(B + cout)
    V = 49
    centre = rs.randint(0, n_in, -(-n_out // group)).repeat(group)[:n_out]
    width = min(n_in, 2 * K if group == 1 else K + 30)
    idx = np.stack([(c + rs.permutation(width)[:K]) % n_in for c in centre], 1).astype(np.int32)     # neighbourhoods of nearby points
    idx[rs.rand(K, n_out) < 0.15] = n_in
    if n_out > 6:
        idx[:, 6] = n_in                                         # a point without neighbours
    tap = rs.randint(0, V, (n_out, K)).astype(np.uint16)
    w = (rs.standard_normal((cout, cin * V)) / np.sqrt(cin * K)).astype(np.float32)
    bias = rs.standard_normal(cout).astype(np.float32)
    x = torch.from_numpy(rs.standard_normal((B, cin, n_in)).astype(np.float32)).to(torch.bfloat16)
    plan = ops.KnnConvPlan(idx, tap, n_in, V, cin, cout, group=group)
    assert plan.group == group
    before = ops.launch_count()
    y = plan.forward(ops.pack_points(x.cuda(), plan), plan.pack_weights(dev(w)), dev(bias), relu=True, batch=B,
                     out_dtype=torch.float32 if f32 else torch.bfloat16)
    plan.check()
    assert ops.launch_count() == before + 3                      # packed points, packed weights, the layer
    rows = np.unique(np.r_[0, 1, 127, 128, min(255, B - 1), min(256, B - 1), rs.randint(0, B, 20), B - 2, B - 1])
    ref = oracle.knnconv_forward_closed_form(x[rows].float().numpy(), idx, tap.astype(np.int64), V, bf16(w), bias, relu=True)
    got = y[torch.from_numpy(rows).cuda()].float().permute(0, 2, 1).cpu().numpy()
    assert np.abs(got - ref).max() < (1e-4 if f32 else 2.0 ** -8) * np.abs(ref).max()
    # every row is the row that the one-tile kernel computes
    small = plan.forward(ops.pack_points(x[B - 100:].cuda(), plan), plan.pack_weights(dev(w)), dev(bias), relu=True, batch=100, out_dtype=torch.float32)
    assert (y[B - 100:].float() - small).abs().max().item() < (1e-4 if f32 else 2.0 ** -8) * small.abs().max().item()
