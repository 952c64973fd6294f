"""GPU: an input gradient that leaves its kernel behind the ReLU mask of the layer below, with its sums per channel, against the separate calls."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]


# the fewest rows of the CTA-pair kernel, an odd last row tile, several tiles per CTA pair; channels that leave half a 64-column piece, two channel tiles; a point
# that no output reads
@pytest.mark.parametrize("B,c_in,c_out,n_in,n_out,K", [(129, 32, 64, 30, 9, 5), (300, 96, 128, 50, 40, 9), (700, 64, 192, 120, 60, 9), (260, 512, 64, 20, 11, 3), (1025, 160, 32, 33, 33, 4)])
def test_masked_input_grad_against_separate_calls(B, c_in, c_out, n_in, n_out, K):
    from fovi_b200 import grad, ops
    rs = np.random.RandomState(B)
    gen = torch.Generator(device="cuda").manual_seed(B)
    idx = rs.randint(0, n_in + 1, (K, n_out)).astype(np.int32)
    idx[idx == 3] = n_in
    g = grad.KnnConvGrad(idx, rs.randint(0, 16, (n_out, K)), n_in, 16, c_in, c_out, torch.device("cuda"))
    gy = torch.randn((B, n_out, c_out), generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn((c_out, c_in * 16), generator=gen, device="cuda") / 8
    act = torch.relu(torch.randn((B, n_in, c_in), generator=gen, device="cuda")).to(torch.bfloat16)
    act[0, 0, :4] = torch.tensor([float("nan"), -0.0, float("inf"), 1e-40])
    gx, sums = g.input_grad_masked(gy, w, act)
    g.check()
    want, want_sums = ops.relu_mask_colsum(g.input_grad(gy, w), act)
    assert torch.equal(gx, want) and (gx[:, 3] == 0).all()
    size = want.double().abs().sum((0, 1))                       # float32 sums in another order: n roundings of at most the sum of the magnitudes
    n = B * n_in
    assert ((sums.double() - want.double().sum((0, 1))).abs() <= n ** 0.5 * 2.0 ** -22 * size + 1e-30).all()
    assert ((sums - want_sums).double().abs() <= n ** 0.5 * 2.0 ** -21 * size + 1e-30).all()
    assert g.input_grad_masked(gy[:128].contiguous(), w, act[:128].contiguous()) is None            # one row tile: the separate calls


@pytest.mark.parametrize("rows,frozen", [(200, False), (200, True), (40, False)])
def test_stack_gradients_do_not_depend_on_it(monkeypatch, rows, frozen):
    from fovi_b200 import grad
    from fovi_b200.coords import get_in_out_coords
    from fovi_b200.knn import KNNConvLayer, KNNConvStack
    ic, oc, _ = get_in_out_coords(20, 16, 1.0, 2, auto_match_cart_resources=0)
    torch.manual_seed(0)
    stack = KNNConvStack([KNNConvLayer(3, 64, 9, ic, oc, device="cuda", ref_frame_side_length=3, bias=True),
                          KNNConvLayer(64, 96, 9, oc, oc, device="cuda", ref_frame_side_length=3, bias=True),
                          KNNConvLayer(96, 32, 9, oc, oc, device="cuda", ref_frame_side_length=3, bias=False)], final_relu=True)
    for L in stack.layers[:2]:
        torch.nn.init.normal_(L.bias, std=0.1)
    if frozen:
        stack.layers[1].weight.requires_grad_(False)
    x = torch.randn((rows, 3, len(ic)), device="cuda").to(torch.bfloat16)
    up = torch.randn((rows, 32, len(oc)), device="cuda").to(torch.bfloat16)

    def grads():
        stack.zero_grad()
        y = stack(x)
        y.backward(up, retain_graph=True)
        first = [p.grad.clone() for p in stack.parameters() if p.grad is not None]
        stack.zero_grad()
        y.backward(up)                                            # the same graph once more
        second = [p.grad for p in stack.parameters() if p.grad is not None]
        for a, b in zip(first, second, strict=True):
            assert (a - b).norm() <= 1e-5 * b.norm()              # float32 sums in no fixed order
        return second
    got = grads()
    monkeypatch.setattr(grad.KnnConvGrad, "input_grad_masked", lambda *a: None)
    want = grads()
    assert len(got) == len(want) == (4 if frozen else 5)
    for a, b in zip(got, want):
        assert (a - b).norm() <= 1e-5 * b.norm()
