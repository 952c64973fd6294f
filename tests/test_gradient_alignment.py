"""Upstream gradients that do not start on a 16-byte boundary (pieces of a larger buffer) give the gradients that aligned ones give."""
import numpy as np
import pytest
import torch


def _shifted(t):
    """t's values in memory of their own, one element past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    flat[1:1 + t.numel()] = t.reshape(-1)
    out = flat[1:1 + t.numel()].view(t.shape)
    assert out.data_ptr() % 16 != 0 and out.is_contiguous()
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_channels_last_copy_is_aligned(dtype):
    from fovi_b200.grad import _channels_last
    t = torch.randn(3, 7, 16).to(dtype)
    got = _channels_last(_shifted(t).permute(0, 2, 1))
    assert got.data_ptr() % 16 == 0 and got.is_contiguous() and torch.equal(got, t.to(torch.bfloat16))


class _Pts:
    def __init__(self, n):
        self.shape, self.dtype = (n, 2), torch.float32


@pytest.mark.gpu
@pytest.mark.autograd
@pytest.mark.parametrize("cin", [3, 16])
@pytest.mark.parametrize("stacked,relu", [(False, False), (True, False), (True, True)])
def test_misaligned_upstream_gradient(cin, stacked, relu):
    from fovi_b200.knn import KNNConvLayer, KNNConvStack
    rs = np.random.RandomState(cin)
    n_in, n_out, K, V, B = 40, 30, 9, 9, 6
    idx = np.stack([rs.permutation(n_in)[:K] for _ in range(n_out)], 1).astype(np.int64)
    layer = KNNConvLayer(cin, 32, K, _Pts(n_in), _Pts(n_out), device="cuda", bias=True,
                         tables_override=dict(knn_indices=idx, tap=rs.randint(0, V, (n_out, K)), V=V))
    net = KNNConvStack([layer], final_relu=relu) if stacked else layer
    torch.manual_seed(0)
    x = torch.randn(B, cin, n_in, device="cuda").to(torch.bfloat16).requires_grad_(cin > 4)
    gy = torch.randn(B, n_out, 32, device="cuda").to(torch.bfloat16)
    grads = []
    for g in (gy, _shifted(gy)):
        layer.weight.grad = layer.bias.grad = x.grad = None
        net(x).backward(g.permute(0, 2, 1))
        layer.plan.check()
        grads.append([p.grad.float() for p in (layer.weight, layer.bias, x) if p.grad is not None])
    for a, b in zip(*grads):
        # the same products, added in any order in float32
        assert (a - b).abs().max().item() <= 1e-5 * a.abs().max().item()
