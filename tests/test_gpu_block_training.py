"""GPU: what surrounds the batch norm of a training step (csrc/blocktrain.cu) against plain torch, at the edges of its tiles and slabs, and the block that runs
it against the block whose modules run one by one."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


# two rows in all, fewer rows than a CTA holds, channels that are no whole slab or tile, slabs of 32, 16 and 8 channels, a row of more than 256 channel
# quads, pads in the pooling lists and an output without neighbours, long lists, no ReLU
@pytest.mark.parametrize("B,N,C,n_out,K,relu", [
    (1, 2, 16, 0, 0, True), (3, 5, 96, 4, 3, True), (2, 230, 136, 60, 9, True), (40, 61, 128, 16, 9, False), (128, 60, 256, 0, 0, False),
    (97, 60, 384, 7, 200, True), (9, 1031, 48, 230, 9, True), (2, 4000, 24, 33, 4, True), (5, 7, 1040, 0, 0, True)])
def test_relu_pool_and_its_gradient_against_float64(B, N, C, n_out, K, relu):
    from fovi_b200 import ops
    rs = np.random.RandomState(B + C)
    gen = torch.Generator(device="cuda").manual_seed(B * C)
    y = torch.randn((B, N, C), generator=gen, device="cuda") * (0.1 + torch.rand(C, generator=gen, device="cuda")) + torch.randn(C, generator=gen, device="cuda")
    gamma, beta = 1 + 0.2 * torch.randn(C, generator=gen, device="cuda"), 0.3 * torch.randn(C, generator=gen, device="cuda")
    plan = sel = None
    if n_out:
        idx = np.stack([rs.randint(0, N, K) for _ in range(n_out)], 1)
        idx[rs.rand(K, n_out) < 0.2] = N
        idx[0, :-1] = rs.randint(0, N, n_out - 1)
        idx[:, -1] = N
        plan, sel = ops.KnnPoolPlan(idx.astype(np.int32), N, device="cuda"), torch.from_numpy(idx[:, :-1]).cuda()
        assert plan.block_supported
    yt = ops.points_to_channels(y)
    assert torch.equal(yt, y.permute(0, 2, 1).contiguous())
    mean, var = y.double().mean((0, 1)), y.double().var((0, 1), unbiased=False)
    rstd = torch.rsqrt(var + 1e-5)
    h = ((yt - mean.float()[:, None]) * rstd.float()[:, None]) * gamma[:, None] + beta[:, None]
    out, arg = ops.relu_pool(h, relu, plan)

    def module(t):                                                 # [B, C, N] -> [B, n_out, C], any dtype
        t = torch.relu(t) if relu else t
        if n_out:
            t = torch.nn.functional.pad(t, (0, 1), value=-np.inf)[:, :, sel].amax(2)
        return t.permute(0, 2, 1)
    assert torch.equal(out[:, :n_out - 1] if n_out else out, module(h))             # exact operations
    if n_out:
        assert torch.isneginf(out[:, -1]).all() and (arg[:, -1] == 255).all()
    up = torch.randn(out.shape, generator=gen, device="cuda")
    act = out if relu and not n_out else None
    dx, dgamma, dbeta = ops.norm_block_backward(y, mean.float(), rstd.float(), gamma, act, up, plan, arg)
    # float64 autograd through the norm, with the masks and maxima of the float32 forward pass above
    y64, g64, b64 = (t.double().requires_grad_() for t in (y, gamma, beta))
    mu, v = y64.mean((0, 1)), y64.var((0, 1), unbiased=False)
    h64 = ((y64 - mu) * torch.rsqrt(v + 1e-5) * g64 + b64).permute(0, 2, 1)
    ht = h.clone().requires_grad_()
    (module(ht) * up[:, :n_out - 1 if n_out else N]).sum().backward()               # (zeros that tie behind the ReLU hand amax's gradient to a mask of zero)
    h64.backward(ht.grad.double())
    n = B * N
    if n > 2:      # (with two values per channel the gradient is their difference's, near zero)
        # float32 sums of n terms, added in chunks of a few hundred and then in double: 1e-5; bf16 results: 2^-8
        assert rel(dbeta, b64.grad) < 1e-5 and rel(dgamma, g64.grad) < 1e-5
        assert rel(dx, y64.grad) < 2.0 ** -8
    again = ops.norm_block_backward(y, mean.float(), rstd.float(), gamma, act, up, plan, arg)
    assert torch.equal(again[0], dx) and torch.equal(again[1], dgamma) and torch.equal(again[2], dbeta)


def test_nan_and_ties_as_the_modules_treat_them():
    from fovi_b200 import ops
    h = torch.randn((4, 16, 6), device="cuda")
    h[1, 3, 2] = float("nan")
    h[2, :, 1] = h[2, :, 0]                                         # a tie: the first neighbour of the list
    idx = np.array([[0, 2, 2], [1, 6, 2]], np.int32)
    out, arg = ops.relu_pool(h, False, ops.KnnPoolPlan(idx, 6, device="cuda"))
    assert torch.isneginf(out[1, 1:, 3]).all() and (arg[1, 1:, 3] == 255).all() and torch.isfinite(out[1, 0]).all() and (arg[2, 0] == 0).all()
    out, arg = ops.relu_pool(h, True, None)
    assert arg is None and torch.equal(out.nan_to_num(7.0), torch.relu(h).permute(0, 2, 1).nan_to_num(7.0))


@pytest.mark.parametrize("pool", [True, False])
def test_fused_block_equals_its_modules(pool):
    from fovi_b200.alexnet import KNNAlexNetBlock

    def make():
        torch.manual_seed(0)
        return KNNAlexNetBlock(32, 64, 9, 16, 0.5, 12, 1, pool=pool, norm_type="force_batch", device="cuda", ref_frame_mult=2).train()
    blk, other = make(), make()
    calls = []
    other.norm.register_forward_hook(lambda *a: calls.append(1))              # a listener: the modules run one by one
    x = torch.randn((50, 32, blk.in_coords.shape[0]), device="cuda")
    xa, xb = x.clone().requires_grad_(), x.clone().requires_grad_()
    assert blk._fused_training(xa) and not other._fused_training(xb)
    ya, yb = blk(xa), other(xb)
    assert calls and ya.shape == yb.shape and torch.equal(ya, yb)
    for p, q in zip(blk.buffers(), other.buffers()):
        assert torch.equal(p, q)
    up = torch.randn(ya.shape, device="cuda")
    ya.backward(up); yb.backward(up)
    for (n, p), q in zip(blk.named_parameters(), other.parameters()):
        assert rel(p.grad, q.grad) < 2.0 ** -8, n                              # the gradient's bf16 roundings in between
    assert rel(xa.grad, xb.grad) < 2.0 ** -8
    # what the fused form does not cover runs as before
    assert not make().eval()._fused_training(x) and not make()._fused_training(x.to(torch.bfloat16))
    other = make()
    other.norm.momentum = None
    assert not other._fused_training(x)
