"""GPU: what a caller may do with the result of a training block does not depend on which path ran it."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = [pytest.mark.gpu, pytest.mark.autograd]


def make(**kw):
    from fovi_b200.alexnet import KNNAlexNetBlock
    torch.manual_seed(0)
    return KNNAlexNetBlock(32, 64, 9, 16, 0.5, 12, 1, norm_type="force_batch", device="cuda", ref_frame_mult=2, **kw).train()


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def pair(**kw):
    """The block in one function, and the one whose modules run one by one because somebody listens."""
    one, other = make(**kw), make(**kw)
    other.norm.register_forward_hook(lambda *a: None)
    x = torch.randn((7, 32, one.in_coords.shape[0]), device="cuda")
    assert one._fused_training(x) and not other._fused_training(x)
    return one, other, x


def twice(h):
    return h.mul_(2)


def dropped(h):
    torch.manual_seed(1)
    return F.dropout(h, 0.3, inplace=True)


def lines(h):
    h[:, 3] += 1
    h[2] = 0
    return h


@pytest.mark.parametrize("change", [twice, dropped, lines, torch.relu_])
@pytest.mark.parametrize("kw", [dict(pool=True), dict(pool=False, activation=None)], ids=["pool", "norm"])
def test_in_place_operations_on_the_result(change, kw):
    one, other, x = pair(**kw)
    got, want = [], []
    for block, into in ((one, got), (other, want)):
        xg = x.clone().requires_grad_()
        h = change(block(xg))
        up = torch.randn(h.shape, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
        h.backward(up)
        into += [h.detach(), xg.grad] + [p.grad for p in block.parameters()]
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:], strict=True):
        assert rel(a, b) < 2.0 ** -8                            # the gradient's bf16 roundings in between


@pytest.mark.parametrize("kw", [dict(pool=True), dict(pool=False), dict(pool=False, activation=None)], ids=["pool", "relu", "norm"])
def test_result_is_contiguous(kw):
    one, other, x = pair(**kw)
    a, b = one(x), other(x)
    assert a.is_contiguous() and b.is_contiguous() and torch.equal(a.view(7, -1), b.view(7, -1))
    random = torch.randn_like(a)
    for g, w in zip(torch.autograd.grad(a, list(one.parameters()), random, retain_graph=True), torch.autograd.grad(b, list(other.parameters()), random), strict=True):
        assert rel(g, w) < 2.0 ** -8
    # upstream gradients of any strides are the same gradient (the filter's is left out: its parts are added in no fixed order)
    params = (one.norm.weight, one.norm.bias)
    for up in (random.transpose(1, 2).contiguous().transpose(1, 2), torch.randn((1, a.shape[1], 1), device="cuda").expand(a.shape)):
        got, want = (torch.autograd.grad(a, params, u, retain_graph=True) for u in (up, up.contiguous()))
        for g, w in zip(got, want, strict=True):
            assert torch.equal(g, w)


@pytest.mark.parametrize("listener", [None, "block", "pre", "inner", "first conv"])
def test_network_features_and_what_hooks_see_are_contiguous(listener):
    from fovi_b200.alexnet import KNNAlexNet

    def net():
        torch.manual_seed(0)
        return KNNAlexNet(12, 16, [32, 48, 32], [1, 1, 1], [0, 2], [9, 9, 9], cmf_a=0.5, ref_frame_mult=2, norm_type="force_batch", device="cuda").train()
    one, other = net(), net()
    seen = []
    see = lambda m, args, out=None: seen.append((args[0] if out is None else out).view(args[0].shape[0], -1).shape)     # noqa: E731
    if listener == "block":
        one.layers[1].register_forward_hook(see)
    elif listener == "pre":
        one.layers[1].register_forward_pre_hook(see)
    elif listener == "inner":
        one.layers[1].norm.register_forward_hook(see)
    elif listener == "first conv":
        one.layers[2].conv.register_forward_pre_hook(see)
    for L in other.layers:
        L.norm.register_forward_hook(lambda *a: None)
    x = torch.randn((9, 16, one.layers[0].in_coords.shape[0]), device="cuda")
    a, b = one(x), other(x)
    assert len(seen) == (listener is not None) and a.is_contiguous() and torch.equal(a.view(9, -1), b.view(9, -1))
    up = torch.randn_like(a)
    got, want = (torch.autograd.grad(y, list(n.parameters()), up) for y, n in ((a, one), (b, other)))
    for g, w in zip(got, want, strict=True):
        assert rel(g, w) < 3 * 2.0 ** -8                        # (three blocks' roundings)


def test_a_frozen_first_block_in_training_mode_is_refused_as_before():
    """Without gradients a block runs on the running statistics, which a norm in training mode does not allow: also in front of a block that trains."""
    from fovi_b200.alexnet import KNNAlexNet
    net = KNNAlexNet(12, 16, [32, 48], [1, 1], [0], [9, 9], cmf_a=0.5, ref_frame_mult=2, norm_type="force_batch", device="cuda").train()
    net.layers[0].requires_grad_(False)
    x = torch.randn((9, 16, net.layers[0].in_coords.shape[0]), device="cuda")
    with pytest.raises(RuntimeError, match="eval"):
        net(x)
    net.layers[0].eval()
    net(x).sum().backward()
    assert net.layers[0].conv.weight.grad is None and net.layers[1].conv.weight.grad is not None
    assert net(x.clone().requires_grad_()).requires_grad


# one sample's slab shared by several CTAs: more CTAs than points to share, a remainder, no pool; slabs of 32, 16 and 8 channels
@pytest.mark.parametrize("N,C,n_out,K", [(5, 16, 3, 2), (230, 40, 61, 9), (1031, 16, 230, 9), (5602, 96, 1401, 5), (700, 32, 0, 0), (2001, 24, 0, 0)])
def test_one_sample_alone_and_in_a_batch(N, C, n_out, K):
    from fovi_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(N)
    h = torch.randn((200, C, N), generator=gen, device="cuda")
    plan = ops.KnnPoolPlan(torch.randint(0, N + 1, (K, n_out), generator=torch.Generator().manual_seed(N)).int().numpy(), N, device="cuda") if n_out else None
    out, arg = ops.relu_pool(h, True, plan)
    for b in (0, 199):
        one, who = ops.relu_pool(h[b:b + 1].contiguous(), True, plan)
        assert torch.equal(one[0], out[b]) and (plan is None or torch.equal(who[0], arg[b]))


@pytest.mark.parametrize("network", [False, True])
def test_running_statistics_that_are_held_still(network):
    """`track_running_stats = False` on a norm that has running statistics: batch statistics are used, the running ones are not written."""
    from fovi_b200.alexnet import KNNAlexNet
    torch.manual_seed(0)
    m = KNNAlexNet(12, 32, [64], [1], [0], [9], cmf_a=0.5, ref_frame_mult=2, norm_type="force_batch", device="cuda").train() if network else make().train()
    block = m.layers[0] if network else m
    x = torch.randn((7, 32, block.in_coords.shape[0]), device="cuda")
    want = m(x)
    assert block.norm.num_batches_tracked == 1
    block.norm.track_running_stats = False
    before = [b.clone() for b in block.norm.buffers()]
    got = m(x)
    assert torch.equal(got, want)
    for a, b in zip(before, block.norm.buffers(), strict=True):
        assert torch.equal(a, b)
