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
    if change is not dropped:                                   # (which elements are dropped depends on the memory order)
        assert torch.equal(got[0], want[0])
        for a, b in zip(got[1:], want[1:], strict=True):
            assert rel(a, b) < 2.0 ** -8                        # the gradient's bf16 roundings in between
