"""The bias sums of a masked input gradient belong to that gradient: passes over one graph that run at the same time, and hooks between the layers, leave every
gradient right.  The kernels are replaced by plain torch (float64 references of the same gradients come from autograd on plain torch)."""
import threading

import pytest
import torch

pytestmark = pytest.mark.autograd
B, N, CHANNELS = 6, 5, (16, 24, 8)


class _Plan:
    tc_supported, x_layout = True, 0

    @staticmethod
    def forward(x, w, bias, relu=False, out_dtype=None, batch=None):
        y = x.float() @ w.float().t() + (0 if bias is None else bias)
        return (torch.relu(y) if relu else y).to(out_dtype)


class _Grads:
    """Gradients of a layer whose every point has itself as only neighbour."""

    def __init__(self):
        self.masked, self.after_masked = 0, lambda: None

    def masking_pays(self, rows):
        return True

    def input_grad(self, gy, weight):
        return (gy.float() @ weight.float()).to(torch.bfloat16)

    def input_grad_masked(self, gy, weight, act):
        g = self.input_grad(gy, weight) * (act > 0)
        self.masked += 1
        return g, g.float().sum((0, 1))

    def weight_grad(self, gy, x, plan, dtype):
        self.after_masked()
        return torch.einsum("bno,bnc->oc", gy.float(), x.float()).to(dtype)


class _Layer(torch.nn.Module):
    precision = "bf16"

    def __init__(self, c_in, c_out):
        super().__init__()
        self.in_channels, self.out_channels, self.plan, self.grad_plans = c_in, c_out, _Plan(), _Grads()
        self.weight, self.bias = torch.nn.Parameter(torch.randn(c_out, c_in) / 4), torch.nn.Parameter(torch.randn(c_out) / 4)

    def packed_weight(self):
        return self.weight.detach()


@pytest.fixture
def stack(monkeypatch):
    from fovi_b200 import ops
    from fovi_b200.knn import KNNConvStack

    def mask(g, act):
        m = g * (act > 0)
        return m, m.float().sum((0, 1))
    monkeypatch.setattr(ops, "relu_mask_colsum", mask)
    monkeypatch.setattr(ops, "column_sum", lambda g: g.float().sum((0, 1)))
    torch.manual_seed(0)
    return KNNConvStack([_Layer(a, b) for a, b in zip(CHANNELS, CHANNELS[1:])], final_relu=True)


def run(stack, seed):
    x = torch.randn((B, CHANNELS[0], N), generator=torch.Generator().manual_seed(seed))
    return stack(x), list(stack.parameters())


def ups(k):
    return [torch.randn((B, CHANNELS[-1], N), generator=torch.Generator().manual_seed(10 + i)) * 10 ** i for i in range(k)]


def alone(stack, monkeypatch, y, params, up):
    """The gradients with the masking pass on its own."""
    with monkeypatch.context() as m:
        for L in stack.layers:
            m.setattr(L.grad_plans, "input_grad_masked", lambda *a: None)
        return torch.autograd.grad(y, params, up, retain_graph=True)


def same(got, want):
    return all(torch.equal(a, b) for a, b in zip(got, want, strict=True))


def test_sums_travel_with_their_gradient(stack, monkeypatch):
    y, params = run(stack, 1)
    up, = ups(1)
    want = alone(stack, monkeypatch, y, params, up)
    calls = []
    from fovi_b200 import ops
    both = ops.relu_mask_colsum
    monkeypatch.setattr(ops, "relu_mask_colsum", lambda *a: calls.append(1) or both(*a))
    assert same(torch.autograd.grad(y, params, up, retain_graph=True), want)
    assert len(calls) == 1 and stack.layers[1].grad_plans.masked == 1          # the top layer's; the other one's sums came with its gradient


def test_two_threads_on_one_retained_graph(stack, monkeypatch):
    y, params = run(stack, 2)
    up = ups(2)
    want = [alone(stack, monkeypatch, y, params, u) for u in up]
    first_in, second_in, first_done, got = threading.Event(), threading.Event(), threading.Event(), [None, None]

    def order():                       # the upper layer's kernel of the first pass, of the second, then the lower layer of the first
        if threading.current_thread().name == "0":
            first_in.set()
            assert second_in.wait(20)
        else:
            second_in.set()
            assert first_done.wait(20)

    def work(i):
        if i:
            assert first_in.wait(20)
        got[i] = torch.autograd.grad(y, params, up[i], retain_graph=True)
        if not i:
            first_done.set()
    stack.layers[1].grad_plans.after_masked = order
    threads = [threading.Thread(target=work, args=(i,), name=str(i)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert same(got[0], want[0]) and same(got[1], want[1])


@pytest.mark.parametrize("change", [lambda g: g * 3, lambda g: g.mul_(3), lambda g: g.clone(), lambda g: None], ids=["new", "in place", "copy", "nothing"])
def test_a_hook_between_the_layers(stack, monkeypatch, change):
    y, params = run(stack, 3)
    up, = ups(1)
    node = next(n for n, _ in _walk(y.grad_fn) if n.name().startswith("_KnnConvPointsFunction"))     # the top layer's
    lower = node.next_functions[0][0]

    def hook(grads):
        new = change(grads[0])
        return None if new is None or new is grads[0] else (new,)
    handle = lower.register_prehook(hook)
    want = alone(stack, monkeypatch, y, params, up)
    got = torch.autograd.grad(y, params, up, retain_graph=True)
    handle.remove()
    assert same(got, want)


def _walk(fn, depth=0):
    yield fn, depth
    for n, _ in fn.next_functions:
        if n is not None:
            yield from _walk(n, depth + 1)


def test_sums_of_one_pass_do_not_reach_another(stack, monkeypatch):
    """A pass that stops above the lower layer leaves nothing behind; a hook that hands in another pass's gradient gets the sums of that gradient."""
    y, params = run(stack, 4)
    up = ups(2)
    want = [alone(stack, monkeypatch, y, params, u) for u in up]
    torch.autograd.grad(y, params[2:], up[1], retain_graph=True)
    assert same(torch.autograd.grad(y, params, up[0], retain_graph=True), want[0])
    node = next(n for n, _ in _walk(y.grad_fn) if n.name().startswith("_KnnConvPointsFunction"))
    kept = []
    handle = node.next_functions[0][0].register_prehook(lambda g: kept.append(g[0]))
    torch.autograd.grad(y, params, up[0], retain_graph=True)
    handle.remove()
    handle = node.next_functions[0][0].register_prehook(lambda g: (kept[0],))
    got = torch.autograd.grad(y, params, up[1], retain_graph=True)
    handle.remove()
    assert same(got[:2], want[0][:2]) and same(got[2:], want[1][2:])           # the lower layer's of pass 0, the upper layer's of pass 1


def test_backward_in_inference_mode(stack, monkeypatch):
    y, params = run(stack, 5)
    up, = ups(1)
    want = alone(stack, monkeypatch, y, params, up)
    with torch.inference_mode():
        got = torch.autograd.grad(y, params, up.clone(), retain_graph=True)
    assert same(got, want)
