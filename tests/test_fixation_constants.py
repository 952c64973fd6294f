"""Constant fixation arguments (the cached device copies of sensing._as_bf2) in the circumstances in which they are first met (on CPU tensors, and captured on the GPU)."""
import pytest
import torch


@pytest.fixture
def sensing(monkeypatch):
    from fovi_b200 import sensing
    monkeypatch.setattr(sensing, "_CONST_CACHE", {})
    return sensing


@pytest.mark.parametrize("value", [(96, 96.0), [64, 48], 32])
@pytest.mark.parametrize("F", [1, 3])
def test_first_use_under_inference_mode_leaves_a_normal_tensor(sensing, value, F):
    """An inference tensor in the cache could not be saved for a later call's backward pass (image gradients of the sensor)."""
    cpu = torch.device("cpu")
    with torch.inference_mode():
        sensing._as_bf2(value, 4, cpu, "fixation_size", F)
    t, _ = sensing._as_bf2(value, 4, cpu, "fixation_size", F)
    assert t.shape == (4, F, 2) and not t.is_inference()


@pytest.mark.parametrize("warm,F", [(1, 3), (3, 1), (2, 5)])
def test_a_new_fixation_count_inside_a_capture_uploads_nothing(sensing, monkeypatch, warm, F):
    """A stream capture may not copy from the host: a constant that has been used with this batch is repeated from its device copy, and what the
    graph's own memory holds is not kept for later calls."""
    class Cuda:
        type = "cuda"
    cpu = torch.device("cpu")
    for value in ((96, 48.0), [64, 32]):
        sensing._as_bf2(value, 4, cpu, "fixation_size", warm)
        before = dict(sensing._CONST_CACHE)
        with monkeypatch.context() as m:
            m.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
            m.setattr(sensing.torch, "device", lambda d: Cuda())
            m.setattr(torch, "as_tensor", lambda *a, **k: pytest.fail("host copy inside a capture"))
            t, multi = sensing._as_bf2(value, 4, cpu, "fixation_size", F)
        assert not multi and t.shape == (4, F, 2) and t.is_contiguous()
        assert (t == torch.tensor([float(v) for v in value])).all()
        assert sensing._CONST_CACHE.keys() == before.keys()


@pytest.mark.gpu
@pytest.mark.parametrize("warm,F", [(1, 3), (4, 2)])
def test_captured_sensor_call_with_a_new_fixation_count(sensing, warm, F):
    retina = sensing.RetinalTransform(24, start_res=64, sampler="grid_bilinear", device="cuda")
    x = torch.rand(2, 3, 64, 64, device="cuda")
    fix = {n: torch.rand(2, n, 2, device="cuda") for n in (warm, F)}
    retina(x, fix[warm])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = retina(x, fix[F])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, retina(x, fix[F]))
