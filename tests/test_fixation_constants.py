"""CPU: constant fixation arguments (the cached device copies of sensing._as_bf2) in the circumstances in which they are first met."""
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
