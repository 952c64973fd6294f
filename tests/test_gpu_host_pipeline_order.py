"""GPU: run_from_host returns with its copies queued; the stream it was called on waits for the last byte of the pinned result."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_completion_is_ordered_on_the_calling_stream():
    from fovi_b200.coords import get_in_out_coords
    from fovi_b200.knn import KNNConvLayer, KNNConvStack
    from fovi_b200.pipeline import FoveatedFrontEnd
    from fovi_b200.sensing import RetinalTransform
    rt = RetinalTransform(resolution=20, start_res=64, fov=16, cmf_a=1.0, sampler="grid_bilinear", fixation_size=64, device="cuda", auto_match_cart_resources=0)
    _, oc, _ = get_in_out_coords(20, 16, 1.0, 2, auto_match_cart_resources=0)
    torch.manual_seed(3)
    front = FoveatedFrontEnd(rt, KNNConvStack([KNNConvLayer(3, 64, 9, rt.sampler.coords, oc, device="cuda", ref_frame_side_length=3)]))
    B, F = 64, 4
    rs = np.random.RandomState(0)
    img = torch.from_numpy(rs.random_sample((B, 3, 64, 64)).astype(np.float32)).pin_memory()
    fix = torch.from_numpy((0.2 + 0.6 * rs.random_sample((B, F, 2))).astype(np.float32)).pin_memory()
    want = front.forward(img.cuda(), fix.cuda()).view(F, B, len(oc), 64).permute(1, 0, 2, 3).cpu()
    out = torch.zeros((B, F, len(oc), 64), dtype=torch.bfloat16).pin_memory()
    side = torch.cuda.Stream()
    for stream in (torch.cuda.current_stream(), side):
        out.zero_()
        with torch.cuda.stream(stream):
            front.run_from_host(img, fix, out)
            done = stream.record_event()
        done.synchronize()                       # this event alone, not the device
        assert torch.equal(out, want)
