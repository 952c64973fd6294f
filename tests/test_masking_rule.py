"""When an input gradient takes its ReLU mask along and when the separate pass is the faster one (grad.KnnConvGrad.masking_pays)."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("c_in,c_out,K,n,rows,pays", [
    (512, 64, 1, 1000, 129, False), (512, 64, 1, 1000, 256, True), (512, 64, 1, 1000, 300, False), (512, 64, 1, 1000, 342, True), (512, 64, 12, 1000, 129, True),
    (256, 256, 1, 1000, 129, False), (256, 256, 3, 1000, 129, True), (512, 64, 1, 60, 129, True), (64, 192, 9, 1000, 129, True), (64, 192, 25, 1023, 1024, True)])
def test_masking_pays(c_in, c_out, K, n, rows, pays):
    from fovi_b200.grad import KnnConvGrad
    g = KnnConvGrad(np.tile(np.arange(n), (K, 1)), np.zeros((n, K)), n, 1, c_in, c_out, torch.device("cpu"))
    assert g.masking_pays(rows) == pays
