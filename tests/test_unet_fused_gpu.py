"""The network's forward pass where its fused pooling and output layer meet tile edges and several z
columns, against the numpy statement."""
import numpy as np
import pytest

from oracle import unet_ref as U
from tests.test_unet_gpu import dev, net_with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 4, 4), (12, 20, 12), (8, 36, 24), (44, 8, 20)])
def test_forward_fused_layers(gpu_lib, shape):
    """What differs is the order of the FP32 accumulations and BF16 ties, a few BF16 ulps (2^-8 each) of
    a layer's inputs: 8e-3 of the output's maximum, as for the forward pass elsewhere."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(19)
    r, lnk = (rng.standard_normal(shape).astype(np.float32) for _ in range(2))
    cap = rng.uniform(0, 1, shape).astype(np.float32)
    params = U.init_params(5)
    h = net_with(gpu_lib, params)
    nz, ny, nx = shape
    tr, tk, tc = dev(torch, r), dev(torch, lnk), dev(torch, cap)
    y = torch.empty_like(tr)
    assert gpu_lib.frehg_unet_forward(h, nx, ny, nz, tr.data_ptr(), tk.data_ptr(), tc.data_ptr(),
                                      y.data_ptr(), None) == 0
    yref, _, rms = U.forward(params, r, lnk, cap)
    assert np.abs(y.cpu().numpy() - yref * rms).max() <= 8e-3 * np.abs(yref * rms).max()
    gpu_lib.frehg_unet_destroy(h)
