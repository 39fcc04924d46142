"""First guess (COM) of small Gaussian windows, which 16 lanes share: FP32 sums run over four pixels at most before
they meet in FP64, so what is left of the error is the rounding of the result itself to FP32. A tenth is allowed on
top of it.
"""
import numpy as np
import pytest

from qtrk_b200 import abi
from qtrk_b200.tracker import QTrkInstance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pitched", [False, True])
@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
@pytest.mark.parametrize("w", [12, 15])
def test_com_error_is_the_results_rounding(w, dtype, pitched):
    import torch

    n = 20000
    rng = np.random.default_rng(w)
    at = np.arange(w)
    c = w / 2 - 0.5 + rng.uniform(-1, 1, (n, 2))
    gx = np.exp(-0.5 * ((at - c[:, :1]) / 2.0) ** 2)
    gy = np.exp(-0.5 * ((at - c[:, 1:]) / 2.0) ** 2)
    rois = rng.poisson(10.0 + 120.0 * gy[:, :, None] * gx[:, None, :]).astype(dtype)
    img = rois.astype(np.float64)
    d = np.abs(img - img.mean((1, 2))[:, None, None])
    want = np.stack([(d.sum(1) * at).sum(1), (d.sum(2) * at).sum(1)], 1) / d.sum((1, 2))[:, None]
    row = w + 4 if pitched else w
    buf = np.zeros((n, w, row), dtype)
    buf[:, :, :w] = rois
    s = abi.settings(width=w, height=w, gauss2D_sigma=2.0, gauss2D_iterations=1, qi_minradius=0.5, zlut_minradius=0.5)
    with QTrkInstance(s) as t:
        t.SetLocalizationMode(abi.LT_Gaussian2D)
        px = torch.from_numpy(buf.view(np.uint8)).cuda()
        out = torch.zeros(n * 52, dtype=torch.uint8, device="cuda")
        b = rois.itemsize
        t.LocalizeDevice(px.data_ptr(), row * b, row * w * b, abi.NUMPY_PDT[rois.dtype], n, out.data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        r = np.frombuffer(out.cpu().numpy().tobytes(), dtype=abi.RESULT_DTYPE)
    err = np.abs(r["firstGuess"].astype(np.float64) - want).mean()
    rounding = np.abs(want.astype(np.float32) - want).mean()
    assert err < 1.1 * rounding
    assert np.abs(r["imageMean"] - img.mean((1, 2))).max() < 1e-5
