"""A ROI whose staged copy is late is given up, not localized from what happens to lie in shared memory: its result
is not a number, the LUT's gradient gets nothing from it, and GetWarnings says so. The copies are made late by a
wait limit of no polls; the kernels then give each copy its last bounded wait, so all have landed when they end.
"""
import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance, computed_config

pytestmark = pytest.mark.gpu
LIMIT = 1 << 22


def setup(w, n, dtype):
    rng = np.random.Generator(np.random.PCG64(w))
    lam = synth.render(w, w, w / 2 + rng.uniform(-1, 1, n), w / 2 + rng.uniform(-1, 1, n),
                       rng.uniform(0.1, 0.4, n) * w, 20.0, 180.0)
    rois = np.minimum(rng.poisson(lam), 255).astype(dtype)
    s = synth.settings_square(w)
    lut = rng.normal(size=(1, 30, computed_config(s).zlut_radialsteps)).astype(np.float32)
    return s, lut, rois


def device(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).cuda()


@pytest.mark.parametrize("mode", [synth.MODE_QI_Z, synth.MODE_QI_Z | abi.LT_B200_ZMatchBF16,
                                  synth.MODE_QI_Z | abi.LT_B200_JointRefine])
@pytest.mark.parametrize("w,dtype", [(48, np.uint8), (61, np.uint16), (80, np.float32)])
def test_late_localization(w, dtype, mode):
    import torch

    n = 20
    s, lut, rois = setup(w, n, dtype)
    d = device(rois)
    k = rois.itemsize
    with QTrkInstance(s) as t:
        t.SetRadialZLUT(lut)
        t.SetLocalizationMode(mode)
        runs = []
        for limit in (LIMIT, 0, LIMIT):
            t.SetCopyWaitLimit(limit)
            out = torch.zeros(n * 52, dtype=torch.uint8, device="cuda")
            t.LocalizeDevice(d.data_ptr(), w * k, w * w * k, abi.NUMPY_PDT[rois.dtype], n, out.data_ptr(),
                             stream=torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            runs.append(np.frombuffer(out.cpu().numpy().tobytes(), dtype=abi.RESULT_DTYPE))
            assert ("staged ROI copy" in t.GetWarnings()) == (limit == 0)
    for f in ("pos", "firstGuess", "imageMean"):
        assert np.isfinite(runs[0][f]).all() and np.array_equal(runs[0][f], runs[2][f]), f
        assert np.isnan(runs[1][f]).all(), f
    assert np.array_equal(runs[1]["frame"], np.arange(n)) and (runs[1]["error"] != 0).all()


@pytest.mark.parametrize("w,dtype", [(48, np.uint8), (61, np.uint16), (80, np.float32)])
def test_late_cost_gradient(w, dtype):
    import torch

    n = 20
    s, lut, rois = setup(w, n, dtype)
    d, k = device(rois), rois.itemsize
    xyz = torch.tensor([[w / 2, w / 2, 10.5]] * n, device="cuda")
    with QTrkInstance(s) as t:
        t.SetRadialZLUT(lut)
        t.SetLocalizationMode(synth.MODE_QI_Z)
        for limit in (0, LIMIT):
            t.SetCopyWaitLimit(limit)
            cost, grad = torch.zeros(n, device="cuda"), torch.zeros(n, 3, device="cuda")
            glut = torch.zeros(lut.shape, device="cuda")
            assert t.lib.QTrkB200ZLUTCostGradient(t.handle, d.data_ptr(), w * k, w * w * k, abi.NUMPY_PDT[rois.dtype], n,
                                                  xyz.data_ptr(), None, cost.data_ptr(), grad.data_ptr(),
                                                  glut.data_ptr(), None) == 0
            torch.cuda.synchronize()
            late = limit == 0
            assert torch.isnan(cost).all() == late and torch.isnan(grad).all() == late
            assert bool((glut == 0).all()) == late and torch.isfinite(glut).all()
            assert ("staged ROI copy" in t.GetWarnings()) == late


def test_late_lut_rows():
    w, planes = 48, 6
    s, _, _ = setup(w, 1, np.uint16)
    stack = synth.render(w, w, np.full(planes, w / 2), np.full(planes, w / 2), np.linspace(4, 20, planes), 200.0,
                         2000.0).astype(np.uint16)
    with QTrkInstance(s) as t:
        t.SetRadialZLUTSize(1, planes)
        t.BeginLUT(True)
        for k in range(planes):
            t.SetCopyWaitLimit(0 if k == 2 else LIMIT)
            t.BuildLUT(stack[k][None], k)
        t.FinalizeLUT()
        lut = t.GetRadialZLUT()
        assert "staged ROI copy" in t.GetWarnings()
    assert np.isnan(lut[0, 2]).all() and np.isfinite(np.delete(lut[0], 2, 0)).all()
