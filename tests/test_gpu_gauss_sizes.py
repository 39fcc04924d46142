"""The Gaussian MLE of small windows at the edges of the kernel's lane layout, against the FP64 oracle.

A ROI of up to 16 columns takes 16 lanes, a wider one 32; columns are rounded up to 8, 16 or 32. The
sizes below have idle lanes, one and several rows per step, odd strides, and ROI counts that leave half
a warp and most of a CTA empty. FP32 model terms (a few 1e-7 relative, random over the pixels) move a
bright spot's fit by about 1e-6 px, and a coordinate's own rounding is up to 2e-6: 2e-5 px is allowed.
"""
import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance

SIZES = [(6, 9), (8, 8), (9, 7), (15, 15), (16, 13), (16, 16), (17, 12), (25, 31), (32, 32)]


def spots(w, h, n, dtype, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    sigma = 0.125 * min(w, h)
    side = max(w, h)
    cx, cy = w / 2 + rng.uniform(-0.06, 0.06, n) * w, h / 2 + rng.uniform(-0.06, 0.06, n) * h
    ph = w * h * rng.uniform(4, 20, n)
    lam = synth.gaussian_spots(n, side, cx, cy, sigma, ph, 10.0)[:, :h, :w]
    return np.ascontiguousarray(rng.poisson(lam).astype(dtype)), sigma


@pytest.mark.gpu
@pytest.mark.parametrize("params", [4, 5])
@pytest.mark.parametrize("w,h", SIZES)
def test_gauss_window_sizes_match_fp64(port, w, h, params):
    iters, n = 14, 13
    for dtype in (np.float32, np.uint16):
        rois, sigma = spots(w, h, n, dtype, 100 * w + h)
        s = abi.settings(width=w, height=h, gauss2D_sigma=sigma, gauss2D_iterations=iters, qi_minradius=1,
                         zlut_minradius=0.25, qi_roi_coverage=1.0)
        with QTrkInstance(s) as t:
            t.SetLocalizationMode(abi.LT_Gaussian2D | (abi.LT_B200_Gaussian5P if params == 5 else 0))
            r = t.Localize(rois)
        checked = 0
        for i in range(n):
            img = rois[i].astype(np.float64)
            com = port.com(img)
            assert np.abs(r["firstGuess"][i] - com[:2]).max() < 1e-5

            def fit(e):  # from a start moved by the relative amount e
                m = com * (1 + e)
                return np.asarray(port.gauss2d(img, m[2], m[:2], iters, sigma) if params == 4 else
                                  port.gauss5(img, [m[0], m[1], m[2] * 0.5 * w * h, m[2] * 0.5, sigma], iters))

            com = np.asarray(com)
            want = fit(0.0)
            if not np.abs(want - fit(1e-6))[:2].max() < 5e-6:  # the iteration amplifies rounding: no defined answer
                continue
            checked += 1
            assert np.abs(r["pos"][i, :2] - want[:2]).max() < 2e-5
            if params == 5:
                assert abs(r["pos"][i, 2] - want[4]) < 2e-5
        assert checked >= n - 3


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", SIZES + [(33, 20)])
def test_gauss_nll_gradient_window_sizes_match_fp64(port, w, h):
    """Likelihood and gradient at the same sizes (33 columns: the CTA form). FP32 residuals of a few 1e-7
    relative, summed in FP64: 1e-6 of the likelihood and 1e-5 of each component's sum of magnitudes."""
    import torch

    n = 13
    for dtype in (np.float32, np.uint16):
        rois, sigma = spots(w, h, n, dtype, 7 * w + h)
        rng = np.random.Generator(np.random.PCG64(w + h))
        prm = np.stack([w / 2 + rng.uniform(-.5, .5, n), h / 2 + rng.uniform(-.5, .5, n), 10.0 * w * h * rng.uniform(.5, 1.5, n),
                        rng.uniform(8, 12, n), sigma * rng.uniform(.9, 1.1, n)], 1).astype(np.float32)
        px = torch.from_numpy(rois if dtype == np.float32 else rois.view(np.int16)).cuda()
        p, nll, grad = torch.from_numpy(prm).cuda(), torch.empty(n, device="cuda"), torch.empty(n, 5, device="cuda")
        s = abi.settings(width=w, height=h, gauss2D_sigma=sigma, qi_minradius=1, zlut_minradius=0.25)
        b = rois.itemsize
        with QTrkInstance(s) as t:
            assert t.lib.QTrkB200GaussianNLLGradient(t.handle, px.data_ptr(), w * b, w * h * b, abi.NUMPY_PDT[rois.dtype], n,
                                                     p.data_ptr(), nll.data_ptr(), grad.data_ptr(), None) == 0
            torch.cuda.synchronize()
        for i in range(n):
            want, g = port.gauss_nll_grad(rois[i].astype(np.float64), prm[i].astype(np.float64))
            assert abs(float(nll[i]) - want) < 1e-6 * max(abs(want), 10.0 * w * h)
            # each residual f is off by a few 1e-7 of max(f, 1); the derivative's magnitudes sum to `scale`
            for k in range(5):
                scale = max(1.0, abs(prm[i, 2]) if k in (0, 1, 4) else float(w * h if k == 3 else 1.0))
                assert abs(float(grad[i, k]) - g[k]) < 1e-5 * scale + 1e-5 * abs(g[k]), (i, k)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(234, 234), (235, 235), (236, 234)])
def test_gauss_windows_at_the_shared_memory_limit(port, w, h):
    """Windows that fit only in the compact layout, whose Gaussian form leaves no room for a raw ROI: fits against
    the FP64 oracle (FP32 terms over 55,000 pixels: 1e-3 px, the bound of QI positions), and a LUT built in that
    mode, whose ROIs do arrive raw, equal to the one built in a QI mode."""
    n, iters = 2, 14
    rois, sigma = spots(w, h, n, np.uint16, w + 3 * h)
    s = abi.settings(width=w, height=h, gauss2D_sigma=sigma, gauss2D_iterations=iters)
    luts = []
    for mode in (abi.LT_Gaussian2D, abi.LT_QI):
        with QTrkInstance(s) as t:
            t.SetLocalizationMode(mode)
            if mode == abi.LT_Gaussian2D:
                r = t.Localize(rois)
            t.SetRadialZLUTSize(n, 2)
            t.BeginLUT(abi.BUILDLUT_NORMALIZE)
            for plane in range(2):
                t.BuildLUT(rois, plane)
            t.FinalizeLUT()
            luts.append(t.GetRadialZLUT())
    assert np.isfinite(luts[0]).all() and np.abs(luts[0]).max() > 0
    np.testing.assert_array_equal(luts[0], luts[1])
    for i in range(n):
        img = rois[i].astype(np.float64)
        com = port.com(img)
        want = np.asarray(port.gauss2d(img, com[2], com[:2], iters, sigma))
        assert np.abs(r["pos"][i, :2] - want[:2]).max() < 1e-3
