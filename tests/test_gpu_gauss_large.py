"""Gaussian windows above 32x32 on both sides of the rule that picks the kernel by the CTAs an SM's shared memory
holds (5 parameters: 88 and 89 px more than five, 90 px five, 100 and 140 px fewer): fits against the FP64 oracle (1e-3
px, the bound of QI positions), and the same bits with a Z-LUT of many planes, which moves 88 and 89 px windows to
the other kernel.
"""
import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance, computed_config

pytestmark = pytest.mark.gpu


def spots(w, n):
    rng = np.random.Generator(np.random.PCG64(w))
    sigma = 0.125 * w
    lam = synth.gaussian_spots(n, w, w / 2 + rng.uniform(-0.06, 0.06, n) * w, w / 2 + rng.uniform(-0.06, 0.06, n) * w, sigma,
                               w * w * rng.uniform(4, 20, n), 10.0)
    return rng.poisson(lam).astype(np.float32), sigma


@pytest.mark.parametrize("params", [4, 5])
@pytest.mark.parametrize("w", [34, 61, 88, 89, 90, 100, 140])
def test_every_kernel_matches_fp64(port, w, params):
    n, iters = 3, 10
    rois, sigma = spots(w, n)
    s = abi.settings(width=w, height=w, gauss2D_sigma=sigma, gauss2D_iterations=iters, qi_minradius=1, zlut_minradius=1)
    mode = abi.LT_Gaussian2D | (abi.LT_B200_Gaussian5P if params == 5 else 0)
    nb = computed_config(s).zlut_radialsteps
    xy = []
    for planes in (0, 10, 1500):                         # 12 KB of scores: fewer CTAs per SM
        with QTrkInstance(s) as t:
            if planes:
                t.SetRadialZLUT(np.random.default_rng(1).normal(size=(1, planes, nb)).astype(np.float32))
            t.SetLocalizationMode(mode | (abi.LT_LocalizeZ if planes else 0))
            xy.append(t.Localize(rois)["pos"][:, :2])
    assert np.array_equal(xy[0], xy[1]) and np.array_equal(xy[0], xy[2])
    for i in range(n):
        img = rois[i].astype(np.float64)
        com = port.com(img)
        want = (port.gauss2d(img, com[2], com[:2], iters, sigma) if params == 4 else
                port.gauss5(img, [com[0], com[1], com[2] * 0.5 * w * w, com[2] * 0.5, sigma], iters))
        assert np.abs(xy[0][i] - want[:2]).max() < 1e-3
