"""The localization kernel's tile: formats, alignments, CTA widths and layouts.

Whatever way a ROI reaches the kernel, its result is the same bit for bit: the pixel sums, the COM's chains and
the circles' direction subsets are cut alike in every form. Against the FP64 oracle the parity tests'
tolerances hold (COM 1e-4 px, QI 1e-3 px, Z 0.01 plane).
"""
import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance, computed_config

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "firstGuess", "error", "imageMean")


def beads(w, n, dtype, seed=3):
    rng = np.random.Generator(np.random.PCG64(seed * 1000 + w))
    cx, cy = w / 2 + rng.uniform(-0.03, 0.03, n) * w, w / 2 + rng.uniform(-0.03, 0.03, n) * w
    bg, amp, top = (200.0, 2000.0, 4095) if dtype == np.uint16 else (20.0, 180.0, 255)
    lam = synth.render(w, w, cx, cy, rng.uniform(0.1, 0.45, n) * w, bg, amp)
    return np.minimum(rng.poisson(8 * lam) // 8, top).astype(dtype)


def device_run(t, rois, offset=0, jobs=None):
    """LocalizeDevice on a stack that starts `offset` pixels into its buffer."""
    import torch

    n, _, w = rois.shape
    flat = np.zeros(offset + rois.size, rois.dtype)
    flat[offset:] = rois.ravel()
    d = torch.from_numpy(flat.view(np.uint8)).cuda()
    out = torch.zeros(n * 52, dtype=torch.uint8, device="cuda")
    b = rois.itemsize
    t.LocalizeDevice(d.data_ptr() + offset * b, w * b, w * w * b, abi.NUMPY_PDT[rois.dtype], n, out.data_ptr(),
                     stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return np.frombuffer(out.cpu().numpy().tobytes(), dtype=abi.RESULT_DTYPE)


def same(a, b, note):
    for f in FIELDS:
        assert np.array_equal(a[f], b[f]), (note, f)


def tracker(s, lut, mode=synth.MODE_QI_Z):
    t = QTrkInstance(s)
    t.SetRadialZLUT(lut)
    t.SetLocalizationMode(mode)
    return t


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("w,bg", [(40, 0.0), (61, 0.5), (64, 0.0), (78, 0.0), (99, 0.5), (100, 0.0), (128, 0.5)])
def test_every_form_gives_the_same_bits(w, bg, dtype):
    n = 1200
    few = beads(w, 40, dtype)
    rois = np.ascontiguousarray(few[np.arange(n) % 40])
    s = synth.settings_square(w, com_bgcorrection=bg)
    cc = computed_config(s)
    lut = np.random.default_rng(w).normal(size=(1, 60, cc.zlut_radialsteps)).astype(np.float32)
    with tracker(s, lut) as t:
        for clear in (0, abi.LT_ClearFirstFourPixels):
            t.SetLocalizationMode(synth.MODE_QI_Z | clear)
            ref = device_run(t, few[:1])                     # one CTA per SM at most: the widest form
            many = device_run(t, rois)                       # several per SM: 128 threads
            same(many[:1], ref, "count")
            same(many[:40], device_run(t, few), "count 40")
            same(many[:250], device_run(t, rois[:250]), "count 250")
            same(many[:40], many[40:80], "repeat")
            for off in (1, 3, 8):                            # unaligned stacks
                same(many[:300], device_run(t, rois[:300], off), f"offset {off}")
            if dtype != np.float32:                          # float tile of the same pixel values
                same(many[:300], device_run(t, rois[:300].astype(np.float32)), "float")
            # frame bands: ROIs cropped at odd positions (bead 0's LUT only for the first)
            cols = 6
            frame = np.zeros((7 * (w + 3), cols * (w + 1) + 1), dtype)
            pos = [(1 + (k % cols) * (w + 1), (k // cols) * (w + 3)) for k in range(40)]
            for k, (x, y) in enumerate(pos):
                frame[y:y + w, x:x + w] = few[k]
            assert t.ScheduleFrame(frame, np.array(pos, np.int32)) == 40
            r = t.WaitForResults(40)
            r = r[np.argsort(r["zlutIndex"])]
            assert np.array_equal(r["pos"][:, :2], many["pos"][:40, :2])
            for f in FIELDS[1:]:
                if f != "error":
                    assert np.array_equal(r[f], many[f][:40]), f
            same(r[:1], many[:1], "frame")


@pytest.mark.parametrize("w,dtype,radial,n", [
    (24, np.uint8, 0.9, 12),                                  # 2 nr = 16: transform through shared memory
    (37, np.uint16, 1.4, 12), (64, np.float32, 0.6, 12),      # 2 nr = 32
    (75, np.uint8, 1.4, 12), (75, np.uint8, 1.4, 700),        # 64
    (100, np.uint16, 1.4, 12), (100, np.uint16, 1.4, 700),    # 128
    (101, np.float32, 2.6, 8),                                # 256
    (64, np.uint16, 8.0, 8),                                  # 512
    (64, np.uint8, 16.0, 6),                                  # 1024: shared memory again
    (236, np.uint16, 1.4, 3), (237, np.uint8, 1.4, 3)])       # compact and packed shared-memory layouts
def test_sizes_match_fp64(port, w, dtype, radial, n):
    few = beads(w, min(n, 12), dtype, seed=5)
    rois = np.ascontiguousarray(few[np.arange(n) % len(few)])
    s = synth.settings_square(w, qi_radial_coverage=radial)
    if w < 32:
        s.qi_minradius = s.zlut_minradius = 1.0
    cc = computed_config(s)
    planes = 50
    stack = synth.render(w, w, np.full(planes, w / 2), np.full(planes, w / 2), np.linspace(0.05, 0.5, planes) * w, 200.0,
                         2000.0).astype(np.float32)
    with QTrkInstance(s) as t:
        t.SetRadialZLUTSize(1, planes)
        t.BeginLUT(True)
        for k in range(planes):
            t.BuildLUT(stack[k][None], k, known_pos=np.array([[w / 2, w / 2]], np.float32))
        t.FinalizeLUT()
        lut = t.GetRadialZLUT()
    want_lut = port.build_lut(cc, stack[:, None], 4, known_pos=np.array([[w / 2, w / 2]], np.float32))
    assert np.abs(lut - want_lut).max() < 1e-4
    with tracker(s, lut) as t:
        r = device_run(t, rois)
    want = port.localize(cc, synth.MODE_QI_Z, few, lut)
    want = want[np.arange(n) % len(few)]
    assert np.abs(r["firstGuess"] - want[:, 3:5]).max() < 1e-4
    assert np.abs(r["pos"][:, :2] - want[:, :2]).max() < 1e-3
    inside = (want[:, 2] > 1) & (want[:, 2] < planes - 2)
    assert inside.any()
    assert np.abs(r["pos"][inside, 2] - want[inside, 2]).max() < 0.01
    assert np.abs(r["imageMean"] - want[:, 6]).max() < 1e-3


@pytest.mark.parametrize("w,dtype", [(48, np.uint8), (61, np.uint16), (75, np.uint8), (80, np.uint16), (81, np.float32),
                                     (100, np.uint8), (237, np.uint16)])
def test_cost_gradient_sizes_match_fp64(port, w, dtype):
    """The adjoint over every tile format, whole and ragged rows, aligned and unaligned stacks, circles inside the
    image and across its edge. FP32 samples: 2e-4 of the cost; a sample within rounding of a pixel edge may take
    the neighbouring cell's derivative, one of a bin's samples in one bin: 5e-3 of the largest component."""
    import torch

    n = 10
    rois = beads(w, n, dtype, seed=7)
    s = synth.settings_square(w)
    cc = computed_config(s)
    rng = np.random.default_rng(w)
    planes = 20
    lut = rng.normal(size=(3, planes, cc.zlut_radialsteps)).astype(np.float32)
    beads_of = (np.arange(n) % 3).astype(np.int32)
    xyz = np.stack([w / 2 + rng.uniform(-1, 1, n), w / 2 + rng.uniform(-1, 1, n), rng.uniform(0, planes - 1, n)], 1)
    xyz[-2:, :2] += w * 0.3  # circles leave the image
    xyz = xyz.astype(np.float32)
    with tracker(s, lut) as t:
        outs = []
        for off in (0, 3):
            flat = np.zeros(off + rois.size, dtype)
            flat[off:] = rois.ravel()
            px, d = torch.from_numpy(flat.view(np.uint8)).cuda(), torch.from_numpy(xyz).cuda()
            b = torch.from_numpy(beads_of).cuda()
            cost, grad = torch.empty(n, device="cuda"), torch.empty(n, 3, device="cuda")
            glut = torch.zeros(lut.shape, device="cuda")
            k = rois.itemsize
            assert t.lib.QTrkB200ZLUTCostGradient(t.handle, px.data_ptr() + off * k, w * k, w * w * k,
                                                  abi.NUMPY_PDT[rois.dtype], n, d.data_ptr(), b.data_ptr(),
                                                  cost.data_ptr(), grad.data_ptr(), glut.data_ptr(), None) == 0
            torch.cuda.synchronize()
            outs.append([v.cpu().numpy().astype(np.float64) for v in (cost, grad, glut)])
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    cost, grad, glut = outs[0]
    want_l = np.zeros(lut.shape)
    for i, img in enumerate(rois.astype(np.float64)):
        c, g, gl = port.zcost_grad(img, img.mean(), xyz[i].astype(np.float64), lut[beads_of[i]], cc.zlut_angularsteps,
                                   s.zlut_minradius, cc.zlut_maxradius, want_lut_grad=True)
        want_l[beads_of[i]] += gl
        assert abs(cost[i] - c) < 2e-4 * c
        assert np.abs(grad[i] - g).max() < 5e-3 * np.abs(g).max()
    assert np.abs(glut - want_l).max() < 2e-3 * np.abs(want_l).max()


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("w", [8, 12, 28, 36, 52, 56, 64, 76, 96, 100, 112, 116, 128, 160, 200])
def test_com_only_sizes_match_fp64(w, dtype):
    """LT_OnlyCOM over the widths that change its form, its warps per ROI and its ROIs in flight, with one ROI, a few
    and more than the GPU holds at once. FP32 sums of at most 32 pixels: 2e-5 px; means of integers to one ulp."""
    few = beads(w, 37, dtype, seed=9)
    img = few.astype(np.float64)
    s = synth.settings_square(w)
    if w < 32:
        s.qi_minradius = s.zlut_minradius = 0.25
    for clear in (0, abi.LT_ClearFirstFourPixels):
        if clear:
            img[:, 0, :4] = 0
        mean = img.mean((1, 2))
        d = np.abs(img - mean[:, None, None])
        at = np.arange(w)
        want = np.stack([(d.sum(1) * at).sum(1), (d.sum(2) * at).sum(1)], 1) / d.sum((1, 2))[:, None]
        with QTrkInstance(s) as t:
            t.SetLocalizationMode(abi.LT_OnlyCOM | clear)
            for n in (1, 7, 37, 3000 if w <= 128 else 400):
                rois = np.ascontiguousarray(few[np.arange(n) % 37])
                r = device_run(t, rois)
                k = np.arange(n) % 37
                assert np.abs(r["pos"][:, :2] - want[k]).max() < 2e-5
                assert np.array_equal(r["pos"][:, :2], r["firstGuess"])
                assert np.abs(r["imageMean"] - mean[k]).max() <= 2e-7 * mean.max() + 1e-7
                assert np.array_equal(r["frame"], np.arange(n))
