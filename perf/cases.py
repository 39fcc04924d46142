"""Performance cases of the localization library: what its users run, through the public entry points.

Each case is a dict of plain values; ``kind`` names the path:

* ``track``    COM + QI + Z-LUT localization of a ROI stack in device memory (`LocalizeDevice`): the
               library's main path, per camera frame or per batch of frames;
* ``com``      the same entry with LT_OnlyCOM, the fast first look at a stack;
* ``gauss``    the 2D Gaussian MLE (4 parameters as in QTrk, or 5 with a free width) of small spots;
* ``zgrad``    the adjoint of the Z match: cost and its gradients with respect to (x, y, z) and the
               LUT, over a calibration stack (`QTrkB200ZLUTCostGradient`);
* ``ggrad``    the adjoint of the Gaussian MLE (`QTrkB200GaussianNLLGradient`);
* ``frame``    a pinned camera frame on the host through ScheduleFrame, Flush and GetResults;
* ``buildlut`` a calibration run: BeginLUT, one BuildLUT per plane from pinned host memory,
               FinalizeLUT and the finished LUT read back.

Images are the bead family p_z(r) = exp(-r^2 / (2 (4 + 0.1 z)^2)) cos(2 pi r / (6 + 0.05 z)) with
Poisson noise (u16: 12-bit, background 200, amplitude 2000; u8 and f32: 20 and 200), the LUT's planes
spanning z = 0 to half the ROI's width, or integrated Gaussian spots of 1000-5000 photons (at 16x16;
in proportion to the window's area), made on the GPU from the seed. ``exact`` restates every path in
FP64 with plain torch.
"""
from __future__ import annotations

import math
import time

import numpy as np
import torch

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance

F64 = torch.float64
BPP = {"u8": 1, "u16": 2, "f32": 4}
PDT = {"u8": abi.QTrkU8, "u16": abi.QTrkU16, "f32": abi.QTrkFloat}
TORCH_DTYPE = {"u8": torch.uint8, "u16": torch.int16, "f32": torch.float32}  # u16 pixels stay below 4096
NUMPY_DTYPE = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32}
QI_WEIGHTS = (0.14, 0.5, 0.85, 1.0, 0.85, 0.5, 0.14)
ZLUT_WEIGHTS = (0.15, 0.5, 0.85, 1.0, 0.85, 0.5, 0.15)
PI = 3.141593  # the angle constant of QTrk's direction tables


def listed() -> list[dict]:
    return [
        # one small frame of a live experiment: 50 beads, each with its own LUT; latency decides
        dict(name="track_128_u8_50", kind="track", width=128, dtype="u8", rois=50, planes=200, luts=50,
             weighted=False, bg=0.0),
        # a 1,000-bead frame of float ROIs (pre-processed images)
        dict(name="track_60_f32_1000", kind="track", width=60, dtype="f32", rois=1000, planes=50, luts=1,
             weighted=False, bg=0.0),
        # a 1,000-bead frame, every bead matched against its own LUT
        dict(name="track_64_u16_1000", kind="track", width=64, dtype="u16", rois=1000, planes=150, luts=1000,
             weighted=False, bg=0.0),
        # odd ROI size with radial weights and COM background correction switched on
        dict(name="track_75_u8_3001", kind="track", width=75, dtype="u8", rois=3001, planes=100, luts=1,
             weighted=True, bg=0.5),
        # the benchmark's workload: a batch of frames
        dict(name="track_100_u16_10000", kind="track", width=100, dtype="u16", rois=10000, planes=200, luts=1,
             weighted=False, bg=0.0),
        # centre of mass only, the benchmark's stack
        dict(name="com_100_u16_10000", kind="com", width=100, dtype="u16", rois=10000, bg=0.0),
        # a single-molecule movie: 100,000 spots, QTrk's 4-parameter fit
        dict(name="gauss4_16_f32_100000", kind="gauss", width=16, dtype="f32", rois=100000, params=4, sigma=2.0),
        # raw camera spots in an odd window, 5-parameter fit
        dict(name="gauss5_15_u16_20000", kind="gauss", width=15, dtype="u16", rois=20000, params=5, sigma=1.8),
        # gradients over a whole calibration stack, as LUT refinement asks for them
        dict(name="zgrad_80_u16_51200", kind="zgrad", width=80, dtype="u16", beads=256, planes=200, weighted=False),
        # gradients of the spot likelihood
        dict(name="ggrad_16_f32_50000", kind="ggrad", width=16, dtype="f32", rois=50000, sigma=2.0),
        # a camera frame on the host, one bead LUT per ROI, results back on the host
        dict(name="frame_100_u16_1000", kind="frame", width=100, dtype="u16", rois=1000, planes=200),
        # calibration of 256 beads, 40 planes
        dict(name="buildlut_80_u16_256x40", kind="buildlut", width=80, dtype="u16", beads=256, planes=40),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["track", "track", "track", "com", "gauss", "zgrad", "ggrad", "frame", "buildlut"])
    if kind == "track":
        w, dt = rng.randint(36, 128), rng.choice(["u8", "u16", "u16", "f32"])
        n = _log_int(rng, 16, min(10000, 100_000_000 // (w * w)))
        return dict(kind=kind, width=w, dtype=dt, rois=n, planes=rng.randint(40, 200),
                    luts=n if n <= 1000 and rng.random() < 0.5 else 1, weighted=rng.random() < 0.3,
                    bg=rng.choice([0.0, 0.0, 0.5]))
    if kind == "com":
        w = rng.randint(24, 128)
        return dict(kind=kind, width=w, dtype=rng.choice(["u8", "u16", "f32"]),
                    rois=_log_int(rng, 100, min(20000, 100_000_000 // (w * w))), bg=rng.choice([0.0, 0.0, 0.5]))
    if kind in ("gauss", "ggrad"):
        w = rng.randint(12, 24)
        c = dict(kind=kind, width=w, dtype=rng.choice(["f32", "u16"]), sigma=round(w * rng.choice([0.11, 0.125, 0.14]), 2),
                 rois=_log_int(rng, 200, 25_600_000 // (w * w)))
        if kind == "gauss":
            c["params"] = rng.choice([4, 5])
        else:
            c["rois"] = min(c["rois"], 50000)
        return c
    if kind == "zgrad":
        w, planes = rng.randint(48, 100), rng.randint(20, 200)
        return dict(kind=kind, width=w, dtype=rng.choice(["u8", "u16"]), planes=planes,
                    beads=_log_int(rng, 2, min(256, 320_000_000 // (w * w * planes))), weighted=rng.random() < 0.3)
    if kind == "frame":
        w, dt = rng.randint(36, 128), rng.choice(["u8", "u16"])
        return dict(kind=kind, width=w, dtype=dt, rois=_log_int(rng, 30, min(2000, 20_000_000 // (w * w))),
                    planes=rng.randint(60, 200))
    w = rng.randint(48, 100)
    return dict(kind=kind, width=w, dtype=rng.choice(["u8", "u16"]), beads=_log_int(rng, 4, 1_600_000 // (w * w)),
                planes=rng.randint(10, 40))


# ---------------------------------------------------------------------------------------------------
# settings and inputs
# ---------------------------------------------------------------------------------------------------
def _settings(case: dict) -> abi.QTrkSettings:
    w = case["width"]
    if case["kind"] in ("gauss", "ggrad"):
        return abi.settings(width=w, height=w, gauss2D_sigma=case["sigma"], gauss2D_iterations=8, qi_minradius=1,
                            zlut_minradius=1)
    if case["kind"] in ("zgrad", "buildlut"):
        return synth.settings_square(w, qi_roi_coverage=0.9, zlut_roi_coverage=0.9, zlut_radial_coverage=48.5 / 33.0,
                                     com_bgcorrection=0.0)
    s = synth.settings_roi60() if w == 60 else synth.settings_square(w)
    s.com_bgcorrection = case.get("bg", 0.0)
    return s


class _Geometry:
    """The step counts that QTrk derives from its settings, in plain Python."""

    def __init__(self, s: abi.QTrkSettings):
        f = lambda v: float(np.float32(v))
        half = s.width // 2
        self.w = s.width
        self.qi_min, self.qi_max = f(s.qi_minradius), f(half * f(s.qi_roi_coverage))
        self.z_min, self.z_max = f(s.zlut_minradius), f(half * f(s.zlut_roi_coverage))
        self.qi_nang = int(f(f(2 * f(PI) * self.qi_max) * f(s.qi_angular_coverage)) / 4)
        nr, p = int(f(f(self.qi_max - self.qi_min) * f(s.qi_radial_coverage))), 1
        while p < nr:
            p *= 2
        self.qi_nr = p if abs(p - nr) < abs(p // 2 - nr) else p // 2
        self.z_nang = int(f(f(2 * f(PI) * self.z_max) * f(s.zlut_angular_coverage)))
        self.z_nb = int(f(f(self.z_max - self.z_min) * f(s.zlut_radial_coverage)))
        self.iterations, self.bg = s.qi_iterations, f(s.com_bgcorrection)


def _levels(dtype: str) -> tuple[float, float, int]:
    """Background, amplitude and the largest pixel value; 8-bit and float cameras count 8 photons a level."""
    return (200.0, 2000.0, 4095) if dtype == "u16" else (20.0, 200.0, 255)


def _z_step(case: dict) -> float:
    return 0.5 * case["width"] / case.get("planes", 200)


def _bead_images(w: int, cx, cy, z, dtype: str, gen=None) -> torch.Tensor:
    """Bead images (n, w, w): Poisson-sampled in `dtype` with a generator, else noise-free in FP64."""
    bg, amp, top = _levels(dtype)
    px = torch.arange(w, device="cuda", dtype=F64 if gen is None else torch.float32)
    out = []
    for a in range(0, len(cx), 4096):
        x, y, k = (t[a:a + 4096].to(px.dtype)[:, None, None] for t in (cx, cy, z))
        r2 = (px[None, None, :] - x) ** 2 + (px[None, :, None] - y) ** 2
        lam = torch.exp(-r2 / (2 * (4 + 0.1 * k) ** 2)) * torch.cos(2 * math.pi * r2.sqrt() / (6 + 0.05 * k))
        lam = (bg + amp * lam).clamp_(min=0)
        if gen is None:
            out.append(lam)
        else:
            v = torch.poisson(lam, generator=gen) if dtype == "u16" else torch.poisson(8 * lam, generator=gen) / 8
            out.append((v if dtype == "f32" else v.round_().clamp_(max=top)).to(TORCH_DTYPE[dtype]))
    return torch.cat(out)


def _lut_rows(case: dict, g: _Geometry) -> torch.Tensor:
    """The bead family's Z-LUT (planes, bins), plane k at profile parameter k w / (2 planes), rows normalised."""
    k = torch.arange(case["planes"], device="cuda", dtype=F64)
    c = torch.full_like(k, g.w / 2)
    img = _bead_images(g.w, c, c, _z_step(case) * k, case["dtype"])
    return _normalised(_profiles(img, c, c, img.mean((1, 2)), g)[0])


def _radial_weights(g: _Geometry) -> np.ndarray:
    return np.sqrt(0.2 + 0.8 * np.sin(np.pi * (np.arange(g.z_nb) + 0.5) / g.z_nb)).astype(np.float32)


def _inputs(case: dict, seed: int) -> dict:
    """The case's inputs on the GPU, from the seed alone."""
    gen = torch.Generator("cuda").manual_seed(seed)
    uni = lambda n, lo, hi: lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda", dtype=F64)
    w, kind, dt = case["width"], case["kind"], case["dtype"]
    s = _settings(case)
    d = {"settings": s}
    if kind in ("gauss", "ggrad"):
        n = case["rois"]
        x, y = (w / 2 + uni(n, -w / 10, w / 10) for _ in range(2))
        ph = (w / 16) ** 2 * torch.exp(uni(n, math.log(1000), math.log(5000)))
        _, DX = _spot_axis(w, x, case["sigma"])
        _, DY = _spot_axis(w, y, case["sigma"])
        lam = 10.0 + ph[:, None, None] * DY[:, :, None] * DX[:, None, :]
        d["pixels"] = torch.poisson(lam.float(), generator=gen).to(TORCH_DTYPE[dt])
        if kind == "ggrad":
            p = torch.stack([x + uni(n, -.1, .1), y + uni(n, -.1, .1), ph * uni(n, .9, 1.1), uni(n, 9, 11),
                             uni(n, 0.95, 1.05) * case["sigma"]], 1)
            d["params"] = p.float().contiguous()
        return d
    g = _Geometry(s)
    planes = case.get("planes", 200)
    if kind in ("zgrad", "buildlut"):
        nb = case["beads"]
        x, y = (w / 2 + uni(nb, -2, 2) for _ in range(2))
        k = torch.arange(planes, device="cuda", dtype=F64).repeat_interleave(nb)
        d["pixels"] = _bead_images(w, x.repeat(planes), y.repeat(planes), _z_step(case) * k, dt, gen)
        if kind == "zgrad":
            lut = _lut_rows(case, g)[None] + 0.03 * torch.randn(nb, planes, g.z_nb, generator=gen, device="cuda",
                                                               dtype=F64)
            d["lut"] = _normalised(lut).float()
            n = nb * planes
            z = (k + uni(n, -0.4, 0.4)).clamp(0, planes - 1)
            xy = [t.repeat(planes) + uni(n, -0.05, 0.05) for t in (x, y)]
            d["xyz"] = torch.stack([*xy, z], 1).float().contiguous()
            d["beads"] = torch.arange(nb, device="cuda", dtype=torch.int32).repeat(planes)
        return d
    n = case["rois"]
    x, y = (w / 2 + uni(n, -0.03 * w, 0.03 * w) for _ in range(2))
    z = uni(n, 0.1 * planes, 0.95 * planes)
    d["pixels"] = _bead_images(w, x, y, _z_step(case) * z, dt, gen)
    if kind != "com":
        luts = n if kind == "frame" else case["luts"]
        lut = _lut_rows(case, g)[None].repeat(luts, 1, 1)
        if luts > 1:
            lut = lut + 0.03 * torch.randn(lut.shape, generator=gen, device="cuda", dtype=F64)
        d["lut"] = _normalised(lut).float()
    return d


# ---------------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    d = _inputs(case, seed)
    kind, w = case["kind"], case["width"]
    t = QTrkInstance(d["settings"])
    st = {"case": case, "tracker": t, "kind": kind, "pdt": PDT[case["dtype"]], "pitch": w * BPP[case["dtype"]],
          "stride": w * w * BPP[case["dtype"]]}
    if kind == "gauss":
        t.SetLocalizationMode(abi.LT_Gaussian2D | (abi.LT_B200_Gaussian5P if case["params"] == 5 else 0))
    elif kind == "com":
        t.SetLocalizationMode(abi.LT_OnlyCOM)
    elif kind != "ggrad":
        t.SetLocalizationMode(synth.MODE_QI_Z)
    if "lut" in d:
        t.SetRadialZLUT(d["lut"].cpu().numpy())
    if case.get("weighted"):
        t.SetRadialWeights(_radial_weights(_Geometry(d["settings"])))
    if kind in ("frame", "buildlut"):  # host data: pinned, as an acquisition program holds it
        host = d["pixels"]
        if kind == "frame":
            n = len(host)
            cols = math.ceil(math.sqrt(n))
            rows = (n + cols - 1) // cols
            grid = torch.zeros(rows * cols, w, w, dtype=host.dtype, device="cuda")
            grid[:n] = host
            host = grid.view(rows, cols, w, w).transpose(1, 2).reshape(rows * w, cols * w)
            ys, xs = np.divmod(np.arange(n), cols)
            st["positions"] = np.ascontiguousarray(np.stack([xs * w, ys * w], 1).astype(np.int32))
        else:
            host = host.view(case["planes"], case["beads"], w, w)
        st["pinned"] = torch.empty(host.shape, dtype=host.dtype).pin_memory()
        st["pinned"].copy_(host)
        st["host"] = st["pinned"].numpy().view(NUMPY_DTYPE[case["dtype"]])
        return st
    px = d["pixels"]
    n = st["n"] = len(px)
    st["pixels"] = px
    if kind in ("zgrad", "ggrad"):
        st |= {k: d[k] for k in ("xyz", "beads", "params") if k in d}
        st["cost"] = torch.empty(n, device="cuda")
        st["grad"] = torch.empty(n, 3 if kind == "zgrad" else 5, device="cuda")
        if kind == "zgrad":
            st["glut"] = torch.zeros_like(d["lut"])
    else:
        if case.get("luts", 1) > 1:  # job i: frame 0, timestamp 0, bead i
            st["jobs"] = torch.zeros(n, 6, dtype=torch.int32, device="cuda")
            st["jobs"][:, 2] = torch.arange(n, dtype=torch.int32, device="cuda")
        st["results"] = torch.empty(n, 13, dtype=torch.int32, device="cuda")
    return st


def run(st: dict):
    t, kind = st["tracker"], st["kind"]
    if kind == "frame":
        n = t.ScheduleFrame(st["host"], st["positions"])
        t.Flush()
        deadline = time.monotonic() + 60
        while t.GetResultCount() < n:
            if time.monotonic() > deadline:
                raise TimeoutError("results did not arrive: " + t.GetWarnings())
        r = t.GetResults(n)
        return {"bead": r["zlutIndex"], "pos": r["pos"], "guess": r["firstGuess"], "error": r["error"],
                "mean": r["imageMean"]}
    if kind == "buildlut":
        host = st["host"]
        t.SetRadialZLUTSize(host.shape[1], host.shape[0])
        t.BeginLUT(True)
        for k in range(host.shape[0]):
            t.BuildLUT(host[k], k)
        t.FinalizeLUT()
        return {"lut": t.GetRadialZLUT()}
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "zgrad":
        st["glut"].zero_()  # the call adds to it
        rc = t.lib.QTrkB200ZLUTCostGradient(t.handle, st["pixels"].data_ptr(), st["pitch"], st["stride"], st["pdt"],
                                            st["n"], st["xyz"].data_ptr(), st["beads"].data_ptr(),
                                            st["cost"].data_ptr(), st["grad"].data_ptr(), st["glut"].data_ptr(), stream)
    elif kind == "ggrad":
        rc = t.lib.QTrkB200GaussianNLLGradient(t.handle, st["pixels"].data_ptr(), st["pitch"], st["stride"], st["pdt"],
                                               st["n"], st["params"].data_ptr(), st["cost"].data_ptr(),
                                               st["grad"].data_ptr(), stream)
    else:
        res = st["results"]
        t.LocalizeDevice(st["pixels"].data_ptr(), st["pitch"], st["stride"], st["pdt"], st["n"], res.data_ptr(),
                         st["jobs"].data_ptr() if "jobs" in st else 0, stream)
        f = res.view(torch.float32)
        return {"job": res[:, :6], "pos": f[:, 6:9], "guess": f[:, 9:11], "error": res[:, 11], "mean": f[:, 12]}
    if rc != 0:
        raise RuntimeError(f"{kind} failed ({rc}): {t.GetWarnings()}")
    return {k: st[k] for k in ("cost", "grad", "glut") if k in st}


def work(case: dict) -> dict:
    kind, w, bpp = case["kind"], case["width"], BPP[case["dtype"]]
    n = case["rois"] if "rois" in case else case["beads"] * case["planes"]
    px = n * w * w
    if kind == "com":
        return {"bytes": px * bpp + n * 52, "flops": px * 7}
    if kind == "gauss":
        return {"bytes": px * bpp + n * 52, "flops": px * 8 * (30 if case["params"] == 4 else 50)}
    if kind == "ggrad":
        return {"bytes": px * bpp + n * (20 + 24), "flops": px * 25}
    g = _Geometry(_settings(case))
    sample = 12  # flops of one bilinear sample and its coordinates
    L = 2 * g.qi_nr
    com = 7 * w * w
    qi = g.iterations * (4 * g.qi_nr * g.qi_nang * sample + 10 * L * math.log2(L))
    prof = g.z_nb * g.z_nang * sample
    lut = g.z_nb * case["planes"]
    if kind == "zgrad":
        return {"bytes": px * bpp + n * (12 + 4 + 16) + 2 * case["beads"] * lut * 4,
                "flops": n * (g.z_nb * g.z_nang * (sample + 8) + 40 * g.z_nb)}
    if kind == "buildlut":
        return {"bytes": px * bpp + 2 * case["beads"] * lut * 4, "flops": n * (com + qi + prof)}
    luts = n if kind == "frame" else case["luts"]
    return {"bytes": px * bpp + n * 52 + (n * 24 if luts > 1 else 0) + luts * lut * 4,
            "flops": n * (com + qi + prof + 3 * lut)}


# ---------------------------------------------------------------------------------------------------
# the same results in FP64
# ---------------------------------------------------------------------------------------------------
def _normalised(p: torch.Tensor) -> torch.Tensor:
    p = p - p.mean(-1, keepdim=True)
    return p / p.square().mean(-1, keepdim=True).sqrt()


def _bilinear(img: torch.Tensor, x: torch.Tensor, y: torch.Tensor, slopes: bool = False):
    """Bilinear samples of img (n, w, w) at x, y (n, ...): value (0 outside), inside, and d/dx, d/dy."""
    n, w = img.shape[0], img.shape[2]
    inside = (x > -1) & (x < w - 1) & (y > -1) & (y < w - 1)
    ix, iy = x.clamp(0, w - 2).long(), y.clamp(0, w - 2).long()
    fx, fy = x - ix, y - iy
    at = (iy * w + ix).view(n, -1)
    flat = img.reshape(n, -1)
    v00, v10, v01, v11 = (flat.gather(1, at + o).view(x.shape) for o in (0, 1, w, w + 1))
    a, b = v00 + (v10 - v00) * fx, v01 + (v11 - v01) * fx
    zero = lambda v: torch.where(inside, v, torch.zeros_like(v))
    if not slopes:
        return zero(a + (b - a) * fy), inside
    return zero(a + (b - a) * fy), inside, zero((v10 - v00) * (1 - fy) + (v11 - v01) * fy), zero(b - a)


def _profiles(img, x, y, mean, g: _Geometry, slopes: bool = False) -> list[torch.Tensor]:
    """Radial profiles (n, bins) around (x, y), and their x and y derivatives."""
    ang = 2 * PI * torch.arange(g.z_nang, device=img.device, dtype=F64) / g.z_nang
    r = g.z_min + (g.z_max - g.z_min) / g.z_nb * torch.arange(g.z_nb, device=img.device, dtype=F64)
    out = []
    step = max(1, 6_000_000 // (g.z_nb * g.z_nang))
    for a in range(0, len(img), step):
        sl = slice(a, a + step)
        X = x[sl, None, None] + r[None, :, None] * torch.cos(ang)
        Y = y[sl, None, None] + r[None, :, None] * torch.sin(ang)
        v = _bilinear(img[sl].to(F64), X, Y, slopes)
        c = v[1].sum(-1)
        few = c <= 4
        p = torch.where(few, mean[sl, None], v[0].sum(-1) / c.clamp(min=1))
        out.append([p, *(torch.where(few, torch.zeros_like(p), d.sum(-1) / c.clamp(min=1)) for d in v[2:])])
    return [torch.cat(t) for t in zip(*out)]


def _peak(v: torch.Tensor, weights) -> torch.Tensor:
    """Vertex of the weighted parabola through the seven values around the maximum of each row."""
    n, length = v.shape
    top = v.argmax(1)
    start, end = (top - 3).clamp(min=0), (top + 4).clamp(max=length)
    j = torch.arange(7, device=v.device)
    wt = torch.tensor(np.float32(weights), device=v.device, dtype=F64) * (j < (end - start)[:, None])
    at = (start[:, None] + j).clamp(max=length - 1)
    x = (at - top[:, None]).to(F64)
    y = v.gather(1, at) - v.gather(1, top[:, None])
    S = lambda t: (wt * t).sum(1)
    Sw, Sx, Sx2, Sx3, Sx4 = (S(x ** k) for k in range(5))
    Sy, Sxy, Sx2y = S(y), S(x * y), S(x * x * y)
    d = Sx4 * (Sx2 * Sw - Sx * Sx) - Sx3 * (Sx3 * Sw - Sx * Sx2) + Sx2 * (Sx3 * Sx - Sx2 * Sx2)
    A = Sx2y * (Sx2 * Sw - Sx * Sx) - Sxy * (Sx3 * Sw - Sx * Sx2) + Sy * (Sx3 * Sx - Sx2 * Sx2)
    B = Sx4 * (Sxy * Sw - Sy * Sx) - Sx3 * (Sx2y * Sw - Sy * Sx2) + Sx2 * (Sx2y * Sx - Sxy * Sx2)
    return torch.where(A.abs() < 1e-9 * d.abs(), top.to(F64), top - B / (2 * A))


def _com(img: torch.Tensor, bg: float):
    """Centre of mass of |v - mean| above bg standard deviations, and the mean."""
    mean = img.mean((1, 2))
    d = (img - mean[:, None, None]).abs()
    if bg:
        std = (img.square().mean((1, 2)) - mean * mean).sqrt()
        d = (d - bg * std[:, None, None]).clamp(min=0)
    at = torch.arange(img.shape[1], device=img.device, dtype=F64)
    m = d.sum((1, 2))
    return (d.sum(1) * at).sum(1) / m, (d.sum(2) * at).sum(1) / m, mean


def _qi(img, x, y, mean, g: _Geometry, windowed: bool):
    """Quadrant interpolation from (x, y); `windowed`: radial bins weighted."""
    dev, nr = img.device, g.qi_nr
    ang = 0.5 * PI * (torch.arange(g.qi_nang, device=dev, dtype=F64) + 0.5) / g.qi_nang
    rstep = (g.qi_max - g.qi_min) / nr
    i = torch.arange(nr, device=dev, dtype=F64)
    r, u = g.qi_min + rstep * i, i / nr
    rw = torch.sqrt((1 - torch.exp(-((1 - u) ** 2) / 0.05)) * (1 - torch.exp(-(u * u) / 0.01)) * u * 2)
    dx, dy = r[:, None] * torch.cos(ang), r[:, None] * torch.sin(ang)
    L = 2 * nr
    k = torch.arange(L, device=dev, dtype=F64)
    turn = torch.polar(torch.ones_like(k), -2 * math.pi * k / L)
    off = lambda m: (m - nr) * (3.14159265359 / 4) * rstep
    for _ in range(g.iterations):
        q = []
        for sx, sy in ((1, 1), (-1, 1), (-1, -1), (1, -1)):
            v, inside = _bilinear(img, x[:, None, None] + sx * dx, y[:, None, None] + sy * dy)
            c = inside.sum(-1)
            p = torch.where(c >= 4, v.sum(-1) / c.clamp(min=1), mean[:, None])
            q.append(p * rw if windowed else p)
        px = torch.cat([(q[1] + q[2]).flip(1), q[0] + q[3]], 1)
        py = torch.cat([(q[2] + q[3]).flip(1), q[0] + q[1]], 1)
        ac = lambda p: torch.fft.ifft(turn * torch.fft.fft(p) ** 2).real.roll(-nr, 1)
        x, y = x + off(_peak(ac(px), QI_WEIGHTS)), y + off(_peak(ac(py), QI_WEIGHTS))
    return x, y


def _track64(px, lut, bead, wz, g: _Geometry) -> list[torch.Tensor]:
    out = []
    step = max(1, 6_000_000 // max(4 * g.qi_nr * g.qi_nang // 4, g.z_nb * g.z_nang, g.z_nb * lut.shape[1]))
    for a in range(0, len(px), step):
        img = px[a:a + step].to(F64)
        gx, gy, mean = _com(img, g.bg)
        x, y = _qi(img, gx, gy, mean, g, True)
        p = _normalised(_profiles(img, x, y, mean, g)[0])
        L = lut[bead[a:a + step]].to(F64)
        z = _peak(-((p[:, None, :] - L) * wz).square().sum(-1), ZLUT_WEIGHTS)
        out.append([torch.stack([x, y, z], 1), torch.stack([gx, gy], 1), mean])
    return [torch.cat(t) for t in zip(*out)]


def _spot_axis(w: int, p: torch.Tensor, sigma, erf=torch.erf):
    """The Gaussian's edge exponentials and pixel integrals along one axis, (n, w)."""
    c = torch.arange(w, device=p.device, dtype=F64)[None]
    sigma = sigma[:, None] if isinstance(sigma, torch.Tensor) else sigma
    e0, e1 = ((c - p[:, None] + s) / (math.sqrt(2) * sigma) for s in (.5, -.5))
    x0, x1 = torch.exp(-e0 * e0), torch.exp(-e1 * e1)
    lo, hi = c - p[:, None] - .5, c - p[:, None] + .5
    return (x1 - x0, lo * x1 - hi * x0), 0.5 * (erf(e0) - erf(e1))


def _erf_qtrk(x: torch.Tensor) -> torch.Tensor:
    """Abramowitz & Stegun 7.1.26, the erf of QTrk's 4-parameter fit."""
    t = 1 / (1 + 0.3275911 * x.abs())
    poly = ((((1.061405429 * t - 1.453152027) * t) + 1.421413741) * t - 0.284496736) * t + 0.254829592
    return torch.where(x < 0, -1.0, 1.0) * (1 - poly * t * torch.exp(-x * x))


def _outer(row: torch.Tensor, col: torch.Tensor) -> torch.Tensor:
    return row[:, :, None] * col[:, None, :]


def _gauss4(img, x, y, mean, sigma: float, iterations: int):
    w = img.shape[1]
    I0, bg = mean * 0.5 * w * w, mean * 0.5
    k2, k3 = (1 / (math.sqrt(2 * math.pi) * sigma ** p) for p in (1, 3))
    S = lambda t: t.sum((1, 2))
    for _ in range(iterations):
        (gX, hX), DX = _spot_axis(w, x, sigma, _erf_qtrk)
        (gY, hY), DY = _spot_axis(w, y, sigma, _erf_qtrk)
        i = I0[:, None, None]
        D = _outer(DY, DX)
        mu = bg[:, None, None] + i * D
        f, q = img / mu - 1, img / (mu * mu)
        jx, jy = i * k2 * _outer(DY, gX), i * k2 * _outer(gY, DX)
        x = x - S(jx * f) / S(i * k3 * _outer(DY, hX) * f - jx * jx * q)
        y = y - S(jy * f) / S(i * k3 * _outer(hY, DX) * f - jy * jy * q)
        I0, bg = I0 - S(D * f) / S(-D * D * q), bg - S(f) / S(-q)
    return torch.stack([x, y, torch.zeros_like(x)], 1)


def _spot_model(w: int, p: torch.Tensor):
    """mu and its derivatives by (x, y, I0, bg, sigma) for parameters p (n, 5)."""
    s = p[:, 4]
    k2 = (1 / (math.sqrt(2 * math.pi) * s))[:, None]
    (gX, hX), DX = _spot_axis(w, p[:, 0], s)
    (gY, hY), DY = _spot_axis(w, p[:, 1], s)
    I0 = p[:, 2, None, None]
    D, k3 = _outer(DY, DX), k2 / s[:, None]
    J = [I0 * _outer(DY, gX * k2), I0 * _outer(gY * k2, DX), D, torch.ones_like(D),
         I0 * (_outer(DY, hX * k3) + _outer(hY * k3, DX))]
    return p[:, 3, None, None] + I0 * D, torch.stack([j.flatten(1) for j in J], 1)


def _gauss5(img, x, y, mean, sigma: float, iterations: int):
    w = img.shape[1]
    p = torch.stack([x, y, mean * 0.5 * w * w, mean * 0.5, torch.full_like(x, sigma)], 1)
    v = img.flatten(1)
    for _ in range(iterations):
        mu, J = _spot_model(w, p)
        mu = mu.flatten(1)
        b = (J * (v / mu - 1)[:, None]).sum(2)
        A = torch.einsum("nip,njp->nij", J / mu[:, None], J)
        p = p + torch.linalg.solve(A, b)
        p = torch.stack([p[:, 0], p[:, 1], p[:, 2].clamp(min=1e-3), p[:, 3].clamp(min=1e-3),
                         p[:, 4].clamp(0.3, 0.5 * w)], 1)
    return torch.stack([p[:, 0], p[:, 1], p[:, 4]], 1)


def _zgrad64(d: dict, g: _Geometry, wz) -> dict:
    lut = d["lut"].to(F64)
    glut = torch.zeros_like(lut)
    planes = lut.shape[1]
    cost, grad = [], []
    for a in range(0, len(d["pixels"]), 2000):
        img = d["pixels"][a:a + 2000].to(F64)
        x, y, z = d["xyz"][a:a + 2000].to(F64).unbind(1)
        bead = d["beads"][a:a + 2000].long()
        p, dx, dy = _profiles(img, x, y, img.mean((1, 2)), g, True)
        rms = p.var(1, correction=0).sqrt()[:, None]
        p = _normalised(p)
        J = [(t - t.mean(1, keepdim=True) - p * (p * t).mean(1, keepdim=True)) / rms for t in (dx, dy)]
        iz = z.floor().long().clamp(0, planes - 2)
        fz = (z - iz)[:, None]
        l0, l1 = lut[bead, iz], lut[bead, iz + 1]
        e = p - (l0 + (l1 - l0) * fz)
        w2 = wz * wz
        cost.append((w2 * e * e).sum(1))
        grad.append(torch.stack([2 * (w2 * e * j).sum(1) for j in (*J, l0 - l1)], 1))
        glut.index_put_((bead, iz), -2 * w2 * e * (1 - fz), accumulate=True)
        glut.index_put_((bead, iz + 1), -2 * w2 * e * fz, accumulate=True)
    return {"cost": torch.cat(cost), "grad": torch.cat(grad), "glut": glut}


def exact(case: dict, seed: int):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("gauss", "ggrad"):
        out = []
        for a in range(0, case["rois"], 5000):
            img = d["pixels"][a:a + 5000].to(F64)
            if kind == "ggrad":
                mu, J = _spot_model(case["width"], d["params"][a:a + 5000].to(F64))
                mu, v = mu.flatten(1), img.flatten(1)
                out.append([(mu - v * mu.log()).sum(1), (J * (1 - v / mu)[:, None]).sum(2)])
            else:
                x, y, mean = _com(img, 0.0)
                fit = _gauss5 if case["params"] == 5 else _gauss4
                pos = fit(img, x, y, mean, case["sigma"], d["settings"].gauss2D_iterations)
                out.append([pos, torch.stack([x, y], 1), mean])
        out = [torch.cat(t) for t in zip(*out)]
        if kind == "ggrad":
            return {"cost": out[0], "grad": out[1]}
        return {"job": None, "pos": out[0], "guess": out[1], "error": None, "mean": out[2]}
    g = _Geometry(d["settings"])
    wz = torch.from_numpy(_radial_weights(g)).cuda().to(F64) if case.get("weighted") else torch.ones(
        g.z_nb, device="cuda", dtype=F64)
    if kind == "zgrad":
        return _zgrad64(d, g, wz)
    if kind == "buildlut":
        rows = []
        for a in range(0, len(d["pixels"]), 1000):
            img = d["pixels"][a:a + 1000].to(F64)
            x, y, mean = _com(img, 0.0)
            x, y = _qi(img, x, y, mean, g, False)
            rows.append(_normalised(_profiles(img, x, y, mean, g)[0]))
        return {"lut": torch.cat(rows).view(case["planes"], case["beads"], -1).transpose(0, 1).contiguous()}
    if kind == "com":
        out = []
        for a in range(0, case["rois"], 1000):
            x, y, mean = _com(d["pixels"][a:a + 1000].to(F64), g.bg)
            out.append([torch.stack([x, y, torch.zeros_like(x)], 1), torch.stack([x, y], 1), mean])
        pos, guess, mean = (torch.cat(t) for t in zip(*out))
    else:
        n = case["rois"]
        own = kind == "frame" or case["luts"] > 1
        bead = torch.arange(n, device="cuda") if own else torch.zeros(n, dtype=torch.long, device="cuda")
        pos, guess, mean = _track64(d["pixels"], d["lut"], bead, wz, g)
    return {"job" if kind != "frame" else "bead": None, "pos": pos, "guess": guess, "error": None, "mean": mean}
