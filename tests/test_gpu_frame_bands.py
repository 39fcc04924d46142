"""ScheduleFrame of a pinned frame that crosses PCIe in several bands: every ROI's result is the device entry's, in
the order the ROIs were listed, for scan-ordered frames (banded), shuffled ones (one band) and overlapping ROIs."""
import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [-1, 1, 2])
@pytest.mark.parametrize("layout", ["grid", "shuffled", "overlapping", "thin"])
def test_banded_frame_equals_device_entry(layout, threads):
    import torch

    w, cols, rows = 64, 40, 22                       # 2560 x 1408 u16: 7 MB
    rng = np.random.Generator(np.random.PCG64(11))
    few = np.minimum(rng.poisson(synth.render(w, w, 32 + rng.uniform(-2, 2, 20), 32 + rng.uniform(-2, 2, 20),
                                              rng.uniform(8, 28, 20), 200.0, 2000.0)), 4095).astype(np.uint16)
    frame = torch.empty((rows * w, cols * w), dtype=torch.int16).pin_memory().numpy().view(np.uint16)
    for k in range(rows * cols):
        frame[k // cols * w:(k // cols + 1) * w, k % cols * w:(k % cols + 1) * w] = few[k % 20]
    pos = np.array([(k % cols * w, k // cols * w) for k in range(rows * cols)], np.int32)
    if layout == "shuffled":
        pos = pos[rng.permutation(len(pos))]
    elif layout == "overlapping":                    # ROIs at any row, sorted by it: bands share rows
        pos = pos + np.stack([np.zeros(len(pos)), rng.integers(-20, 20, len(pos))], 1).astype(np.int32)
        pos[:, 1] = np.clip(pos[:, 1], 0, rows * w - w)
        pos = pos[np.argsort(pos[:, 1], kind="stable")]
    elif layout == "thin":
        pos = pos[::7]
    pos = np.ascontiguousarray(pos)
    rois = np.stack([frame[y:y + w, x:x + w] for x, y in pos])
    s = synth.settings_square(w, numThreads=threads)
    with QTrkInstance(s) as t:
        t.SetLocalizationMode(abi.LT_QI)
        d = torch.from_numpy(rois.view(np.int16)).cuda()
        out = torch.zeros(len(rois) * 52, dtype=torch.uint8, device="cuda")
        t.LocalizeDevice(d.data_ptr(), 2 * w, 2 * w * w, abi.QTrkU16, len(rois), out.data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want = np.frombuffer(out.cpu().numpy().tobytes(), dtype=abi.RESULT_DTYPE)
        for k in range(3):                           # frames back to back
            assert t.ScheduleFrame(frame, pos, frame_no=k, zlut_base=5) == len(pos)
        t.Flush()
        n = 3 * len(pos)
        r = t.WaitForResults(n)
    assert np.array_equal(r["frame"], np.repeat(np.arange(3), len(pos)))
    assert np.array_equal(r["zlutIndex"], np.tile(np.arange(len(pos)) + 5, 3))
    for f in ("pos", "firstGuess", "imageMean", "error"):
        assert np.array_equal(r[f], np.concatenate([want[f]] * 3)), f
