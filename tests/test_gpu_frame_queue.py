"""ScheduleFrame of a pinned frame of several megabytes: how many batches it becomes, and that frames scheduled from
two threads stay whole. A frame is cut into bands only when nothing is in flight, so that its batches take free slots
at once; behind other batches it is one.
"""
import threading
import time

import numpy as np
import pytest

from qtrk_b200 import abi, synth
from qtrk_b200.tracker import QTrkInstance

pytestmark = pytest.mark.gpu
W, COLS, ROWS = 64, 40, 22                               # 2560 x 1408 u16: 7 MB


def make_frame(rows=ROWS):
    import torch

    rng = np.random.Generator(np.random.PCG64(11))
    few = np.minimum(rng.poisson(synth.render(W, W, 32 + rng.uniform(-2, 2, 20), 32 + rng.uniform(-2, 2, 20),
                                              rng.uniform(8, 28, 20), 200.0, 2000.0)), 4095).astype(np.uint16)
    frame = torch.empty((rows * W, COLS * W), dtype=torch.int16).pin_memory().numpy().view(np.uint16)
    for k in range(rows * COLS):
        frame[k // COLS * W:(k // COLS + 1) * W, k % COLS * W:(k % COLS + 1) * W] = few[k % 20]
    return frame, np.array([(k % COLS * W, k // COLS * W) for k in range(rows * COLS)], np.int32)


def fetch(t, n):
    """n results in the order they came."""
    t.Flush()
    end = time.monotonic() + 60
    while t.GetResultCount() < n and time.monotonic() < end:
        time.sleep(0.0005)
    return t.GetResults(n)


@pytest.mark.parametrize("slots,layout,pinned,want", [
    (4, "grid", True, 3), (3, "grid", True, 3), (2, "grid", True, 2), (1, "grid", True, 1), (4, "shuffled", True, 1),
    (4, "grid", False, 1), (4, "small", True, 1)])
def test_batches_per_frame(slots, layout, pinned, want):
    frame, pos = make_frame(ROWS if layout != "small" else 12)  # 12 rows: 3.9 MB
    if layout == "shuffled":
        pos = np.random.default_rng(1).permutation(pos)
    if not pinned:
        frame = frame.copy()
    with QTrkInstance(synth.settings_square(W, numThreads=slots)) as t:
        t.SetLocalizationMode(abi.LT_QI)
        for _ in range(3):
            before = t.KernelLaunchCount()
            assert t.ScheduleFrame(frame, pos) == len(pos)
            assert t.KernelLaunchCount() - before == want
            r = fetch(t, len(pos))
            assert np.array_equal(r["zlutIndex"], np.arange(len(pos)))


def test_one_batch_behind_others():
    frame, pos = make_frame()
    s = synth.settings_square(W, numThreads=4, qi_iterations=30)
    stack = np.ascontiguousarray(np.repeat(frame[None, :W, :W], 4000, 0))
    with QTrkInstance(s) as t:
        t.SetLocalizationMode(abi.LT_QI)
        t.ScheduleStack(stack)
        t.Flush()                                        # several ms on the GPU
        before = t.KernelLaunchCount()
        assert t.ScheduleFrame(frame, pos) == len(pos)
        assert t.KernelLaunchCount() - before == 1
        assert len(fetch(t, len(stack) + len(pos))) == len(stack) + len(pos)


@pytest.mark.parametrize("slots", [2, 3, 4])
def test_frames_of_two_threads_stay_whole(slots):
    frame, pos = make_frame()
    per = 25
    with QTrkInstance(synth.settings_square(W, numThreads=slots)) as t:
        t.SetLocalizationMode(abi.LT_QI)
        bad = []

        def feed(first):
            for k in range(per):
                if t.ScheduleFrame(frame, pos, frame_no=first + k) != len(pos):
                    bad.append(first + k)

        threads = [threading.Thread(target=feed, args=(1000 * i,)) for i in range(2)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        r = fetch(t, 2 * per * len(pos))
    assert not bad and len(r) == 2 * per * len(pos)
    frames = r["frame"].reshape(2 * per, len(pos))
    assert (frames == frames[:, :1]).all()               # each frame's results are one run
    assert np.array_equal(r["zlutIndex"].reshape(2 * per, -1), np.tile(np.arange(len(pos)), (2 * per, 1)))
    assert np.array_equal(np.sort(frames[:, 0]), np.concatenate([np.arange(per), 1000 + np.arange(per)]))
