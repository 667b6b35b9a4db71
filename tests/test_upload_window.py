"""Crops of frames of which only the sampled part is sent to the device, bit for bit the oracle's
(no tolerance)."""
import numpy as np
import pytest

import preprocess as P


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("pad", [0, 5])
def test_device_crops_of_partly_sent_frames(tdi, synth, pad):
    """Only the part of a frame that its crop reads is sent to the device: crops of 1080p frames whose
    windows are narrow, wide, at every edge of the frame, past it, and outside it, with and without
    a row pitch, bit for bit the oracle's."""
    tdi.require_gpu()
    rng = np.random.default_rng(21)
    W, H = 1920, 1080
    cases = [(960, 540, 150), (960, 540, 590), (200, 150, 130), (1800, 1000, 130), (1800, 120, 300), (100, 1000, 594),
             (1919, 1079, 121), (3000, 540, 140), (700, 2400, 200), (960, 540, 40)]
    F = len(cases)
    img = rng.integers(0, 256, (F, H, W, 3), dtype=np.uint8)
    face = np.array([c[2] for c in cases], np.float32)
    t = rng.uniform(-0.5, 0.5, (2, F, 51))
    xp = (np.array([c[0] for c in cases])[:, None] + t[0] * face[:, None]).astype(np.float32)
    yp = (np.array([c[1] for c in cases])[:, None] + t[1] * face[:, None]).astype(np.float32)
    cam = np.tile(np.array([800, 800, W / 2, H / 2], np.float32), (F, 1))
    batch = tdi.Batch(tdi.Model(synth.make_model(5000, 9800, 0, n_id=8, n_tex=8)), F)
    rows = np.zeros((F, H, 3 * W + pad), np.uint8)
    rows[:, :, :3 * W] = img.reshape(F, H, 3 * W)
    if pad:       # the pitched form takes its width from the pitch: whole pixels
        rows = np.concatenate([rows[:, :, :3 * W], np.zeros((F, H, 3 * pad), np.uint8)], 2)
        img = rows.reshape(F, H, W + pad, 3)
    batch.set_video_frames(rows if pad else img, xp, yp, np.zeros((F, 4, 51), np.float32), face, cam, 78.0)
    for f in range(F):
        o_crop = P.video_frame(img[f], xp[f], yp[f], face[f], cam[f], np.float32(78.0))[0]
        assert np.array_equal(_bits(batch.read(f, tdi.READ_CROP)), _bits(o_crop)), f
