"""The fit where the kernels' shapes follow the number of frames in a round: 1 to 6 frame pairs per thread
of the vertex stage and a second tile (97), a frame's normal equations over one block or two (about 10
frames), the render's block sizes (148). Every frame must end exactly where it ends when fitted alone:
a frame's arithmetic does not depend on the batch, so there is no tolerance."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [2, 9, 11, 16, 17, 33, 49, 65, 81, 96, 97, 150]


@pytest.fixture(scope="module")
def alone(tdi, synth, small_case):
    tdi.require_gpu()
    m, fr, _ = small_case
    model = tdi.Model(m)
    return model, [_fit(tdi, synth, model, fr, [i]) for i in range(fr.n_frames)]


def _fit(tdi, synth, model, fr, idx):
    n = fr.n_frames
    sub = dataclasses.replace(fr, **{k.name: np.ascontiguousarray(v[idx]) for k in dataclasses.fields(fr)
                                     if isinstance(v := getattr(fr, k.name), np.ndarray) and v.shape[:1] == (n,)})
    F = len(idx)
    batch = tdi.Batch(model, F)
    lam = np.tile(synth.LAMBDA_INIT, (F, 1))
    x, lamf, rep = batch.fit_frames(sub, sub.state_init, lam, np.full(F, synth.L_INTENSITY, np.float32),
                                    tdi.default_config(max_iters_rigid=3, max_iters_lambda=3))
    return x, lamf, [(r.flags, r.iters_lambda, r.iters_rigid) for r in rep]


@pytest.mark.parametrize("F", COUNTS)
def test_frames_fit_as_alone(tdi, synth, small_case, alone, F):
    model, one = alone
    fr = small_case[1]
    idx = [i % fr.n_frames for i in range(F)]
    x, lam, rep = _fit(tdi, synth, model, fr, idx)
    for i, j in enumerate(idx):
        np.testing.assert_array_equal(x[i], one[j][0][0])
        np.testing.assert_array_equal(lam[i], one[j][1][0])
        assert rep[i] == one[j][2][0]
        assert rep[i][2] > 0
