"""The FP64 correlation of a render does not depend on how many frames run with it: the blocks of 1,024
threads (up to one frame per SM) and of 512 add the fragments' terms in the same order, so the
sums agree bit for bit (there is no tolerance)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scalars(tdi, synth, model, fr, F):
    n = fr.n_frames
    idx = [i % n for i in range(F)]
    sub = dataclasses.replace(fr, **{k.name: np.ascontiguousarray(v[idx]) for k in dataclasses.fields(fr)
                                     if isinstance(v := getattr(fr, k.name), np.ndarray) and v.shape[:1] == (n,)})
    batch = tdi.Batch(model, F)
    batch.set_frames(sub)
    batch.set_state(sub.state_init, np.tile(synth.LAMBDA_INIT, (F, 1)), np.full(F, synth.L_INTENSITY, np.float32))
    batch.evaluate(tdi.default_config())
    return [batch.read(i, tdi.READ_SCALARS) for i in range(F)]


@pytest.mark.parametrize("case_name", ["small_case", "rough_case"])
def test_correlation_is_the_same_in_every_batch(request, tdi, synth, case_name):
    tdi.require_gpu()
    m, fr, _ = request.getfixturevalue(case_name)
    model = tdi.Model(m)
    one = _scalars(tdi, synth, model, fr, fr.n_frames)
    for F in (148, 149, 160):
        got = _scalars(tdi, synth, model, fr, F)
        for i in range(F):
            for key in ("corr", "barrier", "objective"):
                assert got[i][key] == one[i % fr.n_frames][key], (F, i, key)
