"""The landmark initializer at the sizes where its layout changes: the widest of the narrow rows (82
expression components), the narrowest of the wide ones (83), a panel edge of its solve and the
largest it takes (112), against the oracle: success and Newton steps equal, states bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_expr", [9, 41, 82, 83, 112])
def test_landmark_init_sizes(tdi, synth, O, n_expr):
    tdi.require_gpu()
    F = 4
    m = synth.make_model(5000, 9800, 0, n_expr=n_expr, n_id=8, n_tex=8)
    fr = synth.make_frames(m, F, 0, image_wh=(256, 256), tz=0.6)
    fr.target = np.zeros((F, tdi.NPIX), np.float32)
    batch = tdi.Batch(tdi.Model(m), F)
    batch.set_frames(fr)
    batch.set_state(fr.state_init, np.tile(synth.LAMBDA_INIT, (F, 1)), np.full(F, synth.L_INTENSITY, np.float32))
    p0L = np.ascontiguousarray(m.mean[:, m.lis].astype(np.float32))
    ok, slack, it = batch.landmark_init(p0L)
    x, _, _ = batch.get_state()
    om, fs = O.Model(m), O.FrameSet(fr)
    for i in range(F):
        ox, oslack, ook, oit, _ = O.landmark_init(om, fs, i, p0L)
        assert bool(ok[i]) == bool(ook) and it[i] == oit
        np.testing.assert_array_equal(x[i].view(np.uint32), ox.view(np.uint32))


def test_landmark_init_refuses_what_it_refused(tdi, synth):
    tdi.require_gpu()
    m = synth.make_model(5000, 9800, 0, n_expr=113, n_id=8, n_tex=8)
    fr = synth.make_frames(m, 1, 0, image_wh=(256, 256), tz=0.6)
    fr.target = np.zeros((1, tdi.NPIX), np.float32)
    batch = tdi.Batch(tdi.Model(m), 1)
    batch.set_frames(fr)
    with pytest.raises(tdi.TdiError):
        batch.landmark_init(np.ascontiguousarray(m.mean[:, m.lis].astype(np.float32)))
