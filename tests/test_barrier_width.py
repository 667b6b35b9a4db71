"""Normal equations with more unknowns than the 88 columns of the narrow layouts (tensor-core mode, 83
to 121 expression components): the landmark and bound terms must reach every column of H and g.
Against the oracle's evaluation, with the tensor-core mode's stated bound (1e-5, Frobenius for H and
max norm for g)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_expr", [82, 83, 100, 121])
def test_wide_systems_have_their_barrier_terms(tdi, synth, O, n_expr):
    tdi.require_gpu()
    F = 2
    m = synth.make_model(5000, 9800, 0, n_expr=n_expr, n_id=8, n_tex=8)
    fr = synth.make_frames(m, F, 0, image_wh=(256, 256), tz=0.6)
    batch = tdi.Batch(tdi.Model(m), F)
    L = np.full(F, synth.L_INTENSITY, np.float32)
    lam = np.tile(synth.LAMBDA_INIT, (F, 1))
    fr.target = np.zeros((F, tdi.NPIX), np.float32)
    batch.set_frames(fr)
    batch.set_state(fr.state_true, fr.lam_true, L)
    img, _ = batch.render()
    fr.target = synth.add_noise(img, 0.02, 0)
    batch.set_frames(fr)
    batch.set_state(fr.state_init, lam, L)
    batch.evaluate(tdi.default_config(normal_eq=tdi.NORMAL_EQ_TENSOR))
    om, fs = O.Model(m), O.FrameSet(fr)
    for i in range(F):
        ne = batch.read(i, tdi.READ_NORMAL_EQ)
        e = O.evaluate(om, fs, i, O.config(), fr.state_init[i], lam[i], float(L[i]))
        assert np.linalg.norm(ne["H"] - e["H"]) <= 1e-5 * np.linalg.norm(e["H"])
        assert np.abs(ne["g"] - e["g"]).max() <= 1e-5 * np.abs(e["g"]).max()
