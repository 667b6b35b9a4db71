"""The shape solve at the sizes where its panels, register blocks and the carried right-hand side
change: unknowns on and beside multiples of 16, the largest of the small layout (95), the
smallest and largest of the large one (96, 127). Bit for bit the numpy restatement of the oracle's
solve (every operation is one rounding in a fixed order, so there is no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_expr", [9, 10, 11, 25, 26, 73, 74, 75, 89, 90, 121])
def test_shape_solve_sizes(tdi, synth, O, n_expr):
    tdi.require_gpu()
    F = 3
    m = synth.make_model(5000, 9800, 0, n_expr=n_expr, n_id=8, n_tex=8)
    fr = synth.make_frames(m, F, 0, image_wh=(256, 256), tz=0.6)
    model = tdi.Model(m)
    batch = tdi.Batch(model, F)
    L = np.full(F, synth.L_INTENSITY, np.float32)
    fr.target = np.zeros((F, tdi.NPIX), np.float32)
    batch.set_frames(fr)
    batch.set_state(fr.state_true, fr.lam_true, L)
    img, _ = batch.render()
    fr.target = synth.add_noise(img, 0.02, 0)
    batch.set_frames(fr)
    batch.set_state(fr.state_init, np.tile(synth.LAMBDA_INIT, (F, 1)), L)
    for damping in (0.0, 0.5):
        batch.evaluate(tdi.default_config(normal_eq=tdi.NORMAL_EQ_EXACT if n_expr <= 81 else tdi.NORMAL_EQ_TENSOR,
                                          damping=damping))
        for i in range(F):
            ne = batch.read(i, tdi.READ_NORMAL_EQ)
            d = O.solve_shape(ne["H"], ne["g"], damping)
            assert d is not None and np.isfinite(ne["d"]).all()
            np.testing.assert_array_equal(ne["d"], d)
