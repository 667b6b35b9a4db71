"""Renders and the differentiable loss of models with wide expression bases, where the vertex stage's
tile holds fewer frames (96 up to 168 components, 64 up to 192, 32 up to 224, 16 up to 240), and the
first width that no tile holds. Images bit for bit the oracle's (FP32 in the same operand order, so
there is no tolerance); the loss against the FP64 forward and its gradient against central differences,
with the bounds of the adjoint's own tests (1e-10, and 1e-6 for the directional derivative)."""
import importlib

import numpy as np
import pytest

from test_adjoint import _loss_np

pytestmark = pytest.mark.gpu


def _case(synth, n_expr, F):
    m = synth.make_model(5000, 9800, 0, n_expr=n_expr, n_id=8, n_tex=8)
    fr = synth.make_frames(m, F, 0, image_wh=(256, 256), tz=0.6)
    fr.target = synth.add_noise(np.zeros((F, 65536), np.float32), 0.1, 0)
    return m, fr


@pytest.mark.parametrize("n_expr,F", [(168, 40), (169, 40), (192, 40), (193, 33), (224, 2), (225, 17), (240, 2)])
def test_render_and_loss_of_wide_bases(tdi, synth, O, n_expr, F):
    import torch
    tdi.require_gpu()
    ag = importlib.import_module("3di_b200.autograd")
    m, fr = _case(synth, n_expr, F)
    om, cfg = O.Model(m), tdi.default_config()
    batch = tdi.Batch(tdi.Model(m), F)
    batch.set_frames(fr)
    batch.set_state(fr.state_true, fr.lam_true, np.full(F, synth.L_INTENSITY, np.float32))
    img, _ = batch.render()
    for i in {0, F // 2, F - 1}:
        ref, n, _ = O.render_target(om, fr, i, O.config(), fr.state_true[i], fr.lam_true[i], synth.L_INTENSITY)
        assert n > 1000
        np.testing.assert_array_equal(img[i], ref)
    dev = torch.device("cuda", 0)
    x = torch.from_numpy(np.ascontiguousarray(fr.state_init, np.float32)).to(dev)
    lam = torch.from_numpy(np.tile(synth.LAMBDA_INIT, (F, 1)).astype(np.float32)).to(dev)
    L = torch.full((F,), float(synth.L_INTENSITY), dtype=torch.float32, device=dev)
    loss = ag.render_loss(batch, x, lam, L, cfg)
    gx, glam, gL = ag.loss_gradients(batch, cfg, x, lam, L, torch.ones_like(loss))
    i, taps = F - 1, synth.KERNEL_SIGMA_TAPS[0.75]
    frags, fd = batch.read(i, tdi.READ_FRAGMENTS), batch.read(i, tdi.READ_FRAME_DATA)
    z = np.concatenate([x[i].cpu().numpy(), lam[i].cpu().numpy(), [L[i].item()]]).astype(np.float64)
    ref = _loss_np(m, fd, fr.target[i], frags, z, taps)
    assert abs(ref - loss[i].item()) <= 1e-10 * abs(ref)
    g = np.concatenate([gx[i].cpu().numpy(), glam[i].cpu().numpy(), [gL[i].item()]])
    d = np.random.default_rng(n_expr).normal(size=g.shape)
    d /= np.linalg.norm(d)

    def central(h):
        return (_loss_np(m, fd, fr.target[i], frags, z + h * d, taps)
                - _loss_np(m, fd, fr.target[i], frags, z - h * d, taps)) / (2 * h)
    fdv = (4.0 * central(5e-6) - central(1e-5)) / 3.0
    assert abs(float(g @ d) - fdv) <= 1e-6 * max(abs(fdv), 1e-3 * np.linalg.norm(g))


def test_a_basis_that_no_tile_holds_is_refused(tdi, synth):
    tdi.require_gpu()
    m, fr = _case(synth, 244, 2)
    batch = tdi.Batch(tdi.Model(m), 2)
    batch.set_frames(fr)
    batch.set_state(fr.state_true, fr.lam_true, np.full(2, synth.L_INTENSITY, np.float32))
    with pytest.raises(tdi.TdiError):
        batch.render()
