"""The differentiable loss where its FP64 vertex stage changes form with the number of frames (1, 4 or 8 per
thread) and at ragged ends of their tiles: a frame's loss is bit for bit the one it has alone (every
output is the same chain of operations), its gradients agree to the order of their FP64 atomic sums
(relative to their largest entry, 1e-10)."""
import dataclasses
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loss(tdi, synth, model, fr, F):
    import torch
    ag = importlib.import_module("3di_b200.autograd")
    n = fr.n_frames
    idx = [i % n for i in range(F)]
    sub = dataclasses.replace(fr, **{k.name: np.ascontiguousarray(v[idx]) for k in dataclasses.fields(fr)
                                     if isinstance(v := getattr(fr, k.name), np.ndarray) and v.shape[:1] == (n,)})
    batch = tdi.Batch(model, F)
    batch.set_frames(sub)
    dev = torch.device("cuda", 0)
    x = torch.from_numpy(np.ascontiguousarray(sub.state_init, np.float32)).to(dev)
    lam = torch.from_numpy(np.tile(synth.LAMBDA_INIT, (F, 1)).astype(np.float32)).to(dev)
    L = torch.full((F,), float(synth.L_INTENSITY), dtype=torch.float32, device=dev)
    loss = ag.render_loss(batch, x, lam, L)
    g = ag.loss_gradients(batch, tdi.default_config(), x, lam, L, torch.ones_like(loss))
    return loss.cpu().numpy(), [t.cpu().numpy().reshape(F, -1) for t in g]


def test_loss_does_not_depend_on_the_batch(tdi, synth, small_case):
    tdi.require_gpu()
    m, fr, _ = small_case
    model = tdi.Model(m)
    loss1, g1 = _loss(tdi, synth, model, fr, fr.n_frames)
    for F in (8, 9, 32, 33, 37, 64, 65):
        loss, g = _loss(tdi, synth, model, fr, F)
        for i in range(F):
            j = i % fr.n_frames
            assert loss[i] == loss1[j], (F, i)
            for a, b in zip(g, g1):
                assert np.abs(a[i] - b[j]).max() <= 1e-10 * np.abs(b[j]).max(), (F, i)
