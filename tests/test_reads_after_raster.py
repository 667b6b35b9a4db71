"""What an evaluation left for tdi_batch_read stays readable after further rasters of the batch: a render,
the differentiable loss and tdi_batch_raster at the same states leave the neighbours, the Jacobian and
the normal equations as they were (bit for bit)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case_name", ["small_case", "rough_case"])
def test_evaluation_outlives_a_raster(request, tdi, synth, case_name):
    import torch
    tdi.require_gpu()
    ag = importlib.import_module("3di_b200.autograd")
    m, fr, _ = request.getfixturevalue(case_name)
    F = fr.n_frames
    batch = tdi.Batch(tdi.Model(m), F)
    batch.set_frames(fr)
    lam = np.tile(synth.LAMBDA_INIT, (F, 1)).astype(np.float32)
    L = np.full(F, synth.L_INTENSITY, np.float32)
    batch.set_state(fr.state_init, lam, L)
    batch.evaluate(tdi.default_config())
    items = (tdi.READ_NEIGHBOURS, tdi.READ_GRADIENTS, tdi.READ_JACOBIAN)

    def read():
        return [[batch.read(i, w).copy() for w in items] + list(batch.read(i, tdi.READ_NORMAL_EQ).values())
                for i in range(F)]
    ref = read()
    assert ref[0][0].shape[1] > 1000
    geo = [batch.read(i, tdi.READ_GEOMETRY) for i in range(F)]
    fd = [batch.read(i, tdi.READ_FRAME_DATA) for i in range(F)]

    def raster():
        for i in range(F):
            batch.raster(i, geo[i][3], geo[i][4], geo[i][5], fd[i]["x0"], fd[i]["y0"])

    def loss():
        t = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (fr.state_init, lam, L)]
        ag.loss_gradients(batch, tdi.default_config(), *t, torch.ones(F, dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
    for again in (batch.render, raster, loss):
        again()
        for i, (a, b) in enumerate(zip(ref, read())):
            for k, (u, v) in enumerate(zip(a, b)):
                np.testing.assert_array_equal(u, v, err_msg=f"{again} frame {i} item {k}")
