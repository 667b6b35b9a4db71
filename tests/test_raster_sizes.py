"""The batch raster where its working set changes: more candidate fragments than a frame's buffer
holds (two expression components give the smallest buffer: 26,214), bit sets too large for shared
memory (above 229,376 triangles), and neither. Layers of jittered grids over the crop, each at
its own depth; fragments bit for bit the oracle's (FP32 in the same operand order, so there is no
tolerance). Two rasters in a row show that nothing of the first is left in the second."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(synth, n_layers, nx, ny, step, seed):
    rng = np.random.default_rng(seed)
    gx, gy = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    xs, ys, zs, tl = [], [], [], []
    for k in range(n_layers):
        xs.append(20 + step * gx.ravel() + rng.uniform(-0.3, 0.3, nx * ny) * step)
        ys.append(20 + step * gy.ravel() + rng.uniform(-0.3, 0.3, nx * ny) * step)
        zs.append(500 + rng.normal(0, 5, nx * ny))
        i = (gx[:-1, :-1] * ny + gy[:-1, :-1]).ravel() + k * nx * ny
        tl.append(np.concatenate([np.stack([i, i + ny, i + 1]), np.stack([i + ny, i + ny + 1, i + 1])], 1))
    tl = np.concatenate(tl, 1)
    tl = tl[:, rng.permutation(tl.shape[1])]
    x, y, z = (np.concatenate(a).astype(np.float32) for a in (xs, ys, zs))
    V, K = len(x), 2
    b = np.ones(K, np.float32)
    m = synth.Model(mean=np.stack([x, y, z]), E=np.zeros((V, 3, K), np.float32), tex=np.full(V, 0.5, np.float32),
                    tl=tl.astype(np.int32), lis=np.arange(51, dtype=np.int32), eps_lb=-b, eps_ub=b, eps_lb_ft=-b,
                    eps_ub_ft=b)
    return m, x, y, z


@pytest.mark.parametrize("n_layers,nx,ny,step,over", [(2, 61, 57, 1.1, False), (12, 61, 57, 1.1, True),
                                                      (1, 345, 341, 0.25, False)])
def test_raster_working_sets(tdi, synth, O, n_layers, nx, ny, step, over):
    tdi.require_gpu()
    m, x, y, z = _layers(synth, n_layers, nx, ny, step, 5)
    om = O.Model(m)
    batch = tdi.Batch(tdi.Model(m), 2)
    shifted = (x + np.float32(3.25), y + np.float32(1.5), z)
    for args in ((x, y, z), shifted, (x, y, z)):
        ref = O.raster(om, *args, 0, 0)
        samples = _samples(m, *args) if over else None
        n, _ = batch.raster(1, *args, 0, 0)
        got = batch.read(1, tdi.READ_FRAGMENTS)
        assert n == ref["N"] and n > 1000
        if over:
            assert samples > 26214          # the candidates do not fit
        for k in ("pix", "tri", "owner"):
            np.testing.assert_array_equal(got[k], ref[k])
        for k in ("al", "be"):
            np.testing.assert_array_equal(got[k].view(np.uint32), ref[k].view(np.uint32))


def _samples(m, x, y, z):
    """Integer points inside the triangles (about the number of candidate fragments)."""
    b, c, a = m.tl
    n = 0
    x0, y0 = np.floor(np.minimum.reduce([x[b], x[c], x[a]])), np.floor(np.minimum.reduce([y[b], y[c], y[a]]))
    for i in range(4):
        for j in range(4):
            px, py = x0 + i, y0 + j
            d = (x[b] - x[a]) * (y[c] - y[a]) - (y[b] - y[a]) * (x[c] - x[a])
            al = ((px - x[a]) * (y[c] - y[a]) - (py - y[a]) * (x[c] - x[a])) / d
            be = ((x[b] - x[a]) * (py - y[a]) - (y[b] - y[a]) * (px - x[a])) / d
            n += int(((al > 0) & (be > 0) & (al + be < 1)).sum())
    return n
