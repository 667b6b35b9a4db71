"""The depth pass's early decision on the device: triangles of every kind test_raster_cull.py generates
(slivers, corners on and beside sample points, edges beside a sample column, thin and box-filling ones) go
through the batch raster and the allocation-free one; their fragments equal the oracle's, which decides
nothing early (FP32 in the same operand order, so there is no tolerance). The rule's restated constants
are the source's."""
import os
import re

import numpy as np
import pytest

import test_raster_cull as RC
from test_zz_no_alloc import _noalloc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_restated_constants_are_the_sources():
    src = open(os.path.join(ROOT, "3di_b200", "csrc", "tdi_kernels.cu")).read()
    gap = re.search(r"RC_GAP = 1\.0f / ([0-9.]+)f;", src).group(1)
    shape = re.search(r"RC_SHAPE = ([0-9.e+-]+)f;", src).group(1)
    assert RC.GAP == np.float32(1.0) / np.float32(gap) and RC.SHAPE == np.float32(shape)


def _triangles(n, seed):
    """Corners [3][2][n] in a 256 x 256 crop, six kinds in turn."""
    rng = np.random.default_rng(seed)
    kind = np.arange(n) % 6
    size = 10.0 ** rng.uniform(-3.5, 0.3, n)
    p = rng.uniform(3, 252, (2, n))
    c = np.stack([p + rng.uniform(-0.5, 0.5, (2, n)) * size for _ in range(3)])
    t = rng.uniform(-0.5, 1.5, n)
    sliver = c[0] + t * (c[1] - c[0]) + rng.normal(0, 1, (2, n)) * size * 10.0 ** rng.uniform(-7, -1, n)
    c[2] = np.where(kind == 1, sliver, c[2])
    snap = (np.rint(c[0]) - c[0]) + rng.normal(0, 1, (2, n)) * 10.0 ** rng.uniform(-7, -1, n)
    c = np.where(kind == 2, c + snap, c)
    c[:, 0] += np.where(kind == 3, np.rint(c[0, 0]) - np.minimum(c[0, 0], c[1, 0]) + rng.normal(0, 0.03, n), 0)
    c[:, 1] = np.where(kind == 4, c[0, 1] + (c[:, 1] - c[0, 1]) * 10.0 ** rng.uniform(-4, 0, n), c[:, 1])
    return np.where(kind == 5, np.stack([np.floor(p) + rng.uniform(0, 2, (2, n)) for _ in range(3)]), c).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("seed,offset", [(1, 0), (2, 4096), (3, 60000)])
def test_rasters_of_unusual_triangles(tdi, synth, O, seed, offset):
    import torch
    tdi.require_gpu()
    T = 60_000
    c = _triangles(T, seed) + np.float32(offset)
    rng = np.random.default_rng(seed + 10)
    x, y = c[:, 0].ravel(), c[:, 1].ravel()                 # corner r of triangle t is vertex r T + t
    z = np.tile(rng.uniform(300, 900, T).astype(np.float32), 3)
    V, b = 3 * T, np.ones(2, np.float32)
    m = synth.Model(mean=np.stack([x, y, z]), E=np.zeros((V, 3, 2), np.float32), tex=np.full(V, 0.5, np.float32),
                    tl=np.arange(V, dtype=np.int32).reshape(3, T), lis=np.arange(51, dtype=np.int32), eps_lb=-b, eps_ub=b,
                    eps_lb_ft=-b, eps_ub_ft=b)
    a = [v.reshape(3, T) for v in (x, y)]
    with np.errstate(all="ignore"):
        cut = RC.culled(a[0][0], a[1][0], a[0][1], a[1][1], a[0][2], a[1][2])
    assert cut.sum() > T // 20                              # the rule decides many of them
    ref = O.raster(O.Model(m), x, y, z, offset, offset)
    assert ref["N"] > 1000
    batch = tdi.Batch(tdi.Model(m), 1)
    n, _ = batch.raster(0, x, y, z, offset, offset)
    got = [batch.read(0, tdi.READ_FRAGMENTS)]
    assert n == ref["N"]
    dev = torch.device("cuda", 0)
    d = [torch.from_numpy(v).to(dev) for v in (x, y, z)]
    tl = torch.from_numpy(m.tl).to(dev)
    out = torch.zeros(4 * 65536, dtype=torch.int32, device=dev)
    count, flags = torch.zeros(2, 1, dtype=torch.int32, device=dev)
    assert _noalloc(tdi.load_library(), d, tl, V, T, offset, offset, out, 65536, count, flags) == 0
    torch.cuda.synchronize()
    assert int(count.item()) == ref["N"]
    r = out[:4 * ref["N"]].cpu().numpy().reshape(-1, 4)
    po = r[:, 0].view(np.uint32)
    got.append(dict(pix=(po & 0xFFFF).astype(np.uint16), owner=(po >> 31).astype(np.uint8), tri=r[:, 1],
                    al=r[:, 2].copy().view(np.float32), be=r[:, 3].copy().view(np.float32)))
    for g in got:
        for k in ("pix", "tri", "owner"):
            np.testing.assert_array_equal(g[k], ref[k])
        for k in ("al", "be"):
            np.testing.assert_array_equal(g[k].view(np.uint32), np.ascontiguousarray(ref[k]).view(np.uint32))
