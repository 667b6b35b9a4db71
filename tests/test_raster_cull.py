"""The depth pass's early decision that a triangle has no sample point inside (no_sample_inside in
tdi_kernels.cu) against the exact per-sample test of every sample of its box, in IEEE float32
arithmetic (numpy rounds to nearest, as the device does): triangles of all sizes up to the two
pixels the rule takes, slivers, corners on and next to sample points, and large coordinates."""
import numpy as np
import pytest

F32 = np.float32
GAP, SHAPE = F32(1.0 / 4096.0), F32(2.025e-9)


def culled(bx, by, cx, cy, ax, ay):
    """The device rule, restated."""
    xmax, xmin = np.fmax(np.fmax(bx, cx), ax), np.fmin(np.fmin(bx, cx), ax)
    ymax, ymin = np.fmax(np.fmax(by, cy), ay), np.fmin(np.fmin(by, cy), ay)
    xlo, ylo = np.floor(xmin), np.floor(ymin)
    dom = (np.fmin(xmin, ymin) >= 0) & (np.fmax(xmax, ymax) <= 65535) & (np.fmax(xmax - xmin, ymax - ymin) <= 2)
    gx = np.where(xmax <= xlo + F32(1), xmin - xlo, F32(0))
    gy = np.where(ymax <= ylo + F32(1), ymin - ylo, F32(0))
    g = np.fmax(gx, gy)
    v0x, v1x, v0y, v1y = bx - ax, cx - ax, by - ay, cy - ay
    d00, d01, d11 = v0x * v0x + v0y * v0y, v0x * v1x + v0y * v1y, v1x * v1x + v1y * v1y
    q = d00 * d11
    den = q - d01 * d01
    shape = (den * den) * (den * np.minimum(d00, d11)) * (g * g) > SHAPE * ((q * q) * q)
    return dom & (g > GAP) & shape


def accepted(bx, by, cx, cy, ax, ay):
    """Whether any sample of the box passes the reference's test (funcs.cu:900-1000)."""
    xlo, ylo = np.floor(np.minimum(np.minimum(bx, cx), ax)), np.floor(np.minimum(np.minimum(by, cy), ay))
    xhi, yhi = np.ceil(np.maximum(np.maximum(bx, cx), ax)), np.ceil(np.maximum(np.maximum(by, cy), ay))
    v0x, v1x, v0y, v1y = bx - ax, cx - ax, by - ay, cy - ay
    d00, d01, d11 = v0x * v0x + v0y * v0y, v0x * v1x + v0y * v1y, v1x * v1x + v1y * v1y
    den = d00 * d11 - d01 * d01
    hit = np.zeros(bx.shape, bool)
    for i in range(4):
        for j in range(4):
            x, y = xlo + F32(i), ylo + F32(j)
            d20, d21 = v0x * (x - ax) + v0y * (y - ay), v1x * (x - ax) + v1y * (y - ay)
            al, be = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
            hit |= (x < xhi) & (y < yhi) & (al > 0) & (be > 0) & (al + be <= 1)
    return hit


@pytest.mark.parametrize("offset", [0.0, 100.0, 900.0, 4000.0, 60000.0])
def test_culled_triangles_have_no_sample(offset):
    rng = np.random.default_rng(int(offset) + 3)
    n, taken = 200_000, 0
    for kind in range(6):
        size = 10.0 ** rng.uniform(-3.5, 0.3, n)
        p = rng.uniform(0, 2, (2, n)) + 1
        c = np.stack([p + rng.uniform(-0.5, 0.5, (2, n)) * size for _ in range(3)])
        if kind == 1:                                       # slivers: the third corner near the line of two
            t = rng.uniform(-0.5, 1.5, n)
            c[2] = c[0] + t * (c[1] - c[0]) + rng.normal(0, 1, (2, n)) * size * 10.0 ** rng.uniform(-7, -1, n)
        elif kind == 2:                                     # corners on or beside integer points
            r = np.rint(c[0])
            c += (r - c[0]) + rng.normal(0, 1, (2, n)) * 10.0 ** rng.uniform(-7, -1, n)
        elif kind == 3:                                     # an edge beside an integer column
            c[:, 0] += np.rint(c[0, 0]) - np.minimum(c[0, 0], c[1, 0]) + rng.normal(0, 0.03, n)
        elif kind == 4:                                     # thin in one direction
            c[:, 1] = c[0, 1] + (c[:, 1] - c[0, 1]) * 10.0 ** rng.uniform(-4, 0, n)
        elif kind == 5:                                     # box-filling triangles
            c = np.stack([np.floor(p) + rng.uniform(0, 2, (2, n)) for _ in range(3)])
        c = (c + offset).astype(F32)
        args = [c[0, 0], c[0, 1], c[1, 0], c[1, 1], c[2, 0], c[2, 1]]
        with np.errstate(all="ignore"):
            cut = culled(*args)
            assert not np.any(cut & accepted(*args)), (kind, offset)
        taken += int(cut.sum())
    assert taken > 100_000                                  # the rule decides many of them


def test_unusual_corners_are_not_culled():
    nan, inf = F32(np.nan), F32(np.inf)
    one = [F32(10.3), F32(10.3), F32(10.5), F32(10.3), F32(10.4), F32(10.5)]
    with np.errstate(all="ignore"):
        assert culled(*[np.array([v]) for v in one])[0]
        for q in range(6):
            for bad in (nan, inf, -inf, F32(-3.0), F32(1e6)):
                v = list(one)
                v[q] = bad
                assert not culled(*[np.array([w], F32) for w in v])[0], (q, bad)
        assert not culled(*[np.array([F32(10.3)])] * 6)[0]  # a point: no area
