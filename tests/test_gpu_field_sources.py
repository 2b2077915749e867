"""Which form of the FAST field runs by its sources (csrc/field_fft.cu, `concentrated`): a few charged
bins take the direct sum, whose error is relative to each cell's own terms, charge spread over the
box the convolution.  Charges times 2^90 are out of the convolution's range and always take the
direct sum, with the same roundings: the fields tell which form ran.

Tolerance: a term q R/|R|^3 of the direct sum has the error of |R|^2 (three roundings, to the
power 3/2), of the approximate root (2^-22.9, cubed) and some six roundings, 1.1e-6 in all, and
the split form of the far terms (E = c' S - P about the brick's centre) at most doubles it: 2.5e-6 of the
cell's sum of |q|/|R|^2."""
import numpy as np
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W

pytestmark = pytest.mark.gpu
SCALE = np.float32(2.0 ** 90)


def _config(shape, depth):
    case = W.mhd_plasma(shape=(32, 32, 32), depth=depth, field_mode=1)
    case["config"].update(n_x=shape[0], n_y=shape[1], n_z=shape[2], mhd_lod_depth=depth)
    return W.lbm_config(case)


def _sources(nd, kind, seed=3):
    """Charge [z][y][x] and velocity [3] of the bins (the first fifth is no source)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    q, v = np.zeros((nd, nd, nd)), rng.normal(0.0, 1e-3, (3, nd, nd, nd))
    if kind == "one":
        q[-1, -1, -1] = 1.0
    elif kind == "two":
        q[-1, -1, -1], q[-2, -1, -1] = 1.0, -1.0
    elif kind == "cluster":
        q[-2:, -2:, -2:] = rng.normal(0.0, 1.0, (2, 2, 2))
    elif kind == "line":
        q[:, nd // 2, 1] = 1.0
    elif kind == "current":  # charge spread, the current along x in one bin
        q[:], v[0] = rng.normal(0.0, 1.0, q.shape), 0.0
        v[0, -1, -1, -1] = 1e-3
    else:
        q[:] = rng.normal(0.0, 1.0, q.shape)
    return (q * 1e-2).astype(np.float32), v.astype(np.float32)


def _fields(shape, depth, q, v):
    nd = 1 << depth
    lbm = I.Lbm(_config(shape, depth))
    out = []
    for scale in (np.float32(1.0), SCALE):
        lod = np.zeros((sum(8 ** k for k in range(depth + 1)), 4), np.float32)
        lod[:nd ** 3, 0] = q.reshape(-1) * scale
        lod[:nd ** 3, 1:] = v.reshape(3, -1).T
        lbm.write("qu_lod", lod.reshape(-1))
        lbm.initialize()
        lbm.finish_queues(60000)
        out.append([lbm.read(name)[:3 * lbm.n].reshape(3, -1) / scale for name in ("e_dyn", "b_dyn")])
    lbm.close()
    return out


SHAPES = [((128, 128, 128), 4), ((16, 16, 16), 4), ((48, 32, 80), 4), ((40, 24, 56), 3), ((8, 8, 8), 3)]


@pytest.mark.parametrize("kind", ["one", "two", "cluster", "line"])
@pytest.mark.parametrize("shape,depth", SHAPES)
def test_few_charged_bins_keep_the_error_of_the_direct_sum(shape, depth, kind):
    nd = 1 << depth
    q, v = _sources(nd, kind)
    (e, b), direct = _fields(shape, depth, q, v)
    assert np.array_equal(e, direct[0]) and np.array_equal(b, direct[1])
    n, bs = int(np.prod(shape)), np.array([s // nd for s in shape])
    cells = np.arange(n) if n <= 6000 else np.sort(np.random.default_rng(1).choice(n, 6000, replace=False))
    xyz = np.stack([cells % shape[0], cells // shape[0] % shape[1], cells // (shape[0] * shape[1])])
    own = xyz // bs[:, None]
    first = sum(8 ** k for k in range(depth))
    want, size = np.zeros((3, cells.size)), np.zeros(cells.size)
    flat = q.reshape(-1).astype(np.float64)
    for d in np.flatnonzero(flat[first:]) + first:
        c = np.array([d % nd, d // nd % nd, d // nd ** 2])
        r = xyz - ((c + 0.5) * bs)[:, None]
        r2 = (r * r).sum(0)
        w = np.where((own == c[:, None]).all(0), 0.0, 1.0 / np.where(r2 > 0, r2, 1.0))
        want += flat[d] * r * w / np.sqrt(np.where(r2 > 0, r2, 1.0))
        size += abs(flat[d]) * w
    ke = _config(shape, depth).constants()["ke"]
    err = np.linalg.norm(e[:, cells].astype(np.float64) / ke - want, axis=0)
    assert np.all(err <= 2.5e-6 * size), float((err / np.where(size > 0, size, 1.0)).max())  # the own bin's cells: exactly 0


@pytest.mark.parametrize("kind,convolved", [("spread", True), ("current", False)])
@pytest.mark.parametrize("shape,depth", [((128, 128, 128), 4), ((48, 32, 48), 4), ((40, 24, 32), 3), ((64, 64, 64), 3)])
def test_spread_sources_take_the_convolution(shape, depth, kind, convolved):
    q, v = _sources(1 << depth, kind)
    (e, b), direct = _fields(shape, depth, q, v)
    assert np.array_equal(e, direct[0]) != convolved and np.array_equal(b, direct[1]) != convolved
    assert np.linalg.norm(e - direct[0]) <= 3e-6 * np.linalg.norm(e)
