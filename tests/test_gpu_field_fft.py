"""The FAST field as a convolution over the LOD bins (csrc/field_fft.cu) against the same
sums in 64 bits: bins written by the test, the field that ``initialize`` leaves.

Tolerance of the convolution: a 32-bit transform of 2 nd points along three axes adds a
relative rounding of at most about 3 log2(2 nd) roundings of 2^-24 in the norm, forward and
back, and the products and the scaling a few more: 2 * 15 + 8 = 38 roundings at nd = 16,
38 * 2^-24 = 2.3e-6.  The direct sum that stands by (approximate reciprocal square roots to
a power of three, 4096 terms) is held to 2e-5."""
import numpy as np
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu

CELLS = 4000  # cells compared (all of a smaller box)


def _config(shape, depth):
    case = W.mhd_plasma(shape=(32, 32, 32), depth=depth, field_mode=1)
    case["config"].update(n_x=shape[0], n_y=shape[1], n_z=shape[2], mhd_lod_depth=depth)
    return W.lbm_config(case)


def _bins(depth, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    lod = np.zeros((sum(8 ** k for k in range(depth + 1)), 4), np.float32)
    nb = 8 ** depth
    lod[:nb, 0] = rng.normal(0.0, 1e-2, nb)
    lod[:nb, 1:] = rng.normal(0.0, 1e-3, (nb, 3))
    return lod


def _field(shape, depth, lod):
    cfg = _config(shape, depth)
    lbm = I.Lbm(cfg)
    lbm.write("qu_lod", lod.reshape(-1))
    lbm.initialize()
    lbm.finish_queues(60000)
    n = lbm.n
    e, b = (lbm.read(name)[:3 * n].astype(np.float64).reshape(3, n) for name in ("e_dyn", "b_dyn"))
    k = cfg.constants()
    lbm.close()
    return e, b, k


def _exact(shape, depth, lod, cells, k):
    nd = 1 << depth
    bs = np.array([s // nd for s in shape], np.float64)
    first, nb = sum(8 ** i for i in range(depth)), nd ** 3
    d = np.arange(first, nb)
    c = np.stack([d % nd, d // nd % nd, d // nd ** 2])
    pos = (c + 0.5) * bs[:, None]
    q = lod[first:nb, 0].astype(np.float64)
    j = (lod[first:nb, 0:1] * lod[first:nb, 1:]).astype(np.float64).T  # q v is rounded to 32 bits first
    e, b = np.zeros((3, cells.size)), np.zeros((3, cells.size))
    xyz = np.stack([cells % shape[0], cells // shape[0] % shape[1], cells // (shape[0] * shape[1])])
    own = xyz // bs[:, None].astype(np.int64)
    with np.errstate(all="ignore"):
        for i in range(cells.size):
            r = xyz[:, i:i + 1] - pos
            w = ((r * r).sum(0)) ** -1.5
            w[(c == own[:, i:i + 1]).all(0)] = 0.0  # the own bin counts with weight 0
            e[:, i] = (q * r * w).sum(1)
            b[:, i] = (np.cross(j.T, r.T).T * w).sum(1)
    return k["ke"] * e, k["kmu"] * b


def _cells(shape, seed=1):
    n = shape[0] * shape[1] * shape[2]
    return np.arange(n) if n <= CELLS else np.sort(np.random.default_rng(seed).choice(n, CELLS, replace=False))


@pytest.mark.parametrize("shape,depth", [((8, 8, 8), 3), ((16, 16, 16), 4), ((24, 40, 56), 3), ((16, 48, 32), 4),
                                         ((48, 16, 80), 4), ((144, 16, 16), 4), ((136, 8, 16), 3), ((256, 256, 256), 4)])
def test_convolution_against_float64(shape, depth):
    """Bins of 1, 2, 3, 5, 7, 9, 16 and 17 cells an edge; rows of one and of two tiles; the sums
    of 256^3 go in several passes."""
    lod = _bins(depth, 5)
    e, b, k = _field(shape, depth, lod)
    cells = _cells(shape)
    ee, be = _exact(shape, depth, lod, cells, k)
    for got, want in ((e, ee), (b, be)):
        err = np.linalg.norm(got[:, cells] - want) / np.linalg.norm(want)
        assert err <= 2.3e-6, err


@pytest.mark.parametrize("value", [np.nan, np.inf, -1e30])
def test_sources_out_of_range_take_the_direct_sum(value):
    """A bin that is not finite reaches every cell (its own with weight 0: NaN); the transforms of
    a charge of 1e30 could overflow."""
    shape, depth = (32, 16, 48), 4
    lod = _bins(depth, 6)
    lod[2000, 0] = value
    e, b, k = _field(shape, depth, lod)
    cells = _cells(shape)
    own = np.array([2000 % 16, 2000 // 16 % 16, 2000 // 256]) * np.array([2, 1, 3])
    cells = np.union1d(cells, [own[0] + (own[1] + own[2] * 16) * 32])
    ee, be = _exact(shape, depth, lod, cells, k)
    for got, want in ((e, ee), (b, be)):
        got = got[:, cells]
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fine)
        assert fine.any() == (value == -1e30)
        if fine.any():
            err = np.linalg.norm(got[fine] - want[fine]) / np.linalg.norm(want[fine])
            assert err <= 2e-5, err


def test_batch_of_both_forms_equals_individual():
    """Domains of 16^3 and 8^3 bins, one of the direct form and one whose charges are not finite,
    advanced together and alone."""
    cases = [W.mhd_plasma(shape=s, depth=d, field_mode=1, magnet_r=4.0, magnet_t=3.0)
             for s, d in (((48, 32, 16), 4), ((24, 40, 16), 3), ((16, 16, 16), 2), ((32, 32, 32), 4))]
    cases[3]["fields"]["q"] = cases[3]["fields"]["q"].copy()
    cases[3]["fields"]["q"][20000] = np.nan
    steps = 9
    solo = [U.run_gpu(c, steps) for c in cases]
    doms = [U.setup_gpu(c) for c in cases]
    for d in doms:
        d.initialize()
    b = I.Batch(doms)
    b.run(steps)
    b.finish(120000)
    for c, d, s in zip(cases, doms, solo):
        for name in U.field_names(c):
            ft = c["config"]["float_type"] if name in ("fi", "fqi", "ei") else None
            assert U.bit_diff_nan(d.read(name), s.read(name), ft) == 0, name
    b.close()
