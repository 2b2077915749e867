"""A concentrated current that is lost in the rounding of B = B_stat + KMU b keeps the FAST field's
convolution (csrc/field_fft.cu, `concentrated`); where one cell's B is small enough to show it, the direct
sum runs.  As in test_gpu_field_sources.py, E of the charges times 2^90, which always take the
direct sum, tells which form ran.

Tolerance of B where the convolution ran: half an ulp of the sum (2^-24 of B) and of the product with KMU,
half an ulp for the convolution's own error (2^-25), and 2.5e-6 of the cell's sum of |w|/|R|^2."""
import itertools

import numpy as np
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu
SCALE = np.float32(2.0 ** 90)


def _config(shape, depth):
    case = W.mhd_plasma(shape=(32, 32, 32), depth=depth, field_mode=1)
    case["config"].update(n_x=shape[0], n_y=shape[1], n_z=shape[2], mhd_lod_depth=depth)
    return W.lbm_config(case)


def _kappa(edges, nd):
    total = 0.0
    for o in itertools.product(range(4), repeat=3):
        r = [(e * np.arange(-4, 5) + ((2 * k + 1) * e) // 8 - e / 2) ** 2 for e, k in zip(edges, o)]
        r2 = r[0][:, None, None] + r[1][None, :, None] + r[2][None, None, :]
        r2[4, 4, 4] = np.inf
        total += (1.0 / r2 ** 2).sum()
    return (total / 64.0 / (2 * nd) ** 3) ** 0.5


def _fields(lbm, q, v, b_stat):
    nd = q.shape[0]
    out = []
    lbm.write("b_stat", b_stat.reshape(-1))
    for scale in (np.float32(1.0), SCALE):
        lod = np.zeros((sum(8 ** k for k in range(nd.bit_length())), 4), np.float32)
        lod[:nd ** 3, 0] = q.reshape(-1) * scale
        lod[:nd ** 3, 1:] = v.reshape(3, -1).T
        lbm.write("qu_lod", lod.reshape(-1))
        lbm.initialize()
        lbm.finish_queues(60000)
        out.append([lbm.read(name)[:3 * lbm.n].reshape(3, -1) / s for name, s in (("e_dyn", scale), ("b_dyn", np.float32(1.0)))])
    return out[0][0], out[0][1], out[1][0]


@pytest.mark.parametrize("shape,depth", [((128, 128, 128), 4), ((48, 32, 80), 4), ((40, 24, 56), 3), ((8, 8, 8), 3)])
def test_a_current_below_the_rounding_of_b_keeps_the_convolution(shape, depth):
    nd, n = 1 << depth, int(np.prod(shape))
    bs = np.array([s // nd for s in shape])
    rng = np.random.Generator(np.random.PCG64(5))
    q = rng.normal(0.0, 1e-2, (nd, nd, nd)).astype(np.float32)
    v = np.zeros((3, nd, nd, nd), np.float32)
    at = (nd - 2, nd // 2, nd - 1)  # z, y, x
    v[0][at] = 1e-3
    w = float(q[at]) * 1e-3
    cfg = _config(shape, depth)
    kmu = cfg.constants()["kmu"]
    noise = abs(w) * _kappa(bs, nd) * kmu
    xyz = np.stack([np.arange(n) % shape[0], np.arange(n) // shape[0] % shape[1], np.arange(n) // (shape[0] * shape[1])])
    own = (xyz // bs[:, None] == np.array(at[::-1])[:, None]).all(0)
    r = xyz - ((np.array(at[::-1]) + 0.5) * bs)[:, None]
    r2 = (r * r).sum(0)
    size = np.where(own, 0.0, abs(w) * kmu / np.where(r2 > 0, r2, 1.0))
    near = size / np.sqrt(np.where(r2 > 0, r2, 1.0))
    with I.Lbm(cfg) as lbm:
        b_stat = np.zeros((3, n), np.float32)
        b_stat[1] = 1024.0 * noise + 2.0 * size  # above 256 of the noise whatever the current adds
        e, b, direct = _fields(lbm, q, v, b_stat)
        assert not np.array_equal(e, direct)
        want = b_stat.astype(np.float64)
        for c, a, s in ((1, 2, -1.0), (2, 1, 1.0)):  # (w, 0, 0) x R
            want[c] += s * np.sign(w) * near * r[a]
        err = np.linalg.norm(b - want, axis=0)
        assert np.all(err <= (2.0 ** -23 + 2.0 ** -25) * np.linalg.norm(want, axis=0) + 2.5e-6 * size)
        # one cell far from the current without a static field: its B is the current's alone
        b_stat[:, 0] = 0.0
        e, b, direct = _fields(lbm, q, v, b_stat)
        assert np.array_equal(e, direct)


def _moving_cluster(shape, depth):
    """Charge everywhere, a few cells that move, no static field."""
    case = W.mhd_plasma(shape=shape, depth=depth, field_mode=1)
    case["meshes"], case["precompute_b"] = [], False
    nx, ny, nz = shape
    u = np.zeros((3, nz, ny, nx), np.float32)
    u[0, nz // 2:nz // 2 + 2, ny // 2:ny // 2 + 2, nx - 6:nx - 4] = 1e-3
    case["fields"]["u"] = u.reshape(-1)
    return case


@pytest.mark.parametrize("shapes", [[((48, 32, 48), 4), ((40, 24, 32), 3)], [((32, 32, 32), 4)]])
def test_batch_takes_the_direct_sum_as_its_domains_do(shapes):
    cases = [_moving_cluster(*s) for s in shapes] + [W.mhd_plasma(shape=(32, 32, 32), depth=3, field_mode=1)]
    steps = 2
    solo = [U.run_gpu(c, steps) for c in cases]
    for (shape, depth), s in zip(shapes, solo):
        first = sum(8 ** k for k in range(depth))
        lod = s.read("qu_lod").reshape(-1, 4)[first:8 ** depth].astype(np.float64)
        for w, few in ((lod[:, 0], False), (lod[:, 0] * lod[:, 1], True)):  # as many evenly filled bins; the line: 300 and 70
            bins = np.abs(w).sum() ** 2 / (w ** 2).sum()
            assert bins < (150, 40)[depth == 3] if few else bins > (1000, 120)[depth == 3], bins
    doms = [U.setup_gpu(c) for c in cases]
    for d in doms:
        d.initialize()
    b = I.Batch(doms)
    b.run(steps)
    b.finish(120000)
    for c, d, s in zip(cases, doms, solo):
        for name in U.field_names(c):
            assert U.bit_diff_nan(d.read(name), s.read(name)) == 0, name
    b.close()
