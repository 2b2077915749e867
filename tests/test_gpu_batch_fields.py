"""Batches whose domains' FAST fields take different ways: convolutions of one and of two passes (the sums
of more than 48 MB), convolutions at both depths, and domains whose charge sits in a few bins, for which
the direct sum stands by (k_batch_field_gated).  Bit-identical to the domains stepped alone."""
import numpy as np
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu


def _case(shape, depth, concentrated):
    case = W.mhd_plasma(shape=shape, depth=depth, field_mode=1, magnet_r=4.0, magnet_t=3.0)
    if concentrated:
        nx, ny, nz = shape
        q = np.zeros((nz, ny, nx), np.float32)
        q[nz // 2:nz // 2 + 2, ny // 2:ny // 2 + 2, nx - 4:nx - 2] = 0.1
        case["fields"]["q"] = q.reshape(-1)
        case["fields"]["u"] = np.zeros_like(case["fields"]["u"])
    return case


@pytest.mark.parametrize("spec", [
    [((48, 32, 16), 4, True), ((32, 32, 32), 4, False), ((40, 24, 32), 3, True), ((24, 40, 16), 3, False)],
    [((32, 32, 32), 4, True), ((64, 48, 32), 4, True)],
    [((144, 128, 128), 4, False), ((32, 32, 32), 4, False), ((160, 128, 112), 4, True), ((16, 16, 16), 2, False)]],
    ids=["open-and-closed", "all-open", "two-passes"])
def test_batch_equals_individual(spec):
    cases = [_case(*s) for s in spec]
    steps = 5
    solo = [U.run_gpu(c, steps) for c in cases]
    for (shape, depth, concentrated), s in zip(spec, solo):
        first = sum(8 ** k for k in range(depth))
        q = np.abs(s.read("qu_lod").reshape(-1, 4)[first:8 ** depth, 0])
        assert np.isfinite(q).all()
        if depth > 2:  # as many evenly charged bins; the line lies near 300 at depth 4 and 70 at depth 3
            bins = q.sum() ** 2 / (q.astype(np.float64) ** 2).sum()
            assert bins < (150, 40)[depth == 3] if concentrated else bins > (1000, 120)[depth == 3], bins
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
