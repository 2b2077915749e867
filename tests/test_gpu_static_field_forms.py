"""Which form of the magnets' potential runs (csrc/setup_kernels.cu): short lists, and lists whose table
would cost more than it saves, are summed directly, long runs through the table.  Each against the
oracle, bit for bit; the number of launches tells the form: three of the compaction, two of the
direct sum of short lists, one that looks for runs (on fewer than 2^18 points of longer lists only),
then three with a table or two of the direct sum of long lists."""
import numpy as np
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu


def _case(shape, cells, kind, kinds=1):
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.Generator(np.random.PCG64(4))
    if kind == "block":
        e = max(1, int(np.ceil(cells ** (1 / 3))))
        k = np.arange(cells)
        at = (2 + k % e) + ((3 + k // e % e) + (4 + k // (e * e)) * ny) * nx
    else:
        at = np.sort(rng.choice(n, cells, replace=False))
    m = rng.normal(0.0, 1.0, (kinds, 3)).astype(np.float32)
    flags, b = np.zeros(n, np.uint8), np.zeros((3, n), np.float32)
    flags[at] = 0x11
    b[:, at] = m[np.arange(cells) % kinds].T
    case = W.mhd_box(n=16, shape=shape, depth=2, magnet=False)
    case["fields"].update(flags=flags, b_dyn=b.reshape(-1))
    case["precompute_b"] = False
    return case


@pytest.mark.parametrize("shape,cells,kind,kinds,launches", [
    ((24, 20, 28), 0, "block", 1, 5), ((24, 20, 28), 1, "block", 1, 5), ((24, 20, 28), 100, "block", 1, 5),
    ((24, 20, 28), 100, "scattered", 1, 5), ((24, 20, 28), 1200, "block", 1, 9), ((24, 20, 28), 1200, "scattered", 1, 8),
    ((24, 20, 28), 1200, "block", 5, 8), ((32, 24, 28), 2500, "block", 1, 9)])
def test_form_of_the_potential(shape, cells, kind, kinds, launches):
    case = _case(shape, cells, kind, kinds)
    g, o = U.setup_gpu(case), U.setup_oracle(case, canonical_nan=True)
    before = I.kernel_launch_count()
    g.precompute_B()
    assert I.kernel_launch_count() - before == launches
    o.precompute_b()
    assert U.compare_bitwise(g, o, ["b_stat"]) == {"b_stat": 0}
    g.precompute_B()  # adds to the static field again
    o.precompute_b()
    assert U.compare_bitwise(g, o, ["b_stat"]) == {"b_stat": 0}
