"""The BITWISE field from tabulated R/|R|^3 (csrc/field_table.cu) against the direct sum: a
domain stepped alone takes the table, as one of a batch the direct sum (eb_tile); every field is
bit-identical.  Bins of 1, 2, 3, 5, 7 and 17 cells an edge, two and four cells a thread; above
2^25 cells the table of |2 R|."""
import pytest

import ionsolver_gb300 as I
from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,depth", [((16, 16, 16), 4), ((32, 48, 16), 4), ((8, 16, 40), 3), ((24, 40, 56), 3),
                                         ((112, 48, 64), 4), ((136, 64, 40), 3), ((2064, 128, 128), 4),
                                         ((2056, 136, 128), 3)])
def test_table_equals_direct_sum(shape, depth):
    case = W.mhd_plasma(shape=shape, depth=depth, field_mode=0, magnet_r=2.0, magnet_t=2.0)
    solo = U.run_gpu(case, 2)
    dom = U.setup_gpu(case)
    b = I.Batch([dom])
    b.run(2)
    b.finish(120000)
    for name in U.field_names(case):
        assert U.bit_diff_nan(dom.read(name), solo.read(name)) == 0, name
    b.close()
