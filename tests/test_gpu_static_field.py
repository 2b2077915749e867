"""The static magnet field from tabulated terms (csrc/setup_kernels.cu, k_psi_runs_sum) against
the oracle, bit for bit: one to five magnetisations (five: the direct sum), runs from single
cells to more than two table windows, magnets at the edges of the box and below the 64 cells
from which the table is used."""
import pytest

from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu

M = [(0.0, 0.0, 2e4), (1.5e4, -3e3, 0.0), (-2e4, 1e4, 5e3), (0.0, 0.0, -2e4), (1e3, 2e3, 3e3)]


@pytest.mark.parametrize("kinds", [1, 2, 4, 5])
@pytest.mark.parametrize("shape", [(48, 24, 20), (20, 36, 28), (16, 16, 16)])
def test_magnets_bitwise(shape, kinds):
    nx, ny, nz = shape
    case = W.mhd_box(n=16, shape=shape, depth=2, magnet=False)
    case["meshes"] = []
    for k in range(kinds):
        c = (nx * (0.3 + 0.1 * k), ny * (0.5 - 0.08 * k), nz * (0.2 + 0.15 * k))
        mesh = W.cylinder(c, min(nx, ny) / 2.5 if k == 0 else 3.0 + 0.3 * k, 3.0, axis=2 if k == 0 else k % 3)
        case["meshes"].append(tuple(list(mesh) + ["magnet", M[k]]))
    if shape[0] == 48:  # a bar along most of x
        mesh = W.cylinder((nx * 0.5, ny * 0.8, nz * 0.8), 2.5, 42.0, axis=0)
        case["meshes"].append(tuple(list(mesh) + ["magnet", M[0]]))
    case["precompute_b"] = True
    g = U.setup_gpu(case)
    o = U.setup_oracle(case, canonical_nan=True)
    assert U.compare_bitwise(g, o, ["flags", "b_dyn", "b_stat"]) == {"flags": 0, "b_dyn": 0, "b_stat": 0}
    assert ((g.read("flags") & 0x10) != 0).sum() > 20


def test_few_cells_bitwise():
    case = W.mhd_box(n=16, depth=2, magnet=False)
    case["meshes"] = [tuple(list(W.cylinder((8.0, 8.0, 4.0), 2.0, 2.0, axis=2)) + ["magnet", M[1]])]
    case["precompute_b"] = True
    g = U.setup_gpu(case)
    o = U.setup_oracle(case, canonical_nan=True)
    assert U.compare_bitwise(g, o, ["flags", "b_stat"]) == {"flags": 0, "b_stat": 0}
    assert 0 < ((g.read("flags") & 0x10) != 0).sum() < 64
