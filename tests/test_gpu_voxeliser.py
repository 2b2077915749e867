"""The voxeliser's two forms (csrc/setup_kernels.cu) against the oracle."""
import numpy as np
import pytest

from ionsolver_gb300 import workloads as W
from tests import _util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shape", [(96, "cube"), (100, "cube"), (72, "slab")])
def test_voxeliser_forms_against_oracle(n, shape):
    """A thread per column (meshes that span more than 8192 columns; few triangles) and a warp
    per column mark the same cells as the oracle."""
    nz = n if shape == "cube" else 24
    v = np.array([[x, y, z] for z in (2.4, nz - 3.3) for y in (3.2, n - 2.7) for x in (2.6, n - 3.1)], np.float32)
    f = np.array([[0, 2, 1], [1, 2, 3], [4, 5, 6], [5, 7, 6], [0, 1, 4], [1, 5, 4], [2, 6, 3], [3, 6, 7], [0, 4, 2], [2, 4, 6],
                  [1, 3, 5], [3, 7, 5]])
    mesh = tuple(np.ascontiguousarray(v[f[:, k]]) for k in range(3))
    case = {"config": dict(velocity_set=2, relaxation_time=0, float_type=2, n_x=n, n_y=n, n_z=nz, nu=W.NU_1_30, update_fields=1),
            "fields": {}, "meshes": [(*mesh, "solid", (0.0, 0.0, 0.0))], "precompute_b": False}
    g, o = U.setup_gpu(case), U.setup_oracle(case)
    assert np.array_equal(g.read("flags"), o.field("flags")) and g.read("flags").any()
