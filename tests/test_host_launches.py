"""What the host code launches and keeps, on a CUDA runtime without a device (_fake_cuda.py)."""
import numpy as np
import pytest

import ionsolver_gb300 as I
from tests._fake_cuda import fake  # noqa: F401


def _box(lo, hi):
    v = np.array([[x, y, z] for z in (lo, hi) for y in (lo, hi) for x in (lo, hi)], np.float32)
    f = np.array([[0, 2, 1], [1, 2, 3], [4, 5, 6], [5, 7, 6], [0, 1, 4], [1, 5, 4], [2, 6, 3], [3, 6, 7], [0, 4, 2], [2, 4, 6],
                  [1, 3, 5], [3, 7, 5]])
    return tuple(np.ascontiguousarray(v[f[:, k]]) for k in range(3))


@pytest.mark.parametrize("n,form", [(40, "k_voxelize_warp"), (91, "k_voxelize_warp"), (96, "k_voxelizeE"), (200, "k_voxelizeE")])
def test_voxeliser_form_by_columns(fake, n, form):  # noqa: F811
    """Twelve triangles: a warp per column up to 8192 columns inside the mesh's bounds, then a
    thread (a warp each took 3,440 us where a thread each takes 299)."""
    lbm = I.Lbm(I.LbmConfig(velocity_set=2, float_type=0, n_x=n, n_y=n, n_z=n, nu=1 / 30))
    mesh = lbm.add_mesh(*_box(2.5, n - 2.5))
    fake.lib.fake_clear()
    lbm.voxelise_mesh(mesh, I.ModelType.Solid())
    assert fake.kernel("k_voxelize")["name"].startswith(form)
    lbm.close()


def _mhd(shape, depth, mode=0, **changes):
    c = I.LbmConfig(velocity_set=2, float_type=2, n_x=shape[0], n_y=shape[1], n_z=shape[2], nu=1 / 30, ext_volume_force=True,
                    ext_magneto_hydro=True, mhd_lod_depth=depth, field_mode=mode)
    for k, v in changes.items():
        setattr(c, k, v)
    return I.Lbm(c)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("edge,accepted", [(32, True), (33, False)])
def test_learned_field_bins_of_at_most_32_cells_an_edge(fake, axis, edge, accepted):  # noqa: F811
    """k_surrogate_cells' tables hold 32 cells an axis (a larger bin read past them)."""
    shape = [16, 16, 16]
    shape[axis] = 8 * edge
    lbm = _mhd(shape, 3)
    if accepted:
        lbm.set_field_mode(2)
    else:
        with pytest.raises(I.IonError) as e:
            lbm.set_field_mode(2)
        assert e.value.code == -2
    lbm.close()


def _plain(shape, ft=2):
    lbm = I.Lbm(I.LbmConfig(velocity_set=2, float_type=ft, n_x=shape[0], n_y=shape[1], n_z=shape[2], nu=1 / 30))
    lbm.initialize()
    return lbm


def test_row_plan_belongs_to_its_device(fake):  # noqa: F811
    """The opt-in for more than 48 KB of shared memory is per device: the same grid on a second
    device gets one of its own."""
    shape = (384, 16, 16)
    for device in (0, 1, 0):
        assert fake.lib.ion_select_device(device) == 0
        lbm = _plain(shape)
        lbm.do_time_step()
        k = fake.kernel("k_sc_rows_ws")
        assert k["device"] == device and k["smem"] > 48 * 1024
        lbm.close()


@pytest.mark.parametrize("call", ["cudaFuncSetAttribute", "cudaOccupancy"])
def test_row_plan_that_failed_is_not_kept(fake, call):  # noqa: F811
    """A runtime call that fails once costs one step the row kernels, and its error is not the
    fallback's."""
    lbm = _plain((320, 16, 16))
    fake.fail(call)
    lbm.do_time_step()
    assert fake.launches()[-1]["name"].startswith("k_stream_collide")
    lbm.do_time_step()
    assert fake.launches()[-1]["name"].startswith("k_sc_rows_ws")
    lbm.close()


@pytest.mark.parametrize("shape,ft", [((16, 16, 16), 2), ((16, 16, 2), 0), ((32, 16, 16), 1), ((48, 12, 12), 2)])
@pytest.mark.parametrize("mhd", [False, True])
def test_few_short_rows_are_staged_one_by_one(fake, shape, ft, mhd):  # noqa: F811
    """A row a block while the resident blocks hold all of them (in groups of three to six 16^3
    took 8.4 us instead of 5.2)."""
    if mhd:
        shape = tuple(max(16, s) for s in shape)
        lbm = _mhd(shape, 2, float_type=ft)
        lbm.initialize()
    else:
        lbm = _plain(shape, ft)
    lbm.do_time_step()
    k = fake.kernel("k_sc_rows_ws")
    assert k["grid"] == shape[1] * shape[2] and k["block"] == (shape[0] + 31) // 32 * 32 + 32
    lbm.close()


def test_many_short_rows_are_staged_in_groups(fake):  # noqa: F811
    lbm = _plain((16, 96, 96))
    lbm.do_time_step()
    assert fake.kernel("k_sc_rows_ws")["block"] >= 4 * 16 + 32
    lbm.close()


@pytest.mark.parametrize("shape", [(16, 44, 44), (32, 44, 44), (32, 52, 33)])
def test_rows_that_would_fill_the_resident_blocks_are_staged_in_pairs(fake, shape):  # noqa: F811
    """A row each would take more than half the resident blocks (32x44x44: 7.2 us instead of 6.2)."""
    lbm = _plain(shape)
    lbm.do_time_step()
    k = fake.kernel("k_sc_rows_ws")
    assert k["block"] == 2 * shape[0] + 32 and k["grid"] == (shape[1] + 1) // 2 * shape[2]
    lbm.close()


@pytest.mark.parametrize("shape,mhd,blocks", [((160, 128, 128), False, 4), ((224, 128, 128), False, 3), ((128, 128, 128), False, 5),
                                              ((160, 64, 64), False, 5), ((96, 96, 96), True, 4)])
def test_fp32_rows_beyond_l2_are_staged_on_fewer_blocks(fake, shape, mhd, blocks):  # noqa: F811
    """At most 720 cells of the plain stencil and 400 of the MHD one on an SM (160^3 took 119.7 us with
    the five blocks that fit, 112 with four); a lattice inside L2 keeps them all."""
    lbm = _mhd(shape, 2) if mhd else _plain(shape)
    lbm.initialize()
    lbm.do_time_step()
    assert fake.kernel("k_sc_rows_ws")["grid"] == blocks * 152
    lbm.close()


@pytest.mark.parametrize("ft", [0, 2])
def test_mhd_trt_rows_of_128_keep_four_blocks(ft):
    """At most 102 registers, so that four blocks of 160 threads fit (with 128 registers three: FP32
    112x128x128 144 us instead of 130)."""
    from ionsolver_gb300 import build as B
    log = (B.OUT / "ptxas.log").read_text()
    name = f"k_sc_rows_wsILi{ft}ELb1ELb1ELj128E"
    if name not in log:
        pytest.skip("the stencil was not compiled by the last build")
    used = log[log.index(name):].split("Used ")[1].split()[0]
    assert int(used) <= 102


def test_d2q9_stencils_do_not_spill():
    """(bounded to six blocks an SM the 16-bit ones did: FP16S 700^2 10.1 us instead of 9.3)"""
    import re
    from ionsolver_gb300 import build as B
    log = (B.OUT / "ptxas.log").read_text()
    found = 0
    for ft in range(3):
        for trt in range(2):
            name = f"k_stream_collideILi9ELi{ft}ELb0ELb{trt}ELb0E"
            if name in log:
                found += 1
                assert int(re.search(r"(\d+) bytes spill stores", log[log.index(name):]).group(1)) == 0, name
    if not found:
        pytest.skip("the stencil was not compiled by the last build")


def _fill(fake, mode, depth):
    """Handles of 64^3 until one does not fit."""
    out = []
    try:
        while len(out) < 64:
            out.append(_mhd((64, 64, 64), depth, mode))
    except I.IonError as e:
        assert e.code == -4
    return out


@pytest.mark.parametrize("mode", [0, 1])
def test_handles_that_fit_without_field_tables_fit_with_them(fake, mode):  # noqa: F811
    """Tables and plans take at most an eighth of the device and leave another free: as many handles
    as 7/8 of it hold are created (with a table each 11 of 14)."""
    plain = _mhd((64, 64, 64), 2, mode)  # depth 2: neither table nor plan
    bytes_each = fake.lib.fake_used()
    plain.close()
    assert fake.lib.fake_used() == 0
    fake.lib.fake_memory(1 << 30)
    for _ in range(2):  # what the first handles gave back serves the next ones
        handles = _fill(fake, mode, 4)
        assert len(handles) >= (7 << 27) // bytes_each
        kernel = "k_field_table" if mode == 0 else "k_fft_plan"
        assert sum(x["name"].startswith(kernel) for x in fake.launches()) >= 1
        for h in handles:
            h.close()
        assert fake.lib.fake_used() == 0
        fake.lib.fake_clear()


def test_the_table_goes_with_its_mode(fake):  # noqa: F811
    lbm = _mhd((64, 64, 64), 4, 1)
    fast = fake.lib.fake_used()
    lbm.close()
    lbm = _mhd((64, 64, 64), 4, 0)
    lbm.set_field_mode(1)
    assert fake.lib.fake_used() == fast
    lbm.set_field_mode(0)
    lbm.initialize()
    assert fake.kernel("k_update_e_b_table")
    lbm.close()


@pytest.mark.parametrize("before,after,setup,step", [(0, 1, "k_fft_plan", "k_update_e_b_table"), (1, 0, "k_field_table", "k_fft_sum")])
def test_a_switch_that_failed_leaves_the_mode(fake, before, after, setup, step):  # noqa: F811
    lbm = _mhd((32, 32, 32), 4, before)
    lbm.initialize()
    used = fake.lib.fake_used()
    fake.fail(setup)
    with pytest.raises(I.IonError):
        lbm.set_field_mode(after)
    assert fake.lib.fake_used() == used
    fake.lib.fake_clear()
    lbm.do_time_step()
    assert fake.kernel(step)
    lbm.set_field_mode(after)
    fake.lib.fake_clear()
    lbm.do_time_step()
    assert not any(x["name"].startswith(step) for x in fake.launches())
    lbm.close()


@pytest.mark.parametrize("depth,tuned", [(2, True), (4, False)])
def test_batch_tunes_only_what_it_launches(fake, depth, tuned):  # noqa: F811
    """The shape that the autotuner tries is the direct field sums'; where every field is a convolution
    it timed the same launches several times and reported one of them."""
    doms = [_mhd((32, 32, 32), depth, 1) for _ in range(2)]
    b = I.Batch(doms)
    b.run(40)
    assert bool(b.tuning()) == tuned and b.chosen()[0] in (128, 256)
    b.close()
    for d in doms:
        d.close()
