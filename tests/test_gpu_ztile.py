"""The tiled z kernel (k_zt: 8 columns x 32 levels per block, the default
for FP32 with weno_all) gives the bits of the z march (k_z, selected by an
explicit z chunk): the same primitive fields, wall and periodic halos,
immersed and wall-adjacent stencil modifications, face states, limiter bits
per stencil, Riemann fluxes, stage combination, immersed relaxation and
positivity clip.  Cases: walls with and without an immersed cuboid,
periodic z, three tracers (an odd number of fields), precursor x/y,
Coriolis, a 2-D domain, the warm bubble, and grids whose x and z extents
are not multiples of the tile (partial tiles, several z tiles)."""
import numpy as np
import pytest

from porturb_b200 import cases
from helpers import gpu_run

pytestmark = pytest.mark.gpu

CASES = {
    "walls": lambda: cases.small_mixed(immersed=False),
    "walls_immersed": lambda: cases.small_mixed(),
    "periodic_z_immersed": lambda: cases.small_mixed(bc_z="periodic", nz=40),
    "partial_tiles_immersed": lambda: cases.small_mixed(nx=37, ny=6, nz=75),
    "periodic_z": lambda: cases.small_mixed(bc_z="periodic", immersed=False),
    "periodic_z_tall": lambda: cases.small_mixed(bc_z="periodic", nz=70, immersed=False),
    "three_tracers": lambda: cases.small_mixed(ntr=3, immersed=False),
    "precursor_xy": lambda: cases.small_mixed(bc_x="precursor", bc_y="precursor", immersed=False),
    "coriolis": lambda: cases.small_mixed(latitude=43.29, immersed=False),
    "sim2d": lambda: cases.small_mixed(ny=1, nx=24, nz=16, immersed=False),
    "partial_tiles": lambda: cases.small_mixed(nx=37, ny=6, nz=75, immersed=False),
    "bubble_small": lambda: cases.warm_bubble(nx=64, ny=4, nz=32, xlen=5000.0, ylen=312.5, zlen=2500.0,
                                              radius=500.0, x0=2500.0, z0=600.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tiled_z_kernel_gives_the_march_bits(name, gpu_lib):
    case = CASES[name]()
    _, _, g = gpu_run(case, "f32", 0, 0.0)
    dt = 0.9 * g.compute_time_step()
    st_t, tr_t, _ = gpu_run(case, "f32", 4, dt)
    st_m, tr_m, _ = gpu_run(case, "f32", 4, dt, z_chunk=16)
    st0, _, _ = gpu_run(case, "f32", 0, dt)
    assert not np.array_equal(st_t, st0)
    assert np.array_equal(st_t, st_m), np.abs(st_t - st_m).max()
    assert np.array_equal(tr_t, tr_m), np.abs(tr_t - tr_m).max()


@pytest.mark.parametrize("name", sorted(CASES))
def test_tiled_z_kernel_in_fp64(name, gpu_lib):
    """The FP64 build takes the tile too (weno_all); its arithmetic is the
    march's up to the contraction of products, so after 4 steps the two agree
    to FP64 rounding (2^-53, times ~1e4 for the nonlinear weights where a
    stencil is nearly uniform) of each field's magnitude."""
    case = CASES[name]()
    _, _, g = gpu_run(case, "f64", 0, 0.0)
    dt = 0.9 * g.compute_time_step()
    st_t, tr_t, _ = gpu_run(case, "f64", 4, dt)
    st_m, tr_m, _ = gpu_run(case, "f64", 4, dt, z_chunk=16)
    for a, b in list(zip(st_t, st_m)) + list(zip(tr_t, tr_m)):
        assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("nx,ny,nz,bc_z", [(104, 96, 4, "solid_wall"), (96, 83, 4, "periodic"),
                                           (250, 130, 5, "solid_wall"), (256, 140, 16, "periodic")])
def test_shallow_fp64_grids_keep_the_march(nx, ny, nz, bc_z, gpu_lib):
    """FP64 on up to 16 levels and more than 250 nz tiles of 8 columns (the
    second case is below that: 996 tiles): the march's results, to the last bit
    where the call takes it."""
    case = cases.small_mixed(nx=nx, ny=ny, nz=nz, ntr=1, immersed=False, bc_z=bc_z)
    _, _, g = gpu_run(case, "f64", 0, 0.0)
    dt = 0.9 * g.compute_time_step()
    a = gpu_run(case, "f64", 3, dt)
    b = gpu_run(case, "f64", 3, dt, z_chunk=16)
    marches = -(-nx // 8) * ny > 250 * nz
    for x, y in zip(a[:2], b[:2]):
        assert np.array_equal(x, y) if marches else np.abs(x - y).max() <= 1e-12 * np.abs(y).max()


LARGE = {
    "immersed": lambda: cases.small_mixed(nx=72, ny=40, nz=40),
    "three_tracers_partial": lambda: cases.small_mixed(nx=70, ny=41, nz=45, ntr=3, immersed=False),
    "periodic_z": lambda: cases.small_mixed(nx=64, ny=48, nz=70, bc_z="periodic", immersed=False),
    "thin": lambda: cases.small_mixed(nx=160, ny=5, nz=64),
}


@pytest.mark.parametrize("name", sorted(LARGE))
def test_one_thread_per_cell(name, gpu_lib):
    """Grids of more blocks than fit the SMs at four threads per cell, which the
    grids above all take: the tile gives the march's bits there too, with the
    x/y kernel's tiles staged through TMA or loaded by its threads."""
    case = LARGE[name]()
    _, _, g = gpu_run(case, "f32", 0, 0.0)
    dt = 0.9 * g.compute_time_step()
    st_t, tr_t, _ = gpu_run(case, "f32", 2, dt)
    for kw in (dict(z_chunk=16), dict(thread_loads=True)):
        st_m, tr_m, _ = gpu_run(case, "f32", 2, dt, **kw)
        assert np.array_equal(st_t, st_m) and np.array_equal(tr_t, tr_m), kw
    # A case of one such tile column more or less: four threads per cell.
    block = case.block(0, 0, 16, min(case.ny, 16))
    st_s, tr_s, _ = gpu_run(block, "f32", 2, dt)
    st_c, tr_c, _ = gpu_run(block, "f32", 2, dt, z_chunk=16)
    assert np.array_equal(st_s, st_c) and np.array_equal(tr_s, tr_c)
