"""A periodic domain one thin tile wide in y (ny = 4): the x/y kernel takes the
edges of the halo cells that close a y line from the tile's own first and last
cells.  The same flow repeated once more in y (ny = 8, two tiles, whose closing
cells are reconstructed) gives the same bits, on the same profiles."""
import numpy as np
import pytest

from helpers import gpu_run, twice_in_y
from porturb_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("nx,nz,immersed,ntr", [(32, 32, False, 1), (37, 20, True, 2), (200, 130, False, 2)])
def test_closing_cells_of_a_thin_periodic_domain(gpu_lib, precision, nx, nz, immersed, ntr):
    case = cases.small_mixed(nx=nx, ny=4, nz=nz, immersed=immersed, ntr=ntr)
    _, _, g = gpu_run(case, precision, 0, 0.0)
    dt, cells = 0.9 * g.compute_time_step(), g.get_hydrostasis()[0]
    st4, tr4, _ = gpu_run(case, precision, 3, dt, hydro=cells)
    st8, tr8, _ = gpu_run(twice_in_y(case), precision, 3, dt, hydro=cells)
    for a, b in ((st4, st8), (tr4, tr8)):
        assert np.array_equal(a, b[:, :, :4]) and np.array_equal(a, b[:, :, 4:])
