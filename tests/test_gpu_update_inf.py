"""An infinite residual moves a cell to infinity, as the division by the volume does
(IEEE arithmetic), not to NaN: the Euler update of a coarse level with an
infinite forcing."""
import numpy as np
import pytest

from helpers import make_gpu, small_case

pytestmark = pytest.mark.gpu

F_QF = 19


def test_infinite_forcing(gpu_lib):
    p, bl = small_case(nx=65, ny=17, Ma=0.6, AoA=2.0, Iflag_flux=4, Iflag_Scheme=5, Time_Method=1, Num_Mesh=2, CFL=0.5)
    g = make_gpu(p, bl)
    g.init_flow()
    nx, ny, _ = g.dims(1, 2, 1)
    qf = np.zeros((4, nx - 1, ny - 1))
    qf[:, 3, 2] = [np.inf, -np.inf, np.inf, -np.inf]
    g.set_field(1, 2, 1, F_QF, qf)
    g.time_advance(2)
    U = g.download_U(1, 2, 1)[:, 2:nx + 1, 2:ny + 1]
    np.testing.assert_array_equal(U[:, 3, 2], [np.inf, -np.inf, np.inf, -np.inf])
    U[:, 3, 2] = 0.0
    assert np.all(np.isfinite(U))
    g.close()
