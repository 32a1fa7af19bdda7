"""Norms of the coarse levels of V-cycles smoothed by Euler and RK3 steps, whose
updates leave Res + QF in Res: with the norms on a branch of their own they are
those of the one-stream order, bit for bit, after every cycle."""
import numpy as np
import pytest

from helpers import make_gpu, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("tm,num_mesh", [(1, 2), (1, 3), (3, 2), (3, 3)])
def test_coarse_norms(gpu_lib, monkeypatch, tm, num_mesh, graphs):
    p, bl = small_case(nx=257, ny=65, Ma=0.6, AoA=2.0, Iflag_flux=4, Iflag_Scheme=5, Time_Method=tm, Num_Mesh=num_mesh,
                       CFL=0.5, Pre_Step_Mesh=(0, 5, 5))
    runs = []
    for conc in ("1", "0"):
        monkeypatch.setenv("EC2D_CONCURRENT", conc)
        g = make_gpu(p, bl)
        g.set_graphs(graphs)
        g.init_flow()
        runs.append(g)
    a, b = runs
    for _ in range(6):
        a.step(1), b.step(1)
        for mesh in range(1, num_mesh + 1):
            na, nb = a.norms(1, mesh), b.norms(1, mesh)
            np.testing.assert_array_equal(na[0], nb[0])
            np.testing.assert_array_equal(na[1], nb[1])
    np.testing.assert_array_equal(a.download_U(1, 1, 1), b.download_U(1, 1, 1))
    a.close(), b.close()
