"""Ghost cells by a cluster of CTAs per block (k_bc.cu): which warp takes which
item depends on the cluster's width, which depends on the number of blocks, and
the values must not.  One case alone (the wide cluster) and in a batch of 80 with
160 blocks (the narrow one) give the same bits, at subfaces longer than one pass
of either cluster's warps and on the smallest blocks; the parity tests compare
the ghosts of both with the oracle."""
import numpy as np
import pytest

from ec2d import gpu, grids
from ec2d.inputs import Params
from helpers import copy_state, make_gpu, make_oracle, perturb_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turb", [0, 2, 3])
@pytest.mark.parametrize("twall", [-1.0, 300.0])
@pytest.mark.parametrize("nx,ny", [(3, 3), (18, 9), (1101, 5), (7, 1030)])
def test_cluster_width(gpu_lib, nx, ny, twall, turb):
    kw = dict(Ma=0.4, Re=1e5, If_viscous=1, Iflag_turbulence_model=turb, Iflag_flux=6, Iflag_Scheme=5, CFL=1.0,
              Time_Method=0, P_outlet=1.0 / (1.4 * 0.16), Twall=twall)
    if turb == 3:
        kw.update(Kt_inf=1e-6, Wt_inf=1e-2)
    p, bl = Params(**kw), grids.flat_plate(nx, ny, first=2e-3, ratio=1.02 if ny < 100 else 1.005)
    orc, one, many = make_oracle(p, bl), make_gpu(p, bl), gpu.Solver([(p, bl)] * 80)
    orc.init_flow(), one.init_flow(), many.init_flow()
    perturb_state(orc, amp=0.01, seed=nx)
    copy_state(orc, one)
    for case in (1, 80):
        copy_state(orc, many, case=case)
    for g in (one, many):
        g.bc(1), g.halo(1)
    for b in (1, 2):
        a = one.download_U(1, 1, b)
        assert not np.array_equal(a, orc.get_U(1, b))  # the ghosts were written
        for case in (1, 80):
            assert np.array_equal(a, many.download_U(case, 1, b))
    one.close(), many.close()
