"""Contexts with FP32 sweeps: a level with the slopes pass (k_slopes, from 65536 cells)
gives the bits of one without.  Two cases of 32768 cells in one context take the
pass, each alone does not; their residuals are the same."""
import numpy as np
import pytest

from ec2d import gpu, grids
from ec2d.inputs import Params
from helpers import copy_state, make_oracle, perturb_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux,turb", [(6, 0), (4, 2), (4, -1), (3, 0)])
def test_slopes_same_bits(gpu_lib, flux, turb):
    p = Params(Ma=0.6, Re=1e5, If_viscous=int(turb >= 0), Iflag_turbulence_model=max(turb, 0), Iflag_flux=flux,
               Iflag_Scheme=5, CFL=1.0, Time_Method=0, P_outlet=1.0 / (1.4 * 0.36))
    bl = grids.flat_plate(257, 65, first=2e-3, ratio=1.02)
    orc = make_oracle(p, bl)
    orc.init_flow()
    perturb_state(orc, amp=0.02, seed=flux)
    one, two = gpu.Solver([(p, bl)]), gpu.Solver([(p, bl), (p, bl)])
    for s, cases in ((one, 1), (two, 2)):
        s.set_lusgs_precision(32)
        s.init_flow()
        for case in range(1, cases + 1):
            copy_state(orc, s, case=case)
        s.residual(1)
    for case in (1, 2):
        for b in range(1, len(bl) + 1):
            nx, ny = orc.dims(1, b)
            shape = (orc.nvar(1), nx - 1, ny - 1)
            np.testing.assert_array_equal(two.field(case, 1, b, 0, shape), one.field(1, 1, b, 0, shape))
    one.close(), two.close()
