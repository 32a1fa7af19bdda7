"""Blocks of more rows than a CTA's sweep takes have no array of sweep records: the slopes
of the two directions take turns in planes of the fluxes and of Res.  Residuals against
the CPU oracle, Res and Lc of all entries that a host reads, and RK3 steps."""
import numpy as np
import pytest

from ec2d import grids
from ec2d.inputs import Params
from helpers import compare_U, compare_fields, compare_residual, copy_state, make_gpu, make_oracle, perturb_state

pytestmark = pytest.mark.gpu

F_LCI, F_LCJ = 2, 3


def _case(turb, tm=3, ny=1153, fdm=()):
    p = Params(Ma=0.4, Re=1e5, If_viscous=int(turb >= 0), Iflag_turbulence_model=max(turb, 0), Iflag_flux=6,
               Iflag_Scheme=5, CFL=0.5, Time_Method=tm, P_outlet=1.0 / (1.4 * 0.16),
               **(dict(Kt_inf=1e-6, Wt_inf=1e-2) if turb == 3 else {}))
    return p, grids.flat_plate(129, ny, first=2e-3, ratio=1.002)


@pytest.mark.parametrize("turb,fdm", [(-1, ()), (0, ()), (2, ()), (3, ()), (0, (2,))])
def test_residual(gpu_lib, turb, fdm):
    p, bl = _case(turb)
    orc, g = make_oracle(p, bl, fdm=fdm, threads=16), make_gpu(p, bl, fdm=fdm)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=3)
    copy_state(orc, g)
    orc.residual()
    g.kernel_timing(True)
    g.residual(), g.residual()
    names = {n for n, _ in g.kernel_times()}
    g.kernel_timing(False)
    assert {"k_slopes_i", "k_slopes_j"} <= names and "k_slopes" not in names
    compare_residual(orc, g)
    compare_fields(orc, g, [F_LCI, F_LCJ])
    g.set_lusgs_precision(32)
    g.residual()
    compare_residual(orc, g)
    g.close()


def test_rk3_steps(gpu_lib):
    p, bl = _case(0)
    orc, g = make_oracle(p, bl, threads=16), make_gpu(p, bl)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=3)
    copy_state(orc, g)
    orc.step(2), g.step(2)
    compare_U(orc, g, tol=1e-11, interior_only=True)
    ro, rg = orc.norms(1), g.norms(1)
    np.testing.assert_allclose(rg[1][:4], ro[1][:4], rtol=1e-9)
    g.close()
