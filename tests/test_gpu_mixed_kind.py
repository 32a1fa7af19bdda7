"""Residuals in the arithmetic of contexts with FP32 parts (ec2d_mixed.cuh,
k_turb_mixed.cu) against the CPU oracle within the bound of the FP64 contexts,
over every flux, reconstruction and scheme, the viscous terms, both turbulence
models and the finite-difference patch; and a context that has been switched to
FP32 sweeps and back gives the bits of one that never was."""
import numpy as np
import pytest

from helpers import compare_residual, copy_state, make_gpu, make_oracle, perturb_state, small_case

pytestmark = pytest.mark.gpu

KINDS = [dict(Iflag_flux=f, IFlag_Reconstruction=r, Iflag_Scheme=5) for f in range(1, 7) for r in range(3)]
KINDS += [dict(Iflag_flux=4, IFlag_Reconstruction=0, Iflag_Scheme=s) for s in range(7)]
VISC = dict(Re=5.0e3, If_viscous=1, Iflag_Scheme=5)
TURB = dict(Re=1.0e6, If_viscous=1, Iflag_flux=4, Iflag_Scheme=5, first=2e-4)
KINDS += [dict(VISC, Iflag_flux=6, nblocks=2), dict(VISC, Iflag_flux=4, nblocks=2, IFlag_Reconstruction=2),
          dict(VISC, Iflag_flux=4, fdm=(1, 2), nblocks=2), dict(TURB, Iflag_turbulence_model=2),
          dict(TURB, Iflag_turbulence_model=3, Kt_inf=1e-6, Wt_inf=1e-2)]


@pytest.mark.parametrize("kind", range(len(KINDS)))
def test_mixed_kind(gpu_lib, kind):
    kw = dict(KINDS[kind])
    fdm = kw.pop("fdm", ())
    p, bl = small_case(nx=65, ny=33 if fdm else 17, Ma=0.6, AoA=2.0, **kw)
    orc, g, plain = make_oracle(p, bl, fdm=fdm), make_gpu(p, bl, fdm=fdm), make_gpu(p, bl, fdm=fdm)
    for s in (orc, g, plain):
        s.init_flow()
    for _ in range(3):
        orc.step(1)
    perturb_state(orc, amp=0.005, seed=kind)
    copy_state(orc, g), copy_state(orc, plain)
    g.set_lusgs_precision(32)
    orc.residual(), g.residual()
    compare_residual(orc, g)
    g.set_lusgs_precision(64)
    g.residual(), plain.residual()
    for b in range(1, len(bl) + 1):
        nx, ny = orc.dims(1, b)
        shape = (orc.nvar(1), nx - 1, ny - 1)
        np.testing.assert_array_equal(g.field(1, 1, b, 0, shape), plain.field(1, 1, b, 0, shape))
    g.close(), plain.close()
