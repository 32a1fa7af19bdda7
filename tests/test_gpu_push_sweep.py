"""The eight-lane LU-SGS wavefront (k_sweep_push.cu) against the CPU oracle at
the sizes where its bookkeeping can go wrong: rows that fill or miss a warp's
four, one row beyond a warp or a CTA's band, rows of cells at the edges of the
16-cell record chunks and of the two-chunk ring, the smallest blocks; bands of
one to four warps on one CTA or a cluster; with and without the update of U;
4, 5 and 6 variables."""
import numpy as np
import pytest

from ec2d import grids
from ec2d.inputs import Params
from helpers import copy_state, make_gpu, make_oracle, perturb_state

pytestmark = pytest.mark.gpu

# (nx, ny) nodes per block: (nx - 1) x (ny - 1) cells
SIZES = [(3, 3), (4, 5), (17, 6), (18, 9), (16, 13), (33, 14), (34, 17), (35, 4), (49, 34), (66, 50), (130, 23)]


def _case(nx, ny, turb):
    bl = grids.flat_plate(nx, ny, first=2e-3, ratio=1.05)
    kw = dict(Ma=0.4, Re=1e4 if turb == 0 else 1e6, If_viscous=1, Iflag_turbulence_model=turb, Iflag_flux=6,
              Iflag_Scheme=5, CFL=5.0, Time_Method=0, P_outlet=1.0 / (1.4 * 0.16))
    if turb == 3:
        kw.update(Kt_inf=1e-6, Wt_inf=1e-2)
    return Params(**kw), bl


def _bound(orc, blk, nv, a, c):
    """The bound of a sweep's dU against the oracle's: 1e-12 |dU_m| plus one
    rounding, per hyperplane at most, of the magnitudes a cell's update adds,
    |U_m| of the cell and its neighbours (+ p in the momentum and energy
    rows); 2e-12 for the turbulence rows, whose source terms are thousands of
    times their increment."""
    nx, ny = orc.dims(1, blk)
    U = np.abs(orc.get_U(1, blk)[:nv])
    S = np.maximum.reduce([U[:, 2:nx + 1, 2:ny + 1], U[:, 1:nx, 2:ny + 1], U[:, 3:nx + 2, 2:ny + 1],
                           U[:, 2:nx + 1, 1:ny], U[:, 2:nx + 1, 3:ny + 2]])
    Uc = orc.get_U(1, blk)[:4, 2:nx + 1, 2:ny + 1]
    S[1:4] += 0.4 * (Uc[3] - 0.5 * (Uc[1] ** 2 + Uc[2] ** 2) / Uc[0])
    rel = np.full((nv, 1, 1), 1e-12)
    rel[4:] = 2e-12
    return rel * np.maximum(np.abs(a), np.abs(c)) + np.finfo(np.float64).eps * (nx + ny) * S


@pytest.mark.parametrize("turb", [0, 2, 3])
@pytest.mark.parametrize("rows", [4, 12, 16])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_sweep_edges(gpu_lib, monkeypatch, nx, ny, rows, turb):
    monkeypatch.setenv("EC2D_LUSGS_CLUSTER", "0")
    monkeypatch.setenv("EC2D_LUSGS_ROWS", str(rows))
    monkeypatch.setenv("EC2D_LUSGS_LANES", "8")
    p, bl = _case(nx, ny, turb)
    nv = p.nvar()
    orc, g = make_oracle(p, bl), make_gpu(p, bl)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=nx + ny)
    orc.bc(), orc.halo()
    copy_state(orc, g)
    orc.residual()
    for b in (1, 2):
        for f in range(6):
            g.set_field(1, 1, b, f, orc.field(1, b, f))
    orc.lusgs(1, 1, 0.0), orc.lusgs(1, 2, 0.0)
    g.lusgs(1, 0.0)
    for b in (1, 2):
        a = orc.field(1, b, 6, (nv, nx, ny))[:, :nx - 1, :ny - 1]
        c = g.field(1, 1, b, 6, (nv, nx, ny))[:, :nx - 1, :ny - 1]
        assert np.max(np.abs(a - c) / _bound(orc, b, nv, a, c)) <= 1.0
    # with the update of U inside the sweep: one whole step of both
    copy_state(orc, g)
    orc.step(1), g.step(1)
    assert g.status()[0] == 0
    for b in (1, 2):
        a, c = (U[:, 2:nx + 1, 2:ny + 1] for U in (orc.get_U(1, b), g.download_U(1, 1, b)))
        scale = np.abs(a).reshape(nv, -1).max(axis=1)[:, None, None]
        assert np.max(np.abs(a - c) / scale) <= 1e-10
    g.close()


# rows at the edges of the FP32 sweep's 32-row warps, cells around its ring of
# eight records, and blocks whose rings and inboxes do not fit shared memory
# (the form with a barrier per plane)
SIZES32 = [(3, 3), (8, 33), (9, 34), (10, 32), (17, 65), (40, 66), (70, 98), (18, 340)]


@pytest.mark.parametrize("turb", [0, 2, 3])
@pytest.mark.parametrize("nx,ny", SIZES32)
def test_fp32_sweep_edges(gpu_lib, nx, ny, turb):
    p, bl = _case(nx, ny, turb)
    nv = p.nvar()
    orc, g = make_oracle(p, bl), make_gpu(p, bl)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=nx + ny)
    orc.bc(), orc.halo()
    copy_state(orc, g)
    g.set_lusgs_precision(32)
    orc.residual()
    for b in (1, 2):
        for f in range(6):
            g.set_field(1, 1, b, f, orc.field(1, b, f))
    orc.lusgs(1, 1, 0.0), orc.lusgs(1, 2, 0.0)
    g.lusgs(1, 0.0)
    for b in (1, 2):
        a = orc.field(1, b, 6, (nv, nx, ny))[:, :nx - 1, :ny - 1]
        c = g.field(1, 1, b, 6, (nv, nx, ny))[:, :nx - 1, :ny - 1]
        for m in range(nv):
            # float epsilon (6e-8) times the planes of a sweep, at most
            assert np.abs(a[m] - c[m]).max() <= 6e-8 * max(nx + ny, 40) * np.abs(a[m]).max(), m
    g.step(1)
    g.norms()
    assert g.status()[0] == 0
    g.close()
