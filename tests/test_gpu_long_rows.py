"""LU-SGS on blocks of long rows in tall bands, where the push form of the wavefront has
no room in shared memory and eight lanes per row go on in pull form: against the
CPU oracle; the bounded wait at a band's edge; and the time of such a block beside
that of one a little shorter, whose rows fit."""
import numpy as np
import pytest

from ec2d import gpu, grids
from ec2d.inputs import Params
from helpers import copy_state, make_gpu, make_oracle, perturb_state
from test_gpu_push_sweep import _bound

pytestmark = pytest.mark.gpu

# (cells per row, rows, turbulence model, rows per band): the smallest and largest rows of
# the range, rows that fill their bands or miss one
SHAPES = [(957, 150, 3, 12), (1024, 145, 3, 12), (1024, 192, 3, 12), (700, 200, 2, 16), (1024, 256, 2, 16),
          (560, 193, 3, 16), (1024, 256, 3, 16), (1024, 253, 0, 16)]


def _case(ni, rows, turb):
    bl = grids.flat_plate(ni + 1, rows + 1, first=2e-3, ratio=1.0 + 2.0 / rows)
    kw = dict(Ma=0.4, Re=1e4 if turb == 0 else 1e6, If_viscous=1, Iflag_turbulence_model=turb, Iflag_flux=6,
              Iflag_Scheme=5, CFL=5.0, Time_Method=0, P_outlet=1.0 / (1.4 * 0.16))
    if turb == 3:
        kw.update(Kt_inf=1e-6, Wt_inf=1e-2)
    return Params(**kw), bl


def _shape(monkeypatch, band):
    monkeypatch.setenv("EC2D_LUSGS_CLUSTER", "0")
    monkeypatch.setenv("EC2D_LUSGS_LANES", "0")
    monkeypatch.setenv("EC2D_LUSGS_ROWS", str(band))


@pytest.mark.parametrize("ni,rows,turb,band", SHAPES)
def test_long_rows(gpu_lib, monkeypatch, ni, rows, turb, band):
    _shape(monkeypatch, band)
    p, bl = _case(ni, rows, turb)
    nv, nx, ny = p.nvar(), ni + 1, rows + 1
    orc, g = make_oracle(p, bl, threads=16), make_gpu(p, bl)
    orc.init_flow(), g.init_flow()
    perturb_state(orc, amp=0.01, seed=ni + rows)
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


def test_band_edge_wait_runs_out(gpu_lib, monkeypatch):
    _shape(monkeypatch, 12)
    monkeypatch.setenv("EC2D_TEST_SILENT_BAND_EDGE", "1")
    g = make_gpu(*_case(960, 140, 3))
    g.init_flow()
    g.step(1)
    with pytest.raises(gpu.EC2DError) as e:
        g.norms()
    assert e.value.code == 4 and g.status()[0] == 4
    g.sync()
    g.close()


def _sweep_ms(ni, rows, turb):
    g = make_gpu(*_case(ni, rows, turb))
    g.init_flow()
    g.step(1)
    best = np.inf
    for _ in range(3):
        g.kernel_timing(True)
        g.step(3)
        t = g.kernel_times()
        best = min(best, t[("k_lusgs_sweep", 1)][2] / 3)
    g.close()
    return best


# a plane of the pull form takes some 2.7 times one of the push form, with one lane per
# row 4 to 8 times
@pytest.mark.parametrize("ni,rows,turb,band,fits", [(957, 150, 3, 12, 956), (700, 200, 2, 16, 660),
                                                    (1024, 256, 2, 16, 660), (1024, 256, 3, 16, 550)])
def test_long_rows_keep_eight_lanes(gpu_lib, monkeypatch, ni, rows, turb, band, fits):
    _shape(monkeypatch, band)
    planes = (ni + rows) / (fits + rows)
    assert _sweep_ms(ni, rows, turb) <= 3.5 * planes * _sweep_ms(fits, rows, turb)
