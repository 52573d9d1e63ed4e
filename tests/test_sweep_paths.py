"""Paths of the kernels that the small parity cases do not reach, each bit for bit against the oracle:
the tiled tracer sweep in chunks of tile columns (more tiles than fit on the GPU), both sweeps on
mixing ratios that fall through the subnormal range (exact ties of the divisions included) and on a
grid outside the range of the fast division (every tile and sweep repeated with IEEE division); the
substep, radiation and column solve at every strip width, on the last partial strip, and the column
solve's and the substep's repeat with IEEE division; ensembles of more columns than column strips take."""
import numpy as np
import pytest

from moist2d_b200 import abi, model
from moist2d_b200.init import uniform
from moist2d_b200.params import Params, State, exchange_halo
from oracle import bind
from states import compare, perturb, small_case
from test_zz_no_alloc import _call, _columns

pytestmark = pytest.mark.gpu

SWEEPS = [0, abi.MOIST_FLAG_TRACER_STREAM]
IDS = ["tiles", "stream"]


def _both(p, s, flags, phys=None, tri64=True):
    """One RK stage on the device and by the oracle."""
    z = [np.zeros((p.ka, p.ia), dtype=p.T, order="F") for _ in range(6)] if phys is None else phys
    a, b = s.copy(), s.copy()
    model.compute_step(z, a, s, p, float(p.dt) / 3, 2, flags=flags)
    bind.compute_step(z, b, s, p, float(p.dt) / 3, 2, tri64=tri64)
    compare(a, b, p)


@pytest.mark.parametrize("T,nx,nz", [(np.float32, 1301, 250), (np.float64, 1411, 99)])
def test_tiles_in_chunks(T, nx, nz):
    p, s = small_case(T, nx, nz)
    _both(p, s, 0)


@pytest.mark.parametrize("flags", SWEEPS, ids=IDS)
@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_mixing_ratios_through_the_subnormal_range(T, flags):
    p, s = small_case(T, 70, 37)
    lo = -46.0 if T is np.float32 else -324.0
    u = uniform(3, 21, np.arange(p.Nx * p.Nz)).reshape(p.Nz, p.Nx)
    for j, f in enumerate((s.rho_qc, s.rho_qr)):
        # smooth tails along x and random values, from 1e-3 down past the smallest subnormal
        x = np.linspace(-3.0, lo, p.Nx)[None, :] if j == 0 else -3.0 + (lo + 3.0) * u
        f[:, p.is_ - 1:p.ie] = (10.0 ** np.broadcast_to(x, u.shape)).astype(T)
        exchange_halo(f, p)
    _both(p, s, flags)


@pytest.mark.parametrize("flags", SWEEPS, ids=IDS)
@pytest.mark.parametrize("T,dx", [(np.float32, 3e12), (np.float64, 1e31)])
def test_grid_outside_the_fast_divisions_range(T, dx, flags):
    p, s = small_case(T, 45, 21, Lx=45 * dx)
    assert float(p.dx) > (2.0 ** 40 if T is np.float32 else 2.0 ** 100)
    _both(p, s, flags)


@pytest.mark.parametrize("T,flags", [(np.float32, 0), (np.float32, abi.MOIST_FLAG_TRI_NATIVE), (np.float64, 0)],
                         ids=["f32-tri64", "f32-tri32", "f64"])
@pytest.mark.parametrize("nx,nz", [(299, 3), (601, 6), (1187, 9), (1187, 2), (1190, 66)])
def test_substep_strips(T, flags, nx, nz):
    p, s = small_case(T, nx, nz)
    _both(p, s, flags, tri64=not flags)


def test_substep_quotients_below_the_checked_range():
    """Numerators of 1e-295 are refused by the exactness check: the block repeats with IEEE division."""
    p, s = small_case(np.float64, 37, 21)
    s.rho_w[:] = 0.0
    z = [np.zeros((p.ka, p.ia), order="F") for _ in range(6)]
    a, b = s.copy(), s.copy()
    model.compute_step(z, a, s, p, 3e-295, 2)
    bind.compute_step(z, b, s, p, 3e-295, 2)
    w = np.abs(b.rho_w[:, p.is_ - 1:p.ie])
    assert 0.0 < np.max(w) < 1e-290
    compare(a, b, p)


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("nx,nz", [(37, 9), (299, 5), (601, 33), (1187, 12)])
def test_radiation_strips(T, nx, nz):
    p, s = small_case(T, nx, nz)
    a, b = s.copy(), s.copy()
    model.gray_radiation(a, p)
    bind.gray_radiation(b, p)
    i = slice(p.is_ - 1, p.ie)
    assert np.array_equal(a.d_rho_theta_rd[:, i], b.d_rho_theta_rd[:, i])


@pytest.mark.parametrize("nz,ncols,dt", [(64, 1185, 0.25), (37, 611, 0.25), (300, 299, 0.25), (1024, 3, 0.25),
                                         (33, 41, 3e8)])
@pytest.mark.parametrize("T,flags", [(np.float32, 0), (np.float32, abi.MOIST_FLAG_TRI_NATIVE), (np.float64, 0)],
                         ids=["f32-tri64", "f32-tri32", "f64"])
def test_column_solve_strips(T, flags, nz, ncols, dt):
    import torch
    p, (w, dw, th, r2) = _columns(T, nz, ncols, 5)
    tri64 = T is np.float64 or not (flags & abi.MOIST_FLAG_TRI_NATIVE)
    want = w.copy()
    for j in range(ncols):
        col = want[j].copy()
        bind.implicit_correction(col, dw[j].copy(), th[j].copy(), r2[j].copy(), T(dt), p, tri64=tri64)
        want[j] = col
    dev = [torch.from_numpy(a).cuda() for a in (w, dw, th, r2)]
    rc, msg = _call(p, flags, ncols, dev, T(dt))
    assert rc == abi.MOIST_OK, msg
    torch.cuda.synchronize()
    assert np.array_equal(dev[0].cpu().numpy(), want)


@pytest.mark.parametrize("nz,ncols", [(2, 1), (3, 131), (4, 9600), (5, 9472), (5, 9473), (7, 10001), (10, 9999), (11, 9999)])
@pytest.mark.parametrize("T,flags", [(np.float32, 0), (np.float32, abi.MOIST_FLAG_TRI_NATIVE), (np.float64, 0)],
                         ids=["f32-tri64", "f32-tri32", "f64"])
def test_column_solve_of_few_levels(T, flags, nz, ncols):
    """Both forms of the solve around the lines between them; 41 different columns, repeated."""
    import torch
    m = min(41, ncols)
    p, arrays = _columns(T, nz, m, 6)
    tri64 = T is np.float64 or not (flags & abi.MOIST_FLAG_TRI_NATIVE)
    w, dw, th, r2 = [np.ascontiguousarray(np.resize(a, (ncols, nz))) for a in arrays]
    want = arrays[0].copy()
    for j in range(m):
        col = want[j].copy()
        bind.implicit_correction(col, dw[j].copy(), th[j].copy(), r2[j].copy(), T(0.25), p, tri64=tri64)
        want[j] = col
    dev = [torch.from_numpy(a).cuda() for a in (w, dw, th, r2)]
    rc, msg = _call(p, flags, ncols, dev, T(0.25))
    assert rc == abi.MOIST_OK, msg
    torch.cuda.synchronize()
    assert np.array_equal(dev[0].cpu().numpy(), np.resize(want, (ncols, nz)))


@pytest.mark.parametrize("T,flags", [(np.float32, 0), (np.float32, abi.MOIST_FLAG_TRI_NATIVE), (np.float64, 0)],
                         ids=["f32-tri64", "f32-tri32", "f64"])
@pytest.mark.parametrize("shapes", [[(6501, 9), (6397, 12), (6303, 7)],
                                    [(3905, 7), (3841, 12), (3839, 5), (3840, 9), (3907, 17)]], ids=["3", "5"])
def test_ensembles_of_many_columns(T, flags, shapes):
    """More columns than the column strips take by default, in one chain of members and in several."""
    mem = [small_case(T, nx, nz) for nx, nz in shapes]
    with model.Ensemble([p for p, _ in mem], flags) as e:
        for i, (_, s) in enumerate(mem):
            e.upload(i, s)
        e.step(3)
        got = [e.download(i, s.copy()) for i, (_, s) in enumerate(mem)]
    for (p, s), g in zip(mem, got):
        compare(g, model.rk3_step(s.copy(), p, 3, flags=flags), p)


@pytest.mark.parametrize("T,flags,nzs", [(np.float32, 0, (184, 185)), (np.float32, abi.MOIST_FLAG_TRI_NATIVE, (256, 129)),
                                         (np.float64, 0, (157, 158))], ids=["f32-tri64", "f32-tri32", "f64"])
@pytest.mark.parametrize("nx", [395, 150, 50])
def test_ensemble_strips_at_the_most_shared_memory(T, flags, nzs, nx):
    """Column strips of the widest width, the last level count that has it and the first that has not, with
    columns enough for it and for half and a quarter of it."""
    mem = [small_case(T, nx, nz, dz0=50.0, H=50.0 * nz * 1.02) for nz in nzs]
    with model.Ensemble([p for p, _ in mem], flags) as e:
        for i, (_, s) in enumerate(mem):
            e.upload(i, s)
        e.step(2)
        got = [e.download(i, s.copy()) for i, (_, s) in enumerate(mem)]
    for (p, s), g in zip(mem, got):
        o = s.copy()
        bind.rk3_step(o, p, 2, tri64=not flags)
        compare(g, o, p)
