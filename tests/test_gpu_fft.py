"""Transforms of the Poisson solvers at every shape of their stage plan (one to three register stages with each
radix, lengths beyond them, odd lengths, ragged line counts) through the periodic solver against
numpy's FFT, the y solve at the ends of its piece sizes, and the FP32 spectrum of the mixed form against the
FP64 path."""
import numpy as np
import pytest
import scipy.fft as sf

from chapsim2_b200 import config as C
from chapsim2_b200 import initial as I
from chapsim2_b200 import solver as S
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

LENGTHS = [8, 9, 12, 16, 18, 24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128, 144, 162, 192, 216, 243, 256, 288, 324,
           384, 432, 486, 512, 576, 648, 729, 768, 1024]


@pytest.mark.parametrize("n", LENGTHS)
def test_lengths(n):
    for axis in range(3):
        nc = [18, 9, 12]
        nc[axis] = n
        cfg = C.taylor_green(16, iacc=C.IACCU_CD2)
        cfg.nc = tuple(nc)
        g = S.Solver(cfg)
        rhs = np.random.default_rng(n).standard_normal((nc[2], nc[1], nc[0]))
        got = g.solve_fft_poisson(rhs)
        g.close()
        h = (cfg.lxx / nc[0], (cfg.lyt - cfg.lyb) / nc[1], cfg.lzz / nc[2])
        k2 = [(2.0 / h[d] * np.sin(np.pi * np.arange(nc[d]) / nc[d])) ** 2 for d in range(3)]
        k2 = k2[2][:, None, None] + k2[1][None, :, None] + k2[0][None, None, :]
        f = np.fft.fftn(rhs)
        k2[0, 0, 0] = 1.0
        f /= -k2
        f[0, 0, 0] = 0.0
        ref = np.fft.ifftn(f).real
        # error growth of an FFT is O(eps log n); five passes over values of the result's size
        assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max(), axis


@pytest.mark.parametrize("nc", [(24, 24, 24), (64, 64, 64), (96, 9, 96), (216, 9, 216), (216, 216, 8), (144, 9, 108),
                                (324, 9, 54)])
def test_error(nc):
    """Residual of the periodic solver in extended precision.  A transform of length n whose factors are rounded once errs
    by 0.55 to 0.66 sqrt(log2 n) units of 2^-53 (rms); three forward and three backward add up in quadrature, the
    wavenumbers and the division bring the 0.6 to 0.73 at most.  Factors that err systematically took it to 0.79 (24) to
    1.1 (324)."""
    L = np.longdouble
    cfg = C.taylor_green(16, iacc=C.IACCU_CD2)
    cfg.nc = nc
    h = (cfg.lxx / nc[0], (cfg.lyt - cfg.lyb) / nc[1], cfg.lzz / nc[2])
    k2 = [(L(2) / L(h[d]) * np.sin(L(np.pi) * np.arange(nc[d]).astype(L) / nc[d])) ** 2 for d in range(3)]
    k2 = k2[2][:, None, None] + k2[1][None, :, None] + k2[0][None, None, :nc[0] // 2 + 1]
    # the right-hand side of a white solution, so that no mode stands out
    phi = np.random.default_rng(3).standard_normal(nc[::-1])
    rhs = sf.irfftn(sf.rfftn(phi) * -k2.astype(float), s=phi.shape)
    g = S.Solver(cfg)
    got = g.solve_fft_poisson(rhs)
    g.close()
    f = sf.rfftn(rhs.astype(L))
    e = sf.rfftn(got.astype(L)) * -k2 - f
    e[0, 0, 0] = 0.0
    norm = lambda a: np.linalg.norm(np.abs(a).astype(float).ravel())  # noqa: E731
    assert norm(e) <= 0.78 * np.sqrt(2 * np.log2(np.array(nc)).sum()) * 2.0 ** -53 * norm(f)


@pytest.mark.parametrize("ny", [8, 9, 15, 16, 17, 127, 128, 129, 160, 255, 256, 257])
def test_y_solve(ny):
    cfg = C.channel(nc=(18, ny, 12), iacc=1)
    o, g = po.Oracle(cfg), S.Solver(cfg)
    rhs = np.random.default_rng(ny).standard_normal(o.shape_ccc)
    rhs -= rhs.mean(axis=(0, 2), keepdims=True)
    # the mean mode's last pivot is zero up to round-off, so its constant is round-off too where it is not pinned
    ref, got = [a - a.mean() for a in (o.poisson(rhs), g.solve_fft_poisson(rhs))]
    assert np.abs(ref - got).max() / np.abs(ref).max() < 1e-11
    g.close()


@pytest.mark.parametrize("ny", [8, 9, 33, 128, 129, 144, 160, 161, 256])
def test_y_solve_mean_mode(ny):
    # the singular column with a mean in every row, through 8- and 16-row pieces and the lines kernel; uniform rows leave
    # its last pivot exactly zero at some sizes and at round-off in others: the constant is free in the latter
    for istret in (C.ISTRET_NO, C.ISTRET_2SIDES):
        cfg = C.channel(nc=(18, ny, 12), iacc=1, istret=istret)
        o, g = po.Oracle(cfg), S.Solver(cfg)
        rhs = np.random.default_rng(ny).standard_normal(o.shape_ccc)
        geo = C.geometry(cfg)
        dy = geo["h"][1] / geo["mpcc"] if cfg.stretch_y else np.full(ny, geo["h"][1])
        rhs -= (rhs.mean(axis=(0, 2)) * dy).sum() / dy.sum()  # solvable
        assert np.abs(rhs.mean(axis=(0, 2))).max() > 1e-3
        ref, got = [a - a.mean() for a in (o.poisson(rhs), g.solve_fft_poisson(rhs))]
        assert np.abs(ref - got).max() / np.abs(ref).max() < 1e-11, istret
        g.close()


@pytest.mark.parametrize("nc", [(8, 9, 16), (54, 17, 108), (162, 24, 8), (18, 130, 256), (384, 12, 24)])
def test_fp32_spectrum(nc):
    cfg = C.channel(nc=nc, iacc=1, dt=1e-3)
    f = I.channel_fields(cfg)
    res = []
    for prec in (S.CHS_FP64, S.CHS_MIXED):
        g = S.Solver(cfg, precision=prec)
        g.set_fields(*f)
        g.Solve_momentum_eq(0)
        g.step(1)
        res.append(g.get_fields())
        g.close()
    # eps of FP32 times the velocity scale; the pressure's source is a velocity difference over the spacing
    # and dt, and its inverse Laplacian gains a spacing squared: eps q h / dt for each of four substeps
    q = max(np.abs(a).max() for a in res[0][:3])
    for a, b in zip(res[1][:3], res[0][:3]):
        assert np.abs(a - b).max() <= 1e-5 * q
    h = max(cfg.lxx / nc[0], cfg.lzz / nc[2])
    assert np.abs(res[1][3] - res[0][3]).max() <= 4 * 2.0 ** -23 * q * h / cfg.dt
