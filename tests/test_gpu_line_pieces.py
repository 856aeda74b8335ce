"""Compact line operators with the line in register pieces: against the oracle at the lengths where
the pieces change (one piece, a short last piece, 8 to 16 and 16 to 24 rows per piece, the longest line
and one beyond it, which runs the tile kernel) with line counts off the 32 of a CTA, and whole substeps,
which form every input expression and store mode, against the oracle's."""
import numpy as np
import pytest
import scipy.fft as sf

from chapsim2_b200 import config as C
from chapsim2_b200 import initial as I
from chapsim2_b200 import solver as S
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _check(cfg, d, bcs, tol):
    o, g = po.Oracle(cfg), S.Solver(cfg)
    rng = np.random.default_rng(11)
    for fam in (2, 3, 4, 5):
        nin3 = list(cfg.nc)
        if fam in (3, 5):
            nin3[d] = cfg.np_[d]
        fi = rng.standard_normal((nin3[2], nin3[1], nin3[0]))
        fb = rng.standard_normal({0: (nin3[2], nin3[1], 4), 1: (nin3[2], 4, nin3[0]), 2: (4, nin3[1], nin3[0])}[d])
        for ibc in bcs:
            for has in ((False, True) if d == 1 else (False,)):
                ref = o.op3d(d, fam, ibc, fi, fb if has else None)
                got = g.op3d(d, fam, ibc, fi, fb if has else None)
                # operators and their inverses have O(1) condition (diagonally dominant lines): a few
                # hundred roundings of 1e-16 relative to the largest value
                assert np.abs(ref - got).max() <= tol * max(1.0, np.abs(ref).max()), (d, fam, ibc, has)
    g.close()


@pytest.mark.parametrize("acc", [3, 4])
@pytest.mark.parametrize("n", [8, 12, 54, 64, 128, 144, 256, 288, 384, 432])
def test_periodic_lines(acc, n):
    for d in (0, 2):
        nc = [18, 9, 12]
        nc[d] = n
        cfg = C.channel(nc=tuple(nc), iacc=acc)
        _check(cfg, d, [(1, 1)], 1e-13 * n)


@pytest.mark.parametrize("acc", [3, 4])
@pytest.mark.parametrize("n", [8, 15, 16, 17, 63, 127, 128, 129, 255, 256, 383, 384, 385])
def test_wall_lines(acc, n):
    # cells n, points n + 1: the input and the output may need different numbers of pieces
    cfg = C.channel(nc=(18, n, 12), iacc=acc)
    _check(cfg, 1, [(4, 4), (5, 5), (6, 6), (4, 5)], 1e-13 * n)


@pytest.mark.parametrize("precision", [S.CHS_FP64, S.CHS_MIXED])
@pytest.mark.parametrize("case,nc", [("tgv", 54), ("fmd", (72, 54, 48)), ("heated", (48, 33, 54)),
                                     ("heated", (144, 129, 18))])
def test_substep(case, nc, precision):
    tc = None
    if case == "tgv":
        cfg = C.taylor_green(nc, iacc=4, dt=1e-3)
        f = I.taylor_green_fields(cfg)
    elif case == "fmd":
        cfg = C.channel(nc=nc, iacc=4, dt=2e-3, rstret=0.25, ifft=C.FFT_2DECOMP_3DFFT)
        f = I.channel_fields(cfg)
    else:
        cfg, tc = C.heated_channel(nc=nc, iacc=3, dt=1e-3)
        f = I.channel_fields(cfg)
    g, o = S.Solver(cfg, precision=precision), po.Oracle(cfg)
    for s in (g, o):
        s.set_fields(*f)
        if tc is not None:
            s.thermo_init(tc)
        for isub in (0, 1, 2, 3):
            s.substep(isub)
    got, ref = g.get_fields()[:4], o.get_fields()[:4]
    q = max(np.abs(a).max() for a in ref[:3])
    # four substeps of round-off: eps times the velocity scale, and for the pressure times 1/(dt dx) of
    # its source over the Laplacian's 1/dx^2, i.e. dx/dt < 500
    eps = 1e-12 if precision == S.CHS_FP64 else 1e-5
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() <= eps * q
    assert np.abs(got[3] - ref[3]).max() <= 500 * eps * q
    if tc is not None:
        assert np.abs(g.get_thermo()["T"] - o.get_thermo()["T"]).max() <= eps
    g.close()


@pytest.mark.parametrize("acc,bound", [(3, (1.4, 1.4)), (4, (1.8, 1.75))])
@pytest.mark.parametrize("n", [64, 128, 144, 256, 288, 384])
def test_error(n, acc, bound):
    """Error of the x operators against their Fourier symbol in extended precision, rms in units of 2^-53: a right-hand side
    of four roundings and the sweeps' two, one and one, as one thread sweeping the whole line makes them, come to 1.3 and
    1.15 (CP4 derivative, interpolation) and 1.7 and 1.65 (CP6).  Corrected rows instead of swept ones, and constants
    rounded once more, made it 1.74 and 1.26, 1.76 and 1.7."""
    L = np.longdouble
    cfg = C.channel(nc=(n, 16, 16), iacc=acc)
    g = S.Solver(cfg)
    for fam in (2, 3, 4, 5):
        f = np.random.default_rng(n + fam).standard_normal((16, 16, n))
        got = g.op3d(0, fam, (1, 1), f, None)
        p = S.plan_inspect(cfg, 0, fam, (1, 1), False)
        at = [np.roll(f.astype(L), -o, axis=2) for o in p["off"]]
        r = (L(p["r1"]) * (at[0] + L(p["sgn"]) * at[1]) + L(p["r2"]) * (at[2] + L(p["sgn"]) * at[3])) * L(p["dd"])
        # the left-hand side's off-diagonal is the plan's a
        w = 1 + 2 * L(p["a"][3]) * np.cos(2 * L(np.pi) * np.arange(n // 2 + 1).astype(L) / n)
        ref = sf.irfft(sf.rfft(r, axis=2) / w, n=n, axis=2)
        err = np.linalg.norm((got - ref).astype(float)) / np.linalg.norm(ref.astype(float))
        assert err <= bound[fam > 3] * 2.0 ** -53, (fam, err * 2.0 ** 53)
    g.close()
