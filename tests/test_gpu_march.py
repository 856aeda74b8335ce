"""The momentum march and the packed projection and divergence against the operator path at the shapes where their
tiles end (x tiles of 32, y tiles of 8, z runs, rows of one pair, odd nx), with walls at rest, moving walls (wall
planes that are not zero), free-slip walls (which the march does not take) and periodic y; the histories too, whose y
wall rows a kernel of their own writes."""
import numpy as np
import pytest

from chapsim2_b200 import config as C
from chapsim2_b200 import initial as I
from chapsim2_b200 import solver as S

pytestmark = pytest.mark.gpu


def _cfg(case, nc):
    tc = None
    if case == "heated":
        cfg, tc = C.heated_channel(nc=nc, iacc=C.IACCU_CD2, dt=0.002, t_ini=0.49)
    elif case == "box":
        cfg = C.taylor_green(16, iacc=C.IACCU_CD2, dt=2e-3)
        cfg.nc = nc
    else:
        cfg = C.channel(nc=nc, iacc=C.IACCU_CD2, dt=0.002)
        if case == "undriven":  # no mass-flux mean: the x field, too, is advanced by the momentum pass
            cfg.idriven = C.IDRVF_NO
        if case == "moving":
            cfg.fbcy_const[C.V_QX] = (0.3, -0.2)
            cfg.fbcy_const[C.V_QZ] = (-0.1, 0.4)
        elif case == "slip":
            cfg.nominal_bc[1, C.V_QX] = C.IBC_SYMMETRIC
            cfg.nominal_bc[1, C.V_QZ] = C.IBC_SYMMETRIC
    if case == "box":
        rng = np.random.default_rng(5)
        f = [rng.standard_normal(s) for s in cfg.shapes()]
        f[3][:] = 0.0
    else:
        f = I.channel_fields(cfg)
    return cfg, tc, f


def _start(cfg, tc, f, fused, precision):
    g = S.Solver(cfg, precision=precision)
    g.set_fusion(fused)
    g.set_fields(*f)
    if tc is not None:
        g.thermo_init(tc)
    return g


def _run(cfg, tc, f, fused, precision):
    g = _start(cfg, tc, f, fused, precision)
    for isub in (0, 1, 2, 3):
        g.substep(isub)
    hist = [g.download(k) for k in (S.CHS_MX_RHS0, S.CHS_MY_RHS0, S.CHS_MZ_RHS0)]
    g.step(1)
    out = list(g.get_fields()[:4])
    g.close()
    return out, hist


@pytest.mark.parametrize("precision", [S.CHS_FP64, S.CHS_MIXED])
@pytest.mark.parametrize("case,nc", [
    ("rest", (8, 8, 8)), ("rest", (32, 16, 16)), ("rest", (36, 17, 12)), ("rest", (64, 9, 54)), ("moving", (24, 15, 32)),
    ("moving", (96, 8, 18)), ("undriven", (24, 15, 32)), ("slip", (24, 16, 12)), ("heated", (8, 8, 8)),
    ("heated", (32, 24, 8)),
    ("heated", (54, 33, 16)), ("heated", (72, 31, 24)), ("box", (16, 8, 12)), ("box", (36, 18, 9)), ("box", (27, 12, 16)),
    ("box", (9, 27, 8))])
def test_fused_matches_operator_path(case, nc, precision):
    cfg, tc, f = _cfg(case, nc)
    (a, ha), (b, hb) = _run(cfg, tc, f, True, precision), _run(cfg, tc, f, False, precision)
    q = max(np.abs(x).max() for x in b[:3])
    # seven substeps of round-off of values of the velocity's size (a velocity difference over the smallest spacing in
    # the histories, over dt in the pressure's source)
    eps = 1e-13 if precision == S.CHS_FP64 else 2e-5
    for x, y in zip(a[:3], b[:3]):
        assert np.abs(x - y).max() <= 10 * eps * q
    for x, y in zip(ha, hb):
        assert np.abs(x - y).max() <= 10 * eps * max(1.0, np.abs(y).max())
    g = C.geometry(cfg)
    assert np.abs(a[3] - b[3]).max() <= 10 * eps * q * max(g["h"][0], g["h"][2], 1.0) / cfg.dt


def _flow_passes(cfg, tc, f):
    """Launches of the flow class in a substep: one momentum pass or three component passes, with walls the divergence,
    with variable properties the energy pass."""
    g = _start(cfg, tc, f, True, S.CHS_FP64)
    g.substep(0)
    n = sum(r["kind"] == 4 for r in g.profile_substep(1))
    g.close()
    return n - (not cfg.periodic_y) - (tc is not None)


@pytest.mark.parametrize("case,nc,passes", [("rest", (8, 8, 8), 1), ("rest", (36, 17, 12), 1), ("moving", (24, 15, 32), 1),
                                            ("heated", (32, 24, 8), 1), ("box", (16, 8, 12), 1), ("slip", (24, 16, 12), 3),
                                            ("box", (27, 12, 16), 3)])
def test_which_pass_runs(case, nc, passes):
    # the comparison above holds for either, so it does not show that the march runs where it should
    assert _flow_passes(*_cfg(case, nc)) == passes


def test_march_on_any_stretching():
    # the host recognises the march's operators by their weights, digit for digit
    rng = np.random.default_rng(1)
    for _ in range(40):
        ny, rst = int(rng.integers(8, 200)), float(rng.uniform(0.02, 0.4))
        cfg = C.channel(nc=(8, ny, 8), iacc=C.IACCU_CD2, dt=1e-4, rstret=rst, lxx=float(rng.uniform(2, 14)),
                        lzz=float(rng.uniform(1, 5)))
        assert _flow_passes(cfg, None, I.channel_fields(cfg)) == 1, (ny, rst)
