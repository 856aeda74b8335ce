"""Constant mass flux over many steps: the mean is subtracted from the increment, not from the advanced field, so that the
velocity is rounded once a substep and a laminar profile does not drift."""
import numpy as np
import pytest

from chapsim2_b200 import config as C
from chapsim2_b200 import solver as S
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,dt", [((8, 24, 8), 0.05), ((16, 48, 16), 0.01)])
def test_laminar_profile(nc, dt):
    cfg = C.channel(nc=nc, iacc=C.IACCU_CD2, dt=dt)
    f = [np.zeros(s) for s in cfg.shapes()]
    f[0][:] = 1.5 * (1 - np.asarray(C.geometry(cfg)["yc"])[None, :, None] ** 2)
    o, g = po.Oracle(cfg), S.Solver(cfg)
    for s in (o, g):
        s.set_fields(*f)
        s.substep(0)
    for n in range(1, 5):
        for _ in range(250):
            for isub in (1, 2, 3):
                o.substep(isub)
        g.step(250)
        # Both round u' = u + (m - bulk) alike, except where the increments' own round-off, 1e-4 of an ulp of u and
        # less, tips a tie: a few ulp.  (u + m) - bulk rounds every row the same way substep after substep: 10 to 30 ulp.
        err = np.abs(g.get_fields()[0] - o.get_fields()[0]).max()
        assert err <= 5 * 1.5 * 2.0 ** -52, (n, err)
    g.close()
