"""Handles driven from several host threads: launches of one kernel with different shared-memory sizes (transforms of 256 and
192 points, compact lines likewise, both above the 48 KB that need no opt-in) do not disturb each other."""
import threading

import numpy as np
import pytest
import torch

from chapsim2_b200 import config as C
from chapsim2_b200 import solver as S

pytestmark = pytest.mark.gpu


def _in_threads(work, items):
    errors = []

    def guarded(item):
        try:
            work(*item)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(i,)) for i in items]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_transforms():
    items = []
    for n in (256, 192):
        g = S.Solver(C.channel(nc=(8, 8, n), iacc=C.IACCU_CD2, dt=1e-3))
        rhs = np.random.default_rng(n).standard_normal((n, 8, 8))
        items.append((g, torch.zeros((n, 8, 8), dtype=torch.float64, device="cuda"), rhs, g.solve_fft_poisson(rhs)))
    torch.cuda.synchronize()

    def work(g, zero, rhs, ref):
        for _ in range(20000):
            rc = g.L.chs_poisson_solve_device(g.h, zero.data_ptr())
            assert rc == 0
        g.sync()
        assert np.array_equal(g.solve_fft_poisson(rhs), ref)

    _in_threads(work, items)
    for g, *_ in items:
        g.close()


def test_lines():
    items = []
    for n in (256, 192):
        g = S.Solver(C.channel(nc=(n, 8, 8), iacc=C.IACCU_CP6, dt=1e-3))
        f = np.random.default_rng(n).standard_normal((8, 8, n))
        items.append((g, f, g.op3d(0, 2, (1, 1), f, None)))

    def work(g, f, ref):
        for _ in range(1500):
            assert np.array_equal(g.op3d(0, 2, (1, 1), f, None), ref)

    _in_threads(work, items)
    for g, _, _ in items:
        g.close()
