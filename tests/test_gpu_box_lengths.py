"""The closed box's x-transform (DST-I by the pruned FFT of the odd extension)
at the lengths where its plan changes: outer radix 16, 8, 4 and 2, the
compile-time lengths and their neighbours, subsequences of length 1, 3 and 5
factors, odd and even numbers of rows, the smallest grid.  The Helmholtz solve
of every mode against the oracle, within the parity contract's 1e-13, and an
FP32 step within its 1e-5."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG, Ensemble
from openqg_b200.params import OQG_MIXED, Basin
from tests.qg_numpy import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


def _box(nxp, nyp, precision=0):
    return Basin(nxp=nxp, nyp=nyp, dx=1e4, dy=1e4, h=[350.0, 750.0, 2900.0], gp=[0.05, 0.025], ah4=[1e9] * 3,
                 ah2=[0.0] * 3, precision=precision)


# M = 2 (nxp - 1) = 8, 10, 12, 16, 18, 20, 24, 30, 32, 40, 48, 50, 54, 64, 72, 80, 96, 128, 150, 160, 162, 192, 240,
# 256, 270, 384, 486, 512, 720, 1000, 1024, 1152
LENGTHS = [5, 6, 7, 9, 10, 11, 13, 16, 17, 21, 25, 26, 28, 33, 37, 41, 49, 65, 76, 81, 82, 97, 121, 129, 136, 193, 244,
           257, 361, 501, 513, 577]


@pytest.mark.parametrize("nxp", LENGTHS)
def test_box_solve_at_every_plan(nxp):
    b = _box(nxp, 12 + nxp % 3)
    g, o = QG(b), oracle.Oracle(b)
    rhs = np.random.default_rng(nxp).standard_normal(b.shape2)
    for m in range(1, b.nl + 1):
        assert rel_l2(g.solve_inhomog_eqn(m, rhs), o.solve_inhomog(m, rhs)) <= 1e-13
    g.close()
    o.close()


@pytest.mark.parametrize("nxp", [6, 17, 37, 76, 97, 193, 361, 513])
def test_box_fp32_step_at_plans(nxp):
    b = _box(nxp, 13, OQG_MIXED)
    x, y = np.linspace(0, 1, nxp), np.linspace(0, 1, 13)
    p = 0.1 * np.stack([np.outer(np.sin(np.pi * k * y), np.sin(np.pi * x)) for k in (1, 2, 1)])
    g, o = QG(b), oracle.Oracle(b)
    for h in (g, o):
        h.set_state(p, p)
        h.set_forcing(np.zeros(b.shape2), None, 0.0, 0.0)
        h.step(600.0, 1)
    assert rel_l2(g.get_state()[0], o.get_state()[0]) <= 1e-5
    g.close()
    o.close()


def test_ensemble_of_plans_equals_single_handles():
    """Members of compile-time and any-length plans in one launch."""
    bs = [_box(n, 23) for n in (65, 76, 129, 37, 193, 97, 361)]
    e = Ensemble(bs)
    rng = np.random.default_rng(3)
    hs = []
    for i, b in enumerate(bs):
        p = np.zeros(b.shape3)
        p[:, 1:-1, 1:-1] = 0.01 * rng.standard_normal((b.nl, b.nyp - 2, b.nxp - 2))
        h = QG(b)
        for s in (lambda *a: e.set_state(i, *a), h.set_state):
            s(p, p)
        e.set_forcing(i, np.zeros(b.shape2))
        h.set_forcing(np.zeros(b.shape2))
        hs.append(h)
    e.step(300.0, 2)
    e.sync()
    for i, h in enumerate(hs):
        h.step(300.0, 2)
        for a, r in zip(e.get_state(i), h.get_state()):
            assert rel_l2(a, r) <= 1e-13
        h.close()
    e.close()
