"""Handles and ensembles made, forced (with entrainment, whose buffer is made on
its first use) and stepped in quick succession, each call right after the one
before: every one ends in the same state as the first, bit for bit."""
import numpy as np
import pytest

from openqg_b200.core import QG, Ensemble
from openqg_b200.params import OQG_MIXED, Basin

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


def _basin(nxp, nyp, cyclic, precision):
    y, x = np.linspace(0, 3, nyp)[:, None], np.linspace(0, 2 * np.pi, nxp)
    return Basin(nxp=nxp, nyp=nyp, dx=2e4, dy=2e4, h=[350.0, 750.0, 2900.0], gp=[0.05, 0.025], ah4=[2e10] * 3,
                 ah2=[0.0] * 3, cyclic=cyclic, dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else 3,
                 bcco=1.0 if cyclic else 1e20, precision=precision, ddyn=1e-6 * np.cos(x) * np.sin(y))


def _fields(b):
    y, x = np.linspace(0, np.pi, b.nyp)[:, None], np.linspace(0, 2 * np.pi, b.nxp)
    p = np.stack([0.1 * np.sin((k + 1) * y) * np.sin(x) for k in range(b.nl)])
    e = 1e-7 * np.stack([np.cos(k * y) * np.cos(x) for k in range(b.nl - 1)])
    return p, 1e-6 * np.cos(y) * np.cos(x), e


@pytest.mark.parametrize("cyclic", [False, True], ids=["box", "channel"])
@pytest.mark.parametrize("precision", [0, OQG_MIXED], ids=["fp64", "fp32"])
def test_handles_in_quick_succession(cyclic, precision):
    b = _basin(28, 33, cyclic, precision)
    p, w, e = _fields(b)
    first = None
    for _ in range(150):
        g = QG(b)
        g.set_state(p, 0.9 * p)
        g.set_forcing(w, e, 0.01, -0.01)
        g.step(300.0, 1)
        got = g.get_state()
        g.close()
        first = first or got
        assert all(np.array_equal(a, r) for a, r in zip(got, first))


@pytest.mark.parametrize("cyclic", [False, True], ids=["box", "channel"])
def test_ensembles_in_quick_succession(cyclic):
    bs = [_basin(n, m, cyclic, 0) for n, m in ((17, 9), (25, 33), (28, 102), (97, 8), (33, 17))]
    first = None
    for _ in range(60):
        e = Ensemble(bs)
        for i, b in enumerate(bs):
            p, w, ent = _fields(b)
            e.set_state(i, p, 0.9 * p)
            e.set_forcing(i, w, ent, 0.01, -0.01)
        e.step(300.0, 2)
        got = [a for i in range(len(bs)) for a in e.get_state(i)]
        e.close()
        first = first or got
        assert all(np.array_equal(a, r) for a, r in zip(got, first))
