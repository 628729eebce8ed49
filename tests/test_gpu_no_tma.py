"""Vorticity tiles without tensor maps (OQG_NO_TMA=1, or a driver that cannot
encode them) come by cp.async: a step of a box or a channel created so, with
ragged last tiles and values on every wall, against the oracle within the parity
contract (1e-12 in FP64, 1e-5 in FP32 storage)."""
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


def _basin(nxp, nyp, cyclic, precision):
    return Basin(nxp=nxp, nyp=nyp, dx=2e4, dy=2e4, h=[350.0, 750.0, 2900.0], gp=[0.05, 0.025], ah2=[10.0] * 3,
                 ah4=[2e10] * 3, cyclic=cyclic, dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else 3, bcco=1.0,
                 precision=precision)


def _state(b):
    """A smooth p and pm that differ from wall to wall (a channel's are periodic), and a wekp."""
    x = np.linspace(0, 2 * np.pi if b.cyclic else 2.0, b.nxp)
    y = np.linspace(0, 2.0, b.nyp)[:, None]
    wave = (lambda k: np.cos(x + k)) if b.cyclic else (lambda k: np.cos((1 + k) * x + 0.3))
    p = np.stack([0.3 * wave(k) * np.cos((1 + 0.5 * k) * y + 0.2) for k in range(b.nl)])
    pm = np.stack([0.3 * wave(k + 0.1) * np.cos((1 + 0.4 * k) * y + 0.2) for k in range(b.nl)])
    if b.cyclic:
        p[..., -1], pm[..., -1] = p[..., 0], pm[..., 0]
    return p, pm, 1e-6 * np.cos(y) * np.cos(x)


def _check(got, b, tol):
    p, pm, w = _state(b)
    o = oracle.Oracle(b)
    o.set_state(p, pm)
    o.set_forcing(w, None, 0.0, 0.0)
    o.step(600.0, 2)
    for name, a, r in zip(("p", "pm", "q", "qm"), got, o.get_state()):
        assert rel_l2(a, r) <= tol, name
    o.close()


def _step(g, b):
    p, pm, w = _state(b)
    g.set_state(p, pm)
    g.set_forcing(w, None, 0.0, 0.0)
    g.step(600.0, 2)
    return g.get_state()


# one CTA per layer, double CTAs, plain CTAs; last tiles of 21, 3 and 1 columns;
# one tile that holds both walls
@pytest.mark.parametrize("nxp,nyp", [(81, 101), (181, 277), (181, 301), (61, 17), (17, 33), (5, 5), (241, 330)])
@pytest.mark.parametrize("cyclic", [False, True], ids=["box", "channel"])
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (OQG_MIXED, 1e-5)], ids=["fp64", "fp32"])
def test_step_without_tensor_maps(monkeypatch, nxp, nyp, cyclic, precision, tol):
    monkeypatch.setenv("OQG_NO_TMA", "1")
    b = _basin(nxp, nyp, cyclic, precision)
    for rows in (8, 12, 16):
        g = QG(b)
        g.set_tile_rows(rows)
        _check(_step(g, b), b, tol)
        g.close()


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (OQG_MIXED, 1e-5)], ids=["fp64", "fp32"])
def test_ensemble_without_tensor_maps(monkeypatch, precision, tol):
    monkeypatch.setenv("OQG_NO_TMA", "1")
    bs = [_basin(nxp, nyp, False, precision) for nxp, nyp in ((81, 101), (65, 33), (37, 61))]
    e = Ensemble(bs)
    for i, b in enumerate(bs):
        p, pm, w = _state(b)
        e.set_state(i, p, pm)
        e.set_forcing(i, w)
    e.step(600.0, 2)
    e.sync()
    for i, b in enumerate(bs):
        _check(e.get_state(i), b, tol)
    e.close()


def test_channel_retiles_without_tensor_maps(monkeypatch):
    """A channel created with tensor maps takes another tile height, alone and in
    an ensemble's tuner, where they can no longer be encoded."""
    b = _basin(181, 101, True, 0)
    monkeypatch.delenv("OQG_NO_TMA", raising=False)
    g, e = QG(b), Ensemble([b, b])
    p, pm, w = _state(b)
    for i in range(2):
        e.set_state(i, p, pm)
        e.set_forcing(i, w)
    monkeypatch.setenv("OQG_NO_TMA", "1")
    for rows in (12, 8, 16):
        g.set_tile_rows(rows)
    _check(_step(g, b), b, 1e-12)
    e.autotune(600.0, 2)
    e.step(600.0, 2)
    e.sync()
    for i in range(2):
        _check(e.get_state(i), b, 1e-12)
    g.close()
    e.close()
