"""Channels of 2049 and 4097 points (2048- and 4096-point transforms, whose
modal rows leave shared memory): the inverse transform runs as a launch of its
own between two padded buffers, and its shared memory must hold both.  The
Helmholtz solve and a step against the oracle, within the parity contract."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG
from openqg_b200.params import OQG_MIXED, atmos_channel, double_gyre_tau, initial_psi
from tests.qg_numpy import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


@pytest.mark.parametrize("nxp,precision", [(2049, 0), (4097, 0), (2049, OQG_MIXED), (4097, OQG_MIXED)])
def test_wide_channel_solve_and_step(nxp, precision):
    b = atmos_channel(nxp, 33, dx=20e3, precision=precision)
    g, o = QG(b), oracle.Oracle(b)
    rhs = np.random.default_rng(1).standard_normal(b.shape2)
    rhs[:, -1] = rhs[:, 0]
    assert rel_l2(g.solve_inhomog_eqn(2, rhs), o.solve_inhomog(2, rhs)) <= 1e-13
    p = b.fnot * initial_psi(b, 2) * 30.0
    w, ts, tn = oracle.ekman_from_tau(b, *double_gyre_tau(b, rho0=b.rho))
    for x in (g, o):
        x.set_state(p, p)
        x.set_forcing(w, None, ts, tn)
        x.step(90.0, 1)
    for a, r in zip(g.get_state()[::2], o.get_state()[::2]):
        assert rel_l2(a, r) <= (1e-12 if precision == 0 else 1e-5)
    g.close()
    o.close()
