"""FP32 storage at transform lengths M with M + M/8 odd: the transform buffers
must keep the 16-byte alignment that the staged copies of the rows need (the
second of a pair of M + M/8 + 4 complex FP32 values would start on 8 bytes).
psi and q within 1e-5 of the FP64 oracle after a step, as at the other
lengths."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG
from openqg_b200.params import OQG_MIXED, Basin, atmos_channel, double_gyre_tau, initial_psi
from tests.qg_numpy import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


def _box(nxp, nyp):
    return Basin(nxp=nxp, nyp=nyp, dx=2e4, dy=2e4, h=[350.0, 750.0, 2900.0], gp=[0.05, 0.025], ah4=[2e10] * 3,
                 ah2=[0.0] * 3, precision=OQG_MIXED)


# (M, separate inverse): box M = 2 (nxp - 1) = 72, 216; channel M = nxp - 1 = 75, 120
@pytest.mark.parametrize("b,sep", [(_box(37, 41), True), (_box(37, 41), False), (_box(109, 57), True),
                                   (_box(109, 57), False),
                                   (atmos_channel(76, 49, precision=OQG_MIXED), False),
                                   (atmos_channel(76, 49, precision=OQG_MIXED), True),
                                   (atmos_channel(121, 49, precision=OQG_MIXED), True)],
                         ids=["box37", "box37-fused", "box109", "box109-fused", "chan76-fused", "chan76", "chan121"])
def test_fp32_step_at_odd_buffer_lengths(b, sep):
    p = b.fnot * initial_psi(b, 2) * (30.0 if b.cyclic else 1.0)
    w, ts, tn = oracle.ekman_from_tau(b, *double_gyre_tau(b, rho0=b.rho))
    g, o = QG(b), oracle.Oracle(b)
    g.set_xinv_sep(sep)
    tdt = 360.0 if b.cyclic else 3600.0
    for x in (g, o):
        x.set_state(p, p)
        x.set_forcing(w, None, ts, tn)
        x.step(tdt, 1)
    for a, r in zip(g.get_state()[::2], o.get_state()[::2]):
        assert rel_l2(a, r) <= 1e-5
    assert np.all(np.isfinite(g.get_state()[0]))
    g.close()
    o.close()
