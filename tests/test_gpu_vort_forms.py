"""The vorticity kernel's forms by tile count (a cluster of one CTA per layer, a
CTA of twice the threads, a plain CTA) at grids on either side of the lines
between them, with ragged last tiles in x and y, two to four layers, boxes and
channels (tiles at the seam and off it): a step against the oracle within the
parity contract (1e-12 in FP64, 1e-5 in FP32 storage)."""
import pytest

from openqg_b200.params import OQG_MIXED, Basin
from tests.qg_numpy import rel_l2
from tests.test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu

H = {2: ([500.0, 3500.0], [0.03]), 3: ([350.0, 750.0, 2900.0], [0.05, 0.025]),
     4: ([300.0, 500.0, 1000.0, 2200.0], [0.05, 0.025, 0.015])}


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


# nxp, nyp: tiles of 60 columns by 8 interior rows.  Clusters while strips + nl
# tiles <= 296, double CTAs while strips + tiles <= 148
GRIDS = [(5, 5), (61, 10), (121, 11), (181, 189), (181, 197), (181, 277), (181, 301), (241, 330)]


@pytest.mark.parametrize("nl", [2, 3, 4])
@pytest.mark.parametrize("nxp,nyp", GRIDS)
@pytest.mark.parametrize("cyclic", [False, True], ids=["box", "channel"])
def test_vorticity_forms(nxp, nyp, nl, cyclic):
    h, gp = H[nl]
    for precision, tol in ((0, 1e-12), (OQG_MIXED, 1e-5)):
        b = Basin(nxp=nxp, nyp=nyp, dx=2e4, dy=2e4, h=h, gp=gp, ah2=[10.0] * nl, ah4=[2e10] * nl, cyclic=cyclic,
                  dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else nl, bcco=1.0 if cyclic else 1e20,
                  precision=precision)
        g, o = make_pair(b, ent=True)
        g.set_tile_rows(8)
        g.step(600.0, 1)
        o.step(600.0, 1)
        for a, r in zip(g.get_state()[::2], o.get_state()[::2]):
            assert rel_l2(a, r) <= tol, (precision, nl)
        g.close()
        o.close()
