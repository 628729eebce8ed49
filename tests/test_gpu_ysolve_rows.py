"""The y-solve at the heights where its shape changes (rows per thread 4, 8 and
16; column groups of 8, 4 and 2 boxes' or 4, 2 and 1 channels' wavenumbers;
one, two and more warps per group; several groups per CTA) and at widths that
leave a group partly empty, with every spread: the Helmholtz solve of every
mode against the oracle, within 1e-13 up to 513 rows and the wide grids' 1e-12
above."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG
from openqg_b200.params import Basin
from tests.qg_numpy import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


def _basin(nxp, ny, cyclic):
    return Basin(nxp=nxp, nyp=ny + 2, dx=1e4, dy=1e4, h=[350.0, 750.0, 2900.0], gp=[0.05, 0.025], ah4=[1e9] * 3,
                 ah2=[0.0] * 3, cyclic=cyclic, dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else 3)


@pytest.mark.parametrize("cyclic", [False, True], ids=["box", "channel"])
@pytest.mark.parametrize("ny", [3, 4, 5, 16, 17, 99, 100, 101, 199, 201, 399, 401, 511, 1023, 1025, 2047, 2049, 3100])
def test_ysolve_heights(ny, cyclic):
    for nxp in ((11, 17) if ny < 600 else (17,)):
        b = _basin(nxp, ny, cyclic)
        g, o = QG(b), oracle.Oracle(b)
        rhs = np.random.default_rng(ny + nxp).standard_normal(b.shape2)
        if cyclic:
            rhs[:, -1] = rhs[:, 0]
        ref = [o.solve_inhomog(m, rhs) for m in range(1, b.nl + 1)]
        for warps in (1, 2, 4):
            g.set_ysolve_warps(warps)
            for m in range(1, b.nl + 1):
                err = rel_l2(g.solve_inhomog_eqn(m, rhs), ref[m - 1])
                assert err <= (1e-13 if ny <= 513 else 1e-12), (nxp, warps, m, err)
        g.close()
        o.close()
