"""The y-solve above 4096 rows (one box column per group, 16 rows per thread, up
to 15 warps), up to the tallest box that each spread admits, and in an ensemble
whose short members share the tall one's shape: the Helmholtz solve of every
mode within the wide grids' 1e-12 of the oracle, a step within the parity
contract's 1e-12 (FP64) and 1e-5 (FP32 storage)."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG, Ensemble, OqgError
from openqg_b200.params import OQG_MIXED, Basin
from tests.qg_numpy import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu(gpu_required):
    pass


def _box(nxp, ny, precision=0):
    return Basin(nxp=nxp, nyp=ny + 2, dx=1e4, dy=1e4, h=[500.0, 3500.0], gp=[0.03], ah4=[1e9] * 2, ah2=[0.0] * 2,
                 precision=precision)


def _p(b):
    x, y = np.linspace(0, 1, b.nxp), np.linspace(0, 1, b.nyp)
    return 0.1 * np.stack([np.outer(np.sin(np.pi * k * y), np.sin(np.pi * x)) for k in (1, 2)])


def _start(b, *handles):
    for h in handles:
        h.set_state(_p(b), 0.9 * _p(b))
        h.set_forcing(np.zeros(b.shape2), None, 0.0, 0.0)
        h.step(600.0, 1)


@pytest.mark.parametrize("nxp,ny,warps", [(11, 4097, (1, 2, 4)), (17, 4500, (1, 2, 4)), (11, 7040, (4,)),
                                          (11, 7168, (2,)), (11, 7200, (1,))])
def test_tall_box(nxp, ny, warps):
    b = _box(nxp, ny)
    g, o = QG(b), oracle.Oracle(b)
    rhs = np.random.default_rng(ny).standard_normal(b.shape2)
    for m in range(1, b.nl + 1):
        ref = o.solve_inhomog(m, rhs)
        for w in warps:
            g.set_ysolve_warps(w)
            assert rel_l2(g.solve_inhomog_eqn(m, rhs), ref) <= 1e-12, (m, w)
    _start(b, g, o)
    for a, r in zip(g.get_state()[::2], o.get_state()[::2]):
        assert rel_l2(a, r) <= 1e-12
    g.close()
    f = QG(_box(nxp, ny, OQG_MIXED))
    _start(b, f)
    for a, r in zip(f.get_state()[::2], o.get_state()[::2]):
        assert rel_l2(a, r) <= 1e-5
    f.close()
    o.close()


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (OQG_MIXED, 1e-5)], ids=["fp64", "fp32"])
def test_ensemble_of_tall_and_short_boxes(precision, tol):
    bs = [_box(nxp, ny, precision) for nxp, ny in ((17, 4200), (65, 31), (11, 1100), (129, 600))]
    e = Ensemble(bs)
    for i, b in enumerate(bs):
        e.set_state(i, _p(b), 0.9 * _p(b))
        e.set_forcing(i, np.zeros(b.shape2))
    e.step(600.0, 1)
    e.sync()
    for i, b in enumerate(bs):
        o = oracle.Oracle(b)
        _start(b, o)
        for a, r in zip(e.get_state(i)[::2], o.get_state()[::2]):
            assert rel_l2(a, r) <= tol, i
        o.close()
    e.close()


def _takes(call):
    try:
        call()
    except OqgError as e:
        assert "OQG_EUNSUPPORTED" in str(e)
        return False
    return True


@pytest.mark.parametrize("cyclic,most", [(False, (7200, 7168, 7040)), (True, (3584, 3520, 3456))], ids=["box", "channel"])
def test_height_limits(cyclic, most):
    def basin(ny):
        return Basin(nxp=9, nyp=ny + 2, dx=1e4, dy=1e4, h=[500.0, 3500.0], gp=[0.03], ah4=[1e9] * 2, ah2=[0.0] * 2,
                     cyclic=cyclic, dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else 2)

    for ny in sorted({m + d for m in most for d in (0, 1)}):
        if ny > most[0]:
            assert not _takes(lambda: QG(basin(ny)).close())
            continue
        g = QG(basin(ny))
        assert [_takes(lambda: g.set_ysolve_warps(w)) for w in (1, 2, 4)] == [ny <= m for m in most], ny
        g.close()


# nxp at the one-kernel inverse's limit and the next admitted length
@pytest.mark.parametrize("nl,cyclic,nxp,beyond", [(2, False, 1601, 1621), (3, False, 1025, 1081), (4, False, 801, 811),
                                                  (2, True, 2701, 2881), (3, True, 1801, 1876),
                                                  (4, True, 1351, 1441)])
def test_one_kernel_inverse_limits(nl, cyclic, nxp, beyond):
    for n, ok in ((nxp, True), (beyond, False)):
        g = QG(Basin(nxp=n, nyp=9, dx=1e4, dy=1e4, h=[300.0, 500.0, 1000.0, 2200.0][:nl], gp=[0.05, 0.025, 0.015][:nl - 1],
                     ah4=[1e9] * nl, ah2=[0.0] * nl, cyclic=cyclic, dz_sign=1 if cyclic else -1, k_topo=1 if cyclic else nl))
        assert _takes(lambda: g.set_xinv_sep(False)) == ok
        g.close()
