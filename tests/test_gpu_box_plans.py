"""The closed box's x-transform at the run-time plans (lengths without compiled
stages): every radix as the first and as a later stage of a subsequence, and
plans of three stages with every third radix, under the outer radices 16, 12, 10
and 6 (8 stands in the shortest box alone).  The list is checked against the
plan rule restated here.  The Helmholtz solve of every mode against the oracle
within 1e-13 up to 513 points and the wide grids' 1e-12 above, FP32 storage, an
ensemble and the one-kernel inverse within the parity contract's 1e-5 and 1e-12
for a step."""
import numpy as np
import pytest

import oracle
from openqg_b200.core import QG, Ensemble
from openqg_b200.params import OQG_MIXED, Basin
from tests.qg_numpy import rel_l2

RADICES = (16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2)
COMPILED = (128, 192, 256, 384, 512, 1024, 2048, 4096)


def plan(nxp):
    """The outer radix and a subsequence's radices (odd_r0, odd_split)."""
    m = 2 * (nxp - 1)
    r0 = next((r for r in (16, 12, 10, 8, 6, 4) if m % r == 0), 2)
    best = []

    def go(rest, cur):
        nonlocal best
        if rest == 1:
            if not best or (len(cur), sum(cur)) < (len(best), sum(best)):
                best = cur
            return
        for r in RADICES:
            if rest % r == 0 and (not cur or r <= cur[-1]):
                go(rest // r, cur + [r])

    go(m // r0, [])
    return r0, tuple(best)


def _admitted():
    for n in range(4, 2049):
        rest = n
        for f in (2, 3, 5):
            while rest % f == 0:
                rest //= f
        if rest == 1 and 2 * n not in COMPILED:
            yield n + 1


def _features(nxp):
    r0, rad = plan(nxp)
    return {("outer", r0)} | {(min(s, 2), r) for s, r in enumerate(rad)} | ({("three", r0)} if len(rad) == 3 else set())


# their plans: outer radix: subsequence's radices
WIDTHS = [
    5, 10,       # 8: -; 6: 3
    11, 21,      # 10: 2; 10: 4
    37, 51,      # 12: 6; 10: 10
    28, 76,      # 6: 9; 10: 15
    41, 101,     # 16: 5; 10: 5, 4
    82, 325,     # 6: 9, 3; 12: 9, 6
    385, 501,    # 16: 8, 6; 10: 10, 10
    577, 406,    # 16: 9, 8; 10: 9, 9
    769, 1537,   # 16: 12, 8; 16: 16, 12
    1126, 626,   # 10: 15, 15; 10: 5, 5, 5
    730, 751,    # 6: 9, 9, 3; 12: 5, 5, 5
    1251, 1601,  # 10: 10, 5, 5; 16: 8, 5, 5
    1729, 1876,  # 16: 6, 6, 6; 10: 15, 5, 5
    1216, 1297,  # 10: 9, 9, 3; 16: 9, 6, 3
    2026,        # 10: 9, 9, 5, the most threads of a transform
]


def test_widths_cover_the_plans():
    every = set().union(*map(_features, _admitted()))
    assert {f[1] for f in every if f[0] == "outer"} == {16, 12, 10, 8, 6}
    assert {f[1] for f in every if f[0] in (1, 2)} == set(RADICES) - {16, 2}      # OQG_ODD_LATER
    assert set().union(*map(_features, WIDTHS)) == every


def _box(nxp, nyp, precision=0, nl=3):
    return Basin(nxp=nxp, nyp=nyp, dx=1e4, dy=1e4, h=[350.0, 750.0, 2900.0][3 - nl:], gp=[0.05, 0.025][3 - nl:],
                 ah4=[1e9] * nl, ah2=[0.0] * nl, precision=precision)


def _p(b):
    x, y = np.linspace(0, 1, b.nxp), np.linspace(0, 1, b.nyp)
    return 0.1 * np.stack([np.outer(np.sin(np.pi * k * y), np.sin(3 * np.pi * x)) for k in (1, 2, 1)[:b.nl]])


@pytest.mark.gpu
@pytest.mark.parametrize("nxp", WIDTHS)
def test_solve_at_run_time_plans(gpu_required, nxp):
    b = _box(nxp, 9 + nxp % 2)
    g, o = QG(b), oracle.Oracle(b)
    rhs = np.random.default_rng(nxp).standard_normal(b.shape2)
    for m in range(1, b.nl + 1):
        assert rel_l2(g.solve_inhomog_eqn(m, rhs), o.solve_inhomog(m, rhs)) <= (1e-13 if nxp <= 513 else 1e-12)
    g.close()
    o.close()


# FP32 storage, and the one-kernel inverse where the grid admits it, at plans of
# one, two and three stages of a subsequence
@pytest.mark.gpu
@pytest.mark.parametrize("nxp,nl,precision,sep", [(626, 3, OQG_MIXED, True), (1729, 2, OQG_MIXED, True),
                                                  (1126, 2, OQG_MIXED, True), (626, 3, 0, False), (730, 2, 0, False),
                                                  (1251, 2, 0, False), (626, 3, OQG_MIXED, False),
                                                  (1601, 2, OQG_MIXED, False), (385, 3, 0, False), (76, 3, 0, False)])
def test_step_at_run_time_plans(gpu_required, nxp, nl, precision, sep):
    b = _box(nxp, 12, precision, nl)
    p = _p(b)
    g, o = QG(b), oracle.Oracle(b)
    g.set_xinv_sep(sep)
    for h in (g, o):
        h.set_state(p, 0.9 * p)
        h.set_forcing(np.zeros(b.shape2), None, 0.0, 0.0)
        h.step(600.0, 1)
    assert g.xinv_sep() == sep
    for a, r in zip(g.get_state()[::2], o.get_state()[::2]):
        assert rel_l2(a, r) <= (1e-12 if precision == 0 else 1e-5)
    g.close()
    o.close()


@pytest.mark.gpu
def test_ensemble_at_run_time_plans(gpu_required):
    bs = [_box(n, 11) for n in (626, 129, 406, 730, 76)]
    e = Ensemble(bs)
    for i, b in enumerate(bs):
        e.set_state(i, _p(b), 0.9 * _p(b))
        e.set_forcing(i, np.zeros(b.shape2))
    e.step(600.0, 1)
    e.sync()
    for i, b in enumerate(bs):
        o = oracle.Oracle(b)
        o.set_state(_p(b), 0.9 * _p(b))
        o.set_forcing(np.zeros(b.shape2), None, 0.0, 0.0)
        o.step(600.0, 1)
        for a, r in zip(e.get_state(i)[::2], o.get_state()[::2]):
            assert rel_l2(a, r) <= 1e-12
        o.close()
    e.close()
