"""Infinities and NaN in the remap of the fast build: what is no number on one
side of a face is none on the other after the remap, whether volume crosses
the face or not, as in the CPU restatement (0 times infinity, and a limiter
with a NaN in it, are NaN).  Where both are numbers the two agree within 1e3
roundings of 1.1e-16 amplified at most 1e2 times: 1e-10 relative L1."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu


def _after_lagstep(flow, slope):
    """A 9x9 box in a uniform flow (none, along x, aslant) with a linear
    energy, after the Lagrangian step of the restatement and of the GPU."""
    from oracle.oracle import Oracle
    pc = Problem.from_deck(configs.noh(9, eulerian=True))
    f = pc.fields
    nd = f[abi.IELND] - 1
    xc, yc = f[abi.NDX][nd].mean(1), f[abi.NDY][nd].mean(1)
    f[abi.NDU][...], f[abi.NDV][...] = flow
    f[abi.ELENERGY][...] = 1.0 + slope[0] * xc + slope[1] * yc
    o = Oracle(pc)
    assert o.getdt(pc.timestep) == 0
    pg = pc.copy()
    s = Solver(pg, fp_mode=abi.FP_FAST)
    assert s.inf_solver_lagstep() == o.lagstep(pc.timestep) == 0
    s.sync_to_host(0)
    return pc, o, pg, s


def _remap(pc, o, pg, s, field, value):
    for p in (pc, pg):
        p.fields[field][CELL] = value
    s.sync_to_device(field)
    s.inf_solver_alestep()
    o.alestep(pc.timestep)
    s.sync_to_host(0)
    s.close()


CELL = 4 * 9 + 4


@pytest.mark.parametrize("value", [np.inf, np.nan], ids=["inf", "nan"])
@pytest.mark.parametrize("field", [abi.ELENERGY, abi.ELDENSITY], ids=["energy", "density"])
@pytest.mark.parametrize("flow", [(0.0, 0.0), (0.25, 0.0), (0.25, -0.125)],
                         ids=["rest", "along", "aslant"])
def test_what_is_no_number_stays_none(flow, field, value):
    pc, o, pg, s = _after_lagstep(flow, (0.0, 0.0))
    _remap(pc, o, pg, s, field, value)
    around = np.append(pc.fields[abi.IELEL][CELL] - 1, CELL)
    assert not np.isfinite(pc.fields[field][around]).any()
    assert not np.isfinite(pg.fields[field][around]).any()
    for fid in (abi.ELENERGY, abi.ELDENSITY, abi.NDU, abi.NDV):
        a, b = pg.fields[fid], pc.fields[fid]
        ok = np.isfinite(a) & np.isfinite(b)
        assert np.sum(np.abs(a[ok] - b[ok])) <= 1e-10 * np.sum(np.abs(b[ok])) + 1e-14


@pytest.mark.parametrize("slope", [(0.3, 0.2), (0.3, -0.2), (-0.3, -0.2)])
@pytest.mark.parametrize("value", [np.inf, np.nan], ids=["inf", "nan"])
def test_limiter_with_one_side_no_number(value, slope):
    """A neighbour of the cell whose own slope on its far side is positive
    has two slopes of one sign, one of them no number; the cell beyond takes
    the flux that they limit."""
    pc, o, pg, s = _after_lagstep((0.25, -0.125), slope)
    e, el = pc.fields[abi.ELENERGY].copy(), pc.fields[abi.IELEL] - 1
    beyond = []
    for n in el[CELL]:
        for i in range(2):
            a, b = el[n, i], el[n, i + 2]  # the slopes e - e[b] and e[a] - e
            if a == CELL and e[n] - e[b] > 0.0:
                beyond.append(b)
            if b == CELL and e[a] - e[n] > 0.0:
                beyond.append(a)
    assert beyond
    _remap(pc, o, pg, s, abi.ELENERGY, value)
    a, b = pg.fields[abi.ELENERGY][beyond], pc.fields[abi.ELENERGY][beyond]
    assert np.array_equal(np.isfinite(a), np.isfinite(b)), (beyond, a, b)
    assert np.isfinite(b).all() == np.isinf(value)
