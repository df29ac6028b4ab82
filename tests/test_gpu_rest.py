"""The edge viscosity of fluid at rest, which the exact build leaves out edge
by edge and the mixed one cell by cell: patches of nodes at rest, of zeros of
either sign, moving alike and moving apart, a cell of infinite density, with
and without the zero cut-off.  The exact build equals the CPU restatement bit
for bit; the mixed build has its zeros, and elsewhere differs by at most some
hundred FP32 roundings (6e-8 each): 1e-5 relative L1.

And the predictor's work, which the fast and mixed builds leave out of cells
at rest with finite forces: one Lagrangian step of the fast build within 1e-10
of the restatement's (1e3 roundings of 1.1e-16, amplified 1e2 times by
differences), and an infinite pressure still makes the energy no number."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu


def _patches(n, zerocut):
    p = Problem.from_deck(configs.sedov(n, kappa=0.01, pmerit=0.1))
    f = p.fields
    p.config.zerocut = zerocut
    x, y = f[abi.NDX], f[abi.NDY]
    top, right = y > 0.5 * y.max(), x > 0.5 * x.max()
    f[abi.NDU][...] = 0.0
    f[abi.NDV][...] = 0.0
    f[abi.NDU][top & ~right] = -0.0
    f[abi.NDV][(top & ~right) & (np.arange(x.size) % 2 == 0)] = -0.0
    f[abi.NDU][right & ~top], f[abi.NDV][right & ~top] = 0.3, -0.2
    apart = right & top
    f[abi.NDU][apart] = -x[apart] ** 2
    f[abi.NDV][apart] = 0.5 * x[apart] * y[apart] - y[apart]
    return p


@pytest.mark.parametrize("zerocut", [1e-40, 1e-6, 0.0])
@pytest.mark.parametrize("n", [5, 12, 33])
def test_exact_edges_at_rest(n, zerocut):
    from oracle.oracle import Oracle
    pg = _patches(n, zerocut)
    pg.fields[abi.ELDENSITY][n + 1] = np.inf
    pc = pg.copy()
    o = Oracle(pc)
    s = Solver(pg, fp_mode=abi.FP_EXACT)
    assert s.inf_solver_getdt() == o.getdt(pc.timestep)
    s.sync_to_host(0)
    s.close()
    assert pg.timestep.as_tuple() == pc.timestep.as_tuple()
    for fid in (abi.ELVISC, abi.CNVISCX, abi.CNVISCY, abi.ELCS2):
        assert np.array_equal(pg.fields[fid], pc.fields[fid], equal_nan=True), abi.NAMES[fid]
    assert np.any(pc.fields[abi.ELVISC] > 0.0)


@pytest.mark.parametrize("n", [5, 12, 33])
def test_mixed_cells_at_rest(n):
    from oracle.oracle import Oracle
    pg = _patches(n, 1e-40)
    pc = pg.copy()
    o = Oracle(pc)
    s = Solver(pg, fp_mode=abi.FP_MIXED)
    assert s.inf_solver_getdt() == o.getdt(pc.timestep) == 0
    s.sync_to_host(0)
    s.close()
    nd = pc.fields[abi.IELND] - 1
    still = np.ones(len(nd), dtype=bool)
    for fid in (abi.NDU, abi.NDV):
        w = pc.fields[fid][nd]
        still &= np.all(w == w[:, :1], axis=1)
    assert 0 < np.sum(still) < len(nd)
    for fid in (abi.ELVISC, abi.CNVISCX, abi.CNVISCY):
        a, b = pg.fields[fid], pc.fields[fid]
        assert np.all(b[still] == 0.0) and np.all(a[still] == 0.0), abi.NAMES[fid]
        assert np.sum(np.abs(a - b)) <= 1e-5 * np.sum(np.abs(b)), abi.NAMES[fid]


@pytest.mark.parametrize("n", [5, 12, 33])
def test_step_of_cells_at_rest(n):
    from oracle.oracle import Oracle
    pc = _patches(n, 1e-40)
    o = Oracle(pc)
    assert o.getdt(pc.timestep) == 0
    pg = pc.copy()
    ts = pc.timestep.copy()
    s = Solver(pg, fp_mode=abi.FP_FAST)
    assert s.inf_solver_lagstep(ts) == o.lagstep(pc.timestep) == 0
    s.sync_to_host(0)
    s.close()
    kinetic = 0.5 * np.sum(pc.fields[abi.NDU] ** 2 + pc.fields[abi.NDV] ** 2)
    for ids in ((abi.ELDENSITY,), (abi.ELENERGY,), (abi.NDU, abi.NDV), (abi.NDX, abi.NDY)):
        off = sum(np.sum(np.abs(pg.fields[f] - pc.fields[f])) for f in ids)
        size = sum(np.sum(np.abs(pc.fields[f])) for f in ids)
        size += kinetic if ids[0] == abi.ELENERGY else 0.0
        assert off <= 1e-10 * size, (abi.NAMES[ids[0]], off, size)


@pytest.mark.parametrize("fp", [abi.FP_FAST, abi.FP_MIXED], ids=["fast", "mixed"])
def test_infinite_pressure_at_rest_is_not_left_out(fp):
    p = _patches(12, 1e-40)
    s = Solver(p, fp_mode=fp)
    assert s.inf_solver_getdt() == 0
    s.sync_to_host(0)
    p.fields[abi.ELPRESSURE][13] = np.inf
    s.sync_to_device(0)
    s.inf_solver_lagstep()
    s.sync_to_host(0)
    s.close()
    assert np.isnan(p.fields[abi.ELENERGY][13])


@pytest.mark.parametrize("n", [5, 12, 33])
def test_exact_step_of_cells_at_rest(n):
    """k_lag_state's energy at rest: bit for bit the restatement's, zero
    energies of either sign among them."""
    from oracle.oracle import Oracle
    pg = _patches(n, 1e-40)
    e = pg.fields[abi.ELENERGY]
    e[1], e[n] = 0.0, -0.0
    pc = pg.copy()
    o = Oracle(pc)
    s = Solver(pg, fp_mode=abi.FP_EXACT)
    for _ in range(3):
        assert s.step() == o.step(pc.timestep) == 0
    s.sync_to_host(0)
    s.close()
    for fid in (abi.ELENERGY, abi.ELDENSITY, abi.ELPRESSURE, abi.NDU, abi.NDV, abi.NDX):
        assert np.array_equal(pg.fields[fid], pc.fields[fid]), abi.NAMES[fid]
