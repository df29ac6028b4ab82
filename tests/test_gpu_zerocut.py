"""Edges whose velocity difference is at most zerocut, but not zero: their
force is cut, their viscosity is not (hydro_kn_edgeviscosity.f90:185-282), and
it counts in the element's largest and so in the time step.

Tolerance: the fast build at most 1e3 roundings (1.1e-16 each), amplified at
most 1e2 times by differences: 1e-10 relative L1, and 1e-11 on the time step.
The mixed build some hundred FP32 roundings of 6e-8: 1e-5."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu


# (the squares of differences around 1e-30 are beyond FP32)
@pytest.mark.parametrize("zerocut,build", [(1e-30, "fast"), (1e-6, "fast"), (1e-3, "fast"),
                                           (1e-6, "mixed"), (1e-3, "mixed")])
@pytest.mark.parametrize("n", [5, 17])
def test_viscosity_of_cut_edges(n, zerocut, build):
    from oracle.oracle import Oracle
    fp, tol, tdt = {"fast": (abi.FP_FAST, 1e-10, 1e-11),
                    "mixed": (abi.FP_MIXED, 1e-5, 1e-5)}[build]
    pc = Problem.from_deck(configs.sedov(n, kappa=0.01, pmerit=0.1))
    f = pc.fields
    pc.config.zerocut = zerocut
    x, y = f[abi.NDX] / f[abi.NDX].max(), f[abi.NDY] / f[abi.NDY].max()
    # differences around a cell of 0.01 to 0.9 of the cut-off, converging
    f[abi.NDU][...] = -0.4 * zerocut * n * x * x
    f[abi.NDV][...] = -0.3 * zerocut * n * y * y
    pg = pc.copy()
    s, o = Solver(pg, fp_mode=fp), Oracle(pc)
    assert s.inf_solver_getdt() == o.getdt(pc.timestep) == 0
    s.sync_to_host(0)
    s.close()
    assert np.sum(pc.fields[abi.ELVISC] > 0.0) > n
    for ids in ((abi.ELVISC,), (abi.ELCS2,), (abi.CNVISCX, abi.CNVISCY)):
        off = sum(np.sum(np.abs(pg.fields[f] - pc.fields[f])) for f in ids)
        size = sum(np.sum(np.abs(pc.fields[f])) for f in ids)
        assert off <= tol * size, (abi.NAMES[ids[0]], off, size)
    assert abs(pg.timestep.dt - pc.timestep.dt) <= tdt * pc.timestep.dt
