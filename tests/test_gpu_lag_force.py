"""One Lagrangian step of the fast build from the CPU restatement's state:
the predictor's work, the half-step geometry from the element coefficients
(and from the corner positions where the coefficients may not be theirs),
and the corrector forces with and without their sub-zonal, hourglass and
mixed-cell parts, on meshes of one element row to a few blocks.

Tolerance: at most 1e3 roundings (1.1e-16 each), amplified at most 1e2 times
by the differences of the forces around a node: 1e-10 relative L1."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu

DECKS = {
    "all_forces": configs.sedov(12, kappa=0.01, pmerit=0.1),
    "subzonal": configs.sedov(16, pmerit=0.3),
    "hourglass": configs.sedov(11, kappa=0.05),
    "pressure": configs.sedov(9),
    "polar": configs.noh_polar(17, 15),
    "mixed_cells": configs.sod_multimaterial(24, 6),
}


@pytest.mark.parametrize("geometry", ["registered", "a2_b2_missing", "positions_alone"])
@pytest.mark.parametrize("name", sorted(DECKS))
def test_step_from_the_restatements_state(name, geometry):
    from oracle.oracle import Oracle
    pc = Problem.from_deck(DECKS[name])
    pg = pc.copy()
    o = Oracle(pc)
    for _ in range(6):
        assert o.step(pc.timestep) == 0
    assert o.getdt(pc.timestep) == 0
    for f in pg.fields:
        pg.fields[f][...] = pc.fields[f]
    if geometry == "a2_b2_missing":
        # the first half step then has only the positions to go by; the
        # corner forces at t^n do not need them without sub-zonal pressures
        if pg.config.zsp:
            pytest.skip("sub-zonal pressures need a2 and b2")
        del pg.fields[abi.A2], pg.fields[abi.B2]
    s = Solver(pg, fp_mode=abi.FP_FAST)
    s.sync_to_device(0)
    if geometry == "positions_alone":
        s.sync_to_device(abi.NDX)
    ts = pc.timestep.copy()
    assert s.inf_solver_lagstep(ts) == 0, s.error.message
    s.sync_to_host(0)
    s.close()
    assert o.lagstep(pc.timestep) == 0
    for ids in ((abi.ELDENSITY,), (abi.ELENERGY,), (abi.ELPRESSURE,), (abi.ELVOLUME,),
                (abi.NDU, abi.NDV), (abi.NDX, abi.NDY)):
        off = sum(np.sum(np.abs(pg.fields[f] - pc.fields[f])) for f in ids)
        size = sum(np.sum(np.abs(pc.fields[f])) for f in ids)
        assert off <= 1e-10 * size, (abi.NAMES[ids[0]], off, size)
