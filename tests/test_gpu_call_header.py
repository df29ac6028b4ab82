"""What the called entry points report: the step header that the kernels
write for the host is the device loop's record of each step, bit for bit; of
several negative volumes, in several blocks, the last element's is returned,
and the next calls start clean."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu

MODES = pytest.mark.parametrize("fp", [abi.FP_FAST, abi.FP_MIXED, abi.FP_EXACT],
                                ids=["fast", "mixed", "exact"])


@MODES
@pytest.mark.parametrize("deck", [configs.sod(1, 1), configs.sod(32, 4), configs.sod(43, 3),
                                  configs.sedov(12, eulerian=True),
                                  configs.sedov(70, kappa=0.01, pmerit=0.1)],
                         ids=["one", "block", "block+1", "eulerian", "blocks"])
def test_calls_report_the_loops_records(deck, fp):
    pa = Problem.from_deck(deck)
    pb = pa.copy()
    sa, sb = Solver(pa, fp_mode=fp), Solver(pb, fp_mode=fp)
    got = []
    for _ in range(9):
        assert sa.step() == 0, sa.error.message
        t = pa.timestep
        got.append((t.nstep, t.time, t.dt, t.idtel, t.sdt.decode().strip()))
    ierr, want = sb.run(max_steps=9)
    assert ierr == 0
    assert got == [r[:4] + (r[4].strip(),) for r in want]
    sa.close()
    sb.close()


@MODES
def test_last_negative_volume_is_returned_and_forgotten(fp):
    from oracle.oracle import Oracle
    good = Problem.from_deck(configs.sod(100, 12))
    bad = good.copy()
    for col in (7, 60, 93):      # nodes across their right-hand neighbours
        bad.fields[abi.NDX][col * 13 + 5] += 2.5 / 100
    pc = bad.copy()
    o = Oracle(pc)
    assert o.getdt(pc.timestep) == 0
    want = o.lagstep(pc.timestep)
    s = Solver(bad, fp_mode=fp)
    first = bad.timestep.copy()
    assert s.inf_solver_getdt() == 0
    assert s.inf_solver_lagstep() == want < 0
    # the sound state in its place: nothing of the failure is left
    for fid, a in good.fields.items():
        if bad.fields[fid] is not None and a.dtype == np.float64:
            bad.fields[fid][...] = a
    s.sync_to_device(0)
    s2 = Solver(good, fp_mode=fp)
    for _ in range(3):
        assert s.step(first) == 0, s.error.message
        assert s2.step() == 0
    assert first.as_tuple() == good.timestep.as_tuple()
    s.close()
    s2.close()
