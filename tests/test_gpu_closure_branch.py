"""The learned closure beside k_lag_state: the cell volumes that it takes
from k_lag_force and from the vertices are those of the element fields, in
device loops and called steps alike, with the remap between the steps and
after an upload, for cells that fill a warp's rows, a block's, and one more.

Tolerance of the volumes: each step adds at most eight roundings to a cell's
two fractions (1.1e-16 each), over 21 steps less than 2e-14; 1e-13."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, closure, configs
from helpers import compare

pytestmark = pytest.mark.gpu

NORM = np.concatenate([[0.5, 1, 0.5, 1, 0.5, 1.4, 1.5, 0, 0.1, 0.3],
                       [3, 2, 3, 2, 3, 2, 2, 300, 5, 2], [1e-3, 10.0]]).astype(np.float32)


@pytest.mark.parametrize("fp", [abi.FP_FAST, abi.FP_MIXED, abi.FP_EXACT],
                         ids=["fast", "mixed", "exact"])
@pytest.mark.parametrize("ny,eul", [(16, False), (17, False), (65, False), (9, True)],
                         ids=["warp", "warp+1", "block+1", "eulerian"])
def test_loop_equals_calls_and_cells_keep_their_volume(ny, eul, fp):
    deck, frac = configs.sod_interface(8 * ny, ny, amplitude=0.0, periods=0, tilt=0.2,
                                       rho_right=0.5, p_right=0.5)
    base = Problem.from_deck(deck, material_fraction=frac)
    if eul:
        c = Problem.from_deck(configs.sod(8, 2, eulerian=True)).config
        for k in ("ale_zexist", "ale_zeul", "ale_adv_type", "ale_mintime", "ale_maxtime"):
            setattr(base.config, k, getattr(c, k))
        base.fields[abi.IELSORT2] = np.arange(1, base.sizes.nel + 1, dtype=np.int32)
    assert base.sizes.nmx >= ny
    net = closure.ClosureNet(closure.init_params(5))
    out = []
    for calls in (True, False):
        p = base.copy()
        s = Solver(p, fp_mode=fp)
        s.set_closure(net, NORM)
        for n in (5, 21):        # the second time after an upload
            if calls:
                for _ in range(n):
                    assert s.step() == 0, s.error.message
            else:
                assert s.run(max_steps=n, history=False)[0] == 0, s.error.message
            s.sync_to_host(0)
            s.sync_to_device(0)
        out.append((p, s.closure_stats()))
        s.close()
    net.close()
    (pa, seen), (pb, seen_b) = out
    assert seen == seen_b and seen[0] == 26 * int(np.sum(base.fields[abi.IMXNCP] == 2))
    assert not compare(pa, pb, exact=True)
    f = pa.fields
    two = f[abi.IMXNCP] == 2
    c0 = f[abi.IMXFCP][two] - 1
    for fid in (abi.CPVOLUME, abi.FRVOLUME, abi.CPENERGY, abi.CPDENSITY):
        assert np.array_equal(f[fid], pb.fields[fid]), abi.NAMES[fid]
    vol = f[abi.ELVOLUME][f[abi.IMXEL][two] - 1]
    if not eul:
        total = f[abi.CPVOLUME][c0] + f[abi.CPVOLUME][c0 + 1]
        assert np.max(np.abs(total - vol) / vol) <= 1e-13
    fractions = f[abi.FRVOLUME][c0] + f[abi.FRVOLUME][c0 + 1]
    assert np.max(np.abs(fractions - 1.0)) <= 1e-13
