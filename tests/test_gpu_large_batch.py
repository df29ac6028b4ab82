"""Batches beyond one table of moves (128 pieces) and beyond one tile of
elements a block of the dt reduction (some 205,000 elements in all meshes):
every mesh moves and ends as it does by itself.

Tolerance of the fast and mixed builds' runs: the same kernels on the same
operands in another grid, so the reduction's choice is the same element and
the fields differ by at most 1e3 roundings of 1.1e-16 amplified 1e2 times:
1e-10 relative L1."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import BatchSolver, Problem, Solver, abi, configs
from helpers import compare
from test_gpu_moves import _pin

pytestmark = pytest.mark.gpu


def test_moves_of_more_than_one_table():
    decks = [configs.sod(5 + k, 2 + k % 3, eulerian=True) for k in range(5)]
    decks += [configs.sedov(4 + k, eulerian=True) for k in range(4)]
    base = [Problem.from_deck(d) for d in decks]
    a, b = [p.copy() for p in base], [_pin(p.copy(), True) for p in base]
    assert len(b) * sum(f.dtype == np.float64 for f in b[0].fields.values()) > 2 * 100
    for probs in (a, b):
        s = BatchSolver(probs, fp_mode=abi.FP_EXACT)
        first = [p.timestep.copy() for p in probs]
        assert s.run(max_steps=3)[0] == 0
        assert s.sync_to_device(0) == 0
        for p, t in zip(probs, first):
            p.timestep = t
        assert s.run(max_steps=5)[0] == 0
        assert s.sync_to_host(0) == 0
        s.close()
    for p, q in zip(a, b):
        assert not compare(p, q, exact=True)


@pytest.mark.parametrize("fp", [abi.FP_FAST, abi.FP_MIXED], ids=["fast", "mixed"])
def test_several_tiles_a_block(fp):
    base = [Problem.from_deck(d) for d in (configs.sod(7, 3), configs.sedov(400),
                                           configs.sod(33, 1), configs.sod(500, 110))]
    assert sum(p.nel for p in base) // 128 + 532 >= 2 * 1064
    together, alone = [p.copy() for p in base], [p.copy() for p in base]
    b = BatchSolver(together, fp_mode=fp)
    assert b.run(max_steps=12)[0] == 0
    assert b.sync_to_host(0) == 0
    b.close()
    for p, q in zip(together, alone):
        s = Solver(q, fp_mode=fp)
        assert s.run(max_steps=12, history=False)[0] == 0
        s.sync_to_host(0)
        s.close()
        assert p.timestep.idtel == q.timestep.idtel
        assert abs(p.timestep.dt - q.timestep.dt) <= 1e-11 * q.timestep.dt
        for ids in ((abi.ELDENSITY,), (abi.ELENERGY,), (abi.NDU, abi.NDV), (abi.NDX, abi.NDY)):
            off = sum(np.sum(np.abs(p.fields[f] - q.fields[f])) for f in ids)
            size = sum(np.sum(np.abs(q.fields[f])) for f in ids)
            assert off <= 1e-10 * size, (abi.NAMES[ids[0]], off, size)
