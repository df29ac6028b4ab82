"""Host arrays that two fields or two meshes share, or whose ends overlap: a
whole download leaves what the last of them in order wrote, whole, as copies
one after the other do, also where the arrays are pinned and each move is a
kernel's."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import BatchSolver, Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
    v = t.numpy().reshape(a.shape)
    v[...] = a
    return t, v


@pytest.mark.parametrize("n", [24, 384])
def test_fields_that_share_an_array(n):
    pa = Problem.from_deck(configs.sedov(n, kappa=0.01))
    pb = pa.copy()
    keep = []
    for f in (abi.ELPRESSURE, abi.ELDENSITY, abi.NDU):
        t, pb.fields[f] = _pinned(pb.fields[f])
        keep.append(t)
    # elvisc on elpressure's array; ndv over the second half of ndu's
    t, both = _pinned(np.zeros(pb.nnd + pb.nnd // 2))
    keep.append(t)
    h = pb.nnd // 2
    both[:pb.nnd] = pb.fields[abi.NDU]
    ndu, ndv = both[:pb.nnd], both[h:h + pb.nnd]
    ndv[...] = 0.0
    both[:h] = pb.fields[abi.NDU][:h]
    assert not pa.fields[abi.NDU].any() and not pa.fields[abi.NDV].any()
    pb.fields[abi.NDU], pb.fields[abi.NDV] = ndu, ndv
    pb.fields[abi.ELVISC] = pb.fields[abi.ELPRESSURE]
    for p in (pa, pb):
        s = Solver(p, fp_mode=abi.FP_EXACT)
        assert s.run(max_steps=4, history=False)[0] == 0
        for _ in range(5):
            s.sync_to_host(0)
        s.close()
    assert np.array_equal(pb.fields[abi.ELDENSITY], pa.fields[abi.ELDENSITY])
    assert np.array_equal(pb.fields[abi.ELPRESSURE], pa.fields[abi.ELVISC])
    assert np.array_equal(ndv, pa.fields[abi.NDV])
    assert np.array_equal(ndu[:h], pa.fields[abi.NDU][:h])


@pytest.mark.parametrize("n", [24, 384])
def test_meshes_that_share_their_arrays(n):
    base = Problem.from_deck(configs.sedov(n, kappa=0.01))
    keep = []
    for f in (abi.ELPRESSURE, abi.ELENERGY, abi.CNWT):
        t, base.fields[f] = _pinned(base.fields[f])
        keep.append(t)
    first, second, alone = base.copy(), base.copy(), base.copy()
    for f in base.fields:          # two meshes of one set of arrays, one a step ahead
        first.fields[f] = second.fields[f] = base.fields[f]
    first.config.dt_initial = 0.5 * second.config.dt_initial
    a = Solver(alone, fp_mode=abi.FP_EXACT)
    assert a.run(max_steps=4, history=False)[0] == 0
    a.sync_to_host(0)
    a.close()
    b = BatchSolver([first, second], fp_mode=abi.FP_EXACT)
    assert b.run(max_steps=4)[0] == 0
    for _ in range(5):
        assert b.sync_to_host(0) == 0
    b.close()
    for f in (abi.ELPRESSURE, abi.ELENERGY, abi.CNWT, abi.ELDENSITY):
        assert np.array_equal(base.fields[f], alone.fields[f]), abi.NAMES[f]
