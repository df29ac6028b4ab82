"""Host arrays that are pinned in part only: a kernel may not address them.
They go to the runtime's copies, which move all of an array or refuse it; an
array that spans two registrations side by side goes there too.  Either way
the context goes on, and the arrays around it move as they do."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import BatchSolver, Problem, Solver, abi, configs

pytestmark = pytest.mark.gpu

PAGE = 65536  # a multiple of every page size


def _aligned(a, pages):
    """a's values at the start of a page of a buffer of its own."""
    raw = np.zeros((pages + 1) * PAGE, dtype=np.uint8)
    o = -raw.ctypes.data % PAGE
    v = raw[o:o + a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    return raw, v


@pytest.mark.parametrize("batch", [False, True], ids=["single", "batch"])
@pytest.mark.parametrize("registered", [[(0, 1)], [(1, 1)], [(0, 1), (1, 1)]],
                         ids=["first_page", "second_page", "two_pages"])
def test_partly_registered_array(registered, batch):
    import torch
    rt = torch.cuda.cudart()
    torch.zeros(1, device="cuda")
    base = Problem.from_deck(configs.sedov(60, kappa=0.01))  # cnwt: 115,200 bytes
    pa, pb = base.copy(), base.copy()
    assert PAGE < pb.fields[abi.CNWT].nbytes <= 2 * PAGE
    raw, pb.fields[abi.CNWT] = _aligned(pb.fields[abi.CNWT], 2)
    at = pb.fields[abi.CNWT].ctypes.data
    sols = [BatchSolver([p]) if batch else Solver(p) for p in (pa, pb)]
    for first, n in registered:
        assert int(rt.cudaHostRegister(at + first * PAGE, n * PAGE, 0)) == 0
    try:
        for s in sols:
            assert s.run(max_steps=3)[0] == 0
            assert s.sync_to_host(abi.ELENERGY) in (None, 0)
        sols[0].sync_to_host(abi.CNWT)
        before = pb.fields[abi.CNWT].copy()
        try:
            came = sols[1].sync_to_host(abi.CNWT) in (None, 0)
        except RuntimeError:
            came = False
        if came:
            assert np.array_equal(pb.fields[abi.CNWT], pa.fields[abi.CNWT])
        else:
            pb.fields[abi.CNWT][...] = before
        try:
            sols[1].sync_to_device(abi.CNWT)
        except RuntimeError:
            pass
        for s in sols:
            assert s.sync_to_host(abi.NDX) in (None, 0)
            s.close()
        for f in (abi.ELENERGY, abi.NDX):
            assert np.array_equal(pa.fields[f], pb.fields[f])
    finally:
        for first, _ in registered:
            assert int(rt.cudaHostUnregister(at + first * PAGE)) == 0
    del raw
