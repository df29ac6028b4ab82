"""The fast build's edge slots (csrc/bl_setup.cuh, k_edge): every face an
element refers to must carry the viscosity the CPU restatement gives it, on
meshes whose edges fill one block, straddle two, continue along mesh lines
or not at all, and on those whose two sides disagree.

Every step starts from the restatement's state (the steps between are
other kernels' work, whose round-off a tube's cross flow consists of).

Tolerance: at most 1e3 roundings (1.1e-16 each) on differences that amplify
them at most 1e2 times over a field: 1e-10 relative L1, and 1e-11 on the
time step."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs
from bookleaf_f90_gb300.setup import mesh as meshmod

pytestmark = pytest.mark.gpu

STEPS = 10


def _rotated(seed):
    """Corner numbering rotated per element: faces 1 and 2 then meet faces
    of every number, and many share no slot."""
    gen0 = meshmod.generate

    def gen(*a, **k):
        out = list(gen0(*a, **k))
        r = np.random.default_rng(seed).integers(0, 4, len(out[3]))
        idx = (np.arange(4)[None, :] + r[:, None]) % 4
        out[3] = np.ascontiguousarray(np.take_along_axis(out[3], idx, axis=1))
        return tuple(out)

    return gen


def _renumbered(p, seed):
    """The same problem with its elements in a random order: no two
    continuing edges are neighbours in the tables."""
    order = np.random.default_rng(seed).permutation(p.nel)
    place = np.empty_like(order)
    place[order] = np.arange(p.nel)
    for f, a in p.fields.items():
        if f not in (abi.IELSORT1, abi.IELSORT2) and len(a) == p.nel and f not in (
                abi.NDX, abi.NDY, abi.NDU, abi.NDV, abi.INDTYPE):
            a[...] = a[order]
    p.fields[abi.IELEL][...] = place[p.fields[abi.IELEL] - 1] + 1
    return p


def _check(p, tol=1e-10):
    from oracle.oracle import Oracle
    pc = p.copy()
    o, s = Oracle(pc), Solver(p, fp_mode=abi.FP_FAST)
    for _ in range(STEPS):
        for f in p.fields:
            p.fields[f][...] = pc.fields[f]
        s.sync_to_device(0)
        p.timestep = s.timestep = pc.timestep.copy()
        assert o.getdt(pc.timestep) == 0
        assert s.inf_solver_getdt() == 0, s.error.message
        assert abs(p.timestep.dt - pc.timestep.dt) <= 1e-11 * pc.timestep.dt
        s.sync_to_host(0)
        for ids in ((abi.ELVISC,), (abi.ELCS2,), (abi.CNVISCX, abi.CNVISCY)):
            off = sum(np.sum(np.abs(p.fields[f] - pc.fields[f])) for f in ids)
            size = sum(np.sum(np.abs(pc.fields[f])) for f in ids)
            assert off <= tol * size, (abi.NAMES[ids[0]], off, size)
        assert o.lagstep(pc.timestep) == 0
    s.close()


SIZES = [(4, 2), (9, 7), (18, 7), (127, 1), (128, 1), (33, 4), (64, 4), (2, 64)]


@pytest.mark.parametrize("nx,ny", SIZES)
def test_slots_over_block_edges(nx, ny):
    _check(Problem.from_deck(configs.sod(nx, ny)))


BLAST = configs.sedov(15, kappa=0.01, pmerit=0.1)
OPTIONS = {
    "blast": BLAST,
    "polar": configs.noh_polar(12, 7),
    # faces shorter than sqrt(zcut): the midpoint distance of the CFL length
    "short_faces": BLAST.replace("&INDICATORS", "&CUTOFF\n zcut=1.0e-1\n/\n&INDICATORS", 1),
    # a zerocut outside the range of k_edge's own limiter
    "general_limiter": BLAST.replace("&INDICATORS", "&CUTOFF\n zerocut=1.0e-30\n/\n&INDICATORS", 1),
    "midlength": BLAST.replace("cvisc2=0.75\n", "cvisc2=0.75\n zmidlength(1)=.TRUE.\n"),
    "no_edge_viscosity": BLAST.replace("cvisc2=0.75\n", "cvisc2=0.75\n visc='TENSOR'\n"),
}


@pytest.mark.parametrize("name", sorted(OPTIONS))
@pytest.mark.parametrize("mesh", ["lines", "rotated", "renumbered", "both"])
def test_options_and_numberings(monkeypatch, name, mesh):
    if mesh in ("rotated", "both"):
        monkeypatch.setattr(meshmod, "generate", _rotated(5))
    p = Problem.from_deck(OPTIONS[name])
    _check(_renumbered(p, 3) if mesh in ("renumbered", "both") else p)
