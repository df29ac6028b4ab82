"""Uploads and downloads of the state between pinned host arrays (moved by
kernels, straight to each mesh's own arrays) and pageable ones (copies):
the same bits either way, for single meshes and batches, fields of odd
length and arrays that start on 8 but not on 16 bytes."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import BatchSolver, Problem, Solver, abi, configs
from helpers import compare

pytestmark = pytest.mark.gpu


def _pin(p, skew):
    """p's arrays as views of one pinned buffer, every other one skewed by
    8 bytes."""
    import torch
    size = sum(-(-a.nbytes // 16) * 16 + 16 for a in p.fields.values())
    buf = torch.empty(size, dtype=torch.uint8, pin_memory=True)
    raw, at = buf.numpy(), 0
    for k, (f, a) in enumerate(p.fields.items()):
        o = at + (8 if skew and k % 2 else 0)
        v = raw[o:o + a.nbytes].view(a.dtype).reshape(a.shape)
        v[...] = a
        p.fields[f] = v
        at += -(-a.nbytes // 16) * 16 + 16
    p.pinned = buf
    return p


SINGLE = {"odd": configs.sod(7, 3), "one_row": configs.sod(33, 1),
          "mixed_cells": configs.sod_multimaterial(20, 5), "blast": configs.sedov(41, kappa=0.01)}


@pytest.mark.parametrize("skew", [False, True], ids=["aligned", "skewed"])
@pytest.mark.parametrize("name", sorted(SINGLE))
def test_single(name, skew):
    base = Problem.from_deck(SINGLE[name])
    pa, pb = base.copy(), _pin(base.copy(), skew)
    for p in (pa, pb):
        s = Solver(p, fp_mode=abi.FP_EXACT)
        ts = p.timestep.copy()
        assert s.run(max_steps=3, history=False)[0] == 0
        s.sync_to_device(0)                       # the initial state again
        assert s.run(max_steps=5, ts=ts, history=False)[0] == 0
        assert s.inf_solver_getdt(ts) == 0        # elcs2 then holds cs2 + viscosity
        s.sync_to_host(0)
        p.fields[abi.NDU] *= 1.5
        s.sync_to_device(abi.NDU)
        s.sync_to_device(abi.ELCS2)
        assert s.inf_solver_lagstep(ts) == 0
        s.sync_to_host(0)
        s.close()
    assert not compare(pa, pb, exact=True)


@pytest.mark.parametrize("pins", ["all", "some"])
def test_batch(pins):
    decks = [configs.sod(9, 3, eulerian=True), configs.sedov(7, eulerian=True),
             configs.sod(5, 5, eulerian=True)]
    base = [Problem.from_deck(d) for d in decks]
    a = [p.copy() for p in base]
    b = [_pin(p.copy(), True) if pins == "all" or i != 1 else p.copy() for i, p in enumerate(base)]
    for probs in (a, b):
        s = BatchSolver(probs, fp_mode=abi.FP_EXACT)
        first = [p.timestep.copy() for p in probs]
        assert s.run(max_steps=3)[0] == 0
        assert s.sync_to_device(0) == 0
        for p, t in zip(probs, first):
            p.timestep = t
        assert s.run(max_steps=6)[0] == 0
        assert s.sync_to_host(0) == 0
        s.close()
    for p, q in zip(a, b):
        assert not compare(p, q, exact=True)
