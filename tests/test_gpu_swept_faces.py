"""The device loop's remap takes a face's swept volume from the element across
it; where the two elements do not hold the same face (connectivity that only
one side has, a face run the same way by both) each must take its own, as the
called step does: the same bits either way."""
import numpy as np
import pytest

from bookleaf_f90_gb300 import Problem, Solver, abi, configs
from helpers import compare

pytestmark = pytest.mark.gpu


def _one_sided(p, seed):
    """Some interior elements' faces 2 and 3 (1-based) lead to a face 1 or 4
    of an element elsewhere, which does not lead back."""
    r = np.random.default_rng(seed)
    el, fc = p.fields[abi.IELEL], p.fields[abi.IELFC]
    inner = np.nonzero(np.all(el != np.arange(1, p.nel + 1)[:, None], axis=1))[0]
    for e in r.choice(inner, 4, replace=False):
        j = int(r.integers(1, 3))
        el[e, j] = 1 + int(r.integers(0, p.nel))
        if el[e, j] == e + 1:
            el[e, j] = el[e, 0]
        fc[e, j] = 1 if r.integers(0, 2) else 4


@pytest.mark.parametrize("fp", [abi.FP_FAST, abi.FP_MIXED, abi.FP_EXACT],
                         ids=["fast", "mixed", "exact"])
@pytest.mark.parametrize("deck", ["blast", "tube"])
def test_loop_equals_calls_on_one_sided_faces(deck, fp):
    base = Problem.from_deck(configs.sedov(12, eulerian=True, kappa=0.01) if deck == "blast"
                             else configs.sod(33, 3, eulerian=True))
    f = base.fields
    x, y = f[abi.NDX] / f[abi.NDX].max(), f[abi.NDY] / f[abi.NDY].max()
    f[abi.NDU] += 0.3 * x * (1.0 - x) + 0.1 * x * y
    f[abi.NDV] += 0.2 * y * (1.0 - y) - 0.1 * x * y
    _one_sided(base, 3)
    pa, pb = base.copy(), base.copy()
    sa, sb = Solver(pa, fp_mode=fp), Solver(pb, fp_mode=fp)
    for _ in range(3):
        assert sa.step() == 0
    assert sb.run(max_steps=3, history=False)[0] == 0
    sa.sync_to_host(0)
    sb.sync_to_host(0)
    sa.close()
    sb.close()
    assert np.all(np.isfinite(pa.fields[abi.ELENERGY]))
    assert not compare(pa, pb, exact=True)
