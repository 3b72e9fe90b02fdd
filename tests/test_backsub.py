"""Back substitution of long Krylov cycles: up to 512 unknowns are kept in
shared memory, longer cycles in global memory. A tolerance that is never
reached runs the cycle to its cap on both sides of that line; the matrix has
to be the converged one. Every further step may only lose rounding: the
1e-10-converged matrix agrees to 1e-8 of the largest entry."""

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 31, 33, 64, 511, 512, 513, 520])
def test_long_cycles(tmp_path, steps):
    path = str(tmp_path / "in.txt")
    geo.crossing_2x2().write(path)
    model = fc.Model.build(path, mesh_eps=0.01)
    assert model.n_panels >= 520
    with fc.Context(0) as ctx:
        p = ctx.problem(model, fc.PREC_FP64)
        p.fill()
        want, its = p.solve(tol=1e-10)
        c, it = p.solve(tol=1e-300, max_iter=steps, refine=-1, allow_not_converged=True)
        if steps > np.max(its):
            assert np.max(it) == steps
            assert np.max(np.abs(c - want)) <= 1e-8 * np.max(np.abs(want))
        else:  # a truncated cycle: the one of the looser tolerance that stops there
            again, _ = p.solve(tol=1e-300, max_iter=steps, refine=-1, allow_not_converged=True)
            assert np.all(np.isfinite(c)) and np.array_equal(c, again)
        p.close()
