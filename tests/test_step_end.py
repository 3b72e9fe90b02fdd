"""The end of an Arnoldi step (norms, Givens rotations, convergence test) on
solves long enough for its passes of 32 rotations: one past them, two and a
remainder, and an iteration cap; a few solves end their steps in the update's
last block, more than four in a kernel of their own.

FP64 against the oracle: the same iteration counts, and matrices that agree to
the solves' own convergence (tolerance 1e-9 relative residual; capped solves are
the same Krylov iterate up to FP64 rounding, 1e-6 as the FP64 path is held to
everywhere).
"""

import os
import sys

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
from pyoracle import Oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1, 2, 3], ids=["two-solves", "four-solves", "six-solves"])
def case(request, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("m") / "crossing.txt")
    geo.Crossing(k=request.param, length=12.0, pitch=3.0, gap=1.0).write(path)
    model = fc.Model.build(path, mesh_eps=0.005)
    oracle = Oracle(model.arrays)
    oracle.fill()
    return model, oracle


@pytest.mark.parametrize("precond", [fc.PRECOND_NONE, fc.PRECOND_JACOBI])
def test_long_solves(case, precond):
    model, oracle = case
    cap, its, _, _ = oracle.solve(1e-9, precond)
    with fc.Context(0) as ctx:
        p = ctx.problem(model, fc.PREC_FP64)
        p.fill()
        got, gits = p.solve(tol=1e-9, precond=precond)
        assert list(gits) == list(its)
        assert np.max(np.abs(got - cap) / np.abs(np.diag(cap)).max()) < 1e-6
        for cut in (31, 32, 33):
            part, pits = p.solve(tol=1e-9, precond=precond, max_iter=cut, allow_not_converged=True)
            assert list(pits) == [min(cut, n) for n in its]
        p.close()


def test_lengths_cover_the_passes(case):
    model, oracle = case
    assert max(oracle.solve(1e-9, fc.PRECOND_NONE)[1]) > 32
