"""Solves stopped at an iteration cap against the same Krylov iterate from an
independent least-squares solution: the charges x0 + D^-1 Q y with Q an
orthonormal basis of the cap's Krylov space (Arnoldi with a second
orthogonalisation) and y the minimiser of |r0 - A D^-1 Q y|, on the oracle's
product with the problem's own coefficients. A cap stops before convergence, so
that an error in the last rotation, in the right-hand side it turns or in the
back substitution of a short cycle shows at the size of the residual left.

The iterate answers a change of the operator by about as much (the operator's
condition on the spaces is below 300). FP64: classical orthogonalisation loses up
to 1e-12 here (measured on the same steps in NumPy); held to 1e-10 of the
charges' norm, the residuals left at 31 to 33 steps being 1e-9 to 1e-3. Mixed:
the charges and row sums of a product are FP32, 6e-8 each, and an operator
perturbed by that moves the iterates by 3e-7; held to 3e-6 (the slab's residuals
there: 4e-4 and more)."""

import os
import sys

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
from pyoracle import Oracle  # noqa: E402

pytestmark = pytest.mark.gpu

CUTS = (1, 2, 5, 31, 32, 33, 40, 64)


@pytest.fixture(scope="module", params=[1, 2, 3, "slab"], ids=["two-solves", "four-solves", "six-solves", "slab"])
def case(request, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("m") / "crossing.txt")
    if request.param == "slab":
        geo.Crossing(k=2, length=10.0, pitch=3.0, gap=1.0, eps_r=3.9, slab=(4.0, 1.0, 3.9, 15.0)).write(path)
        model = fc.Model.build(path, mesh_eps=2e-3)
    else:
        geo.Crossing(k=request.param, length=12.0, pitch=3.0, gap=1.0).write(path)
        model = fc.Model.build(path, mesh_eps=0.005)
    return model, Oracle(model.arrays)


def iterates(oracle, coef, self_coef, b, precond, cuts):
    """charges after cut Arnoldi steps for every cut, and the residuals left"""
    d = self_coef if precond == fc.PRECOND_JACOBI else np.ones_like(b)

    def product(x):
        return oracle.matvec(x, coef, self_coef)

    x0 = b / d if precond == fc.PRECOND_JACOBI else np.zeros_like(b)
    r0 = b - product(x0)
    q, w, out = [r0 / np.linalg.norm(r0)], [], {}
    for step in range(1, max(cuts) + 1):
        w.append(product(q[-1] / d))
        v = w[-1].copy()
        for _ in range(2):
            v -= np.array(q).T @ (np.array(q) @ v)
        q.append(v / np.linalg.norm(v))
        if step in cuts:
            y, _, _, s = np.linalg.lstsq(np.array(w).T, r0, rcond=None)
            assert s[0] < 300 * s[-1]
            left = np.linalg.norm(r0 - np.array(w).T @ y) / np.linalg.norm(b)
            out[step] = x0 + np.array(q[:step]).T @ y / d, left
    return out


@pytest.mark.parametrize("precision,bound", [(fc.PREC_FP64, 1e-10), (fc.PREC_MIXED, 3e-6)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("precond", [fc.PRECOND_NONE, fc.PRECOND_JACOBI])
def test_iterates(case, precision, bound, precond):
    model, oracle = case
    a = model.arrays
    with fc.Context(0) as ctx:
        p = ctx.problem(model, precision)
        p.fill()
        coef, self_coef = p.coefficients()
        want = []
        for c in np.flatnonzero(a["cond_is_diel"] == 0):
            b = np.zeros(model.n_panels)
            b[a["cond_leaf_first"][c]:a["cond_leaf_first"][c] + a["cond_leaf_count"][c]] = 1.0
            want.append(iterates(oracle, coef, self_coef, b, precond, CUTS))
        if precond == fc.PRECOND_NONE:  # the passes' edges lie before convergence
            assert min(it[33][1] for it in want) > 1e-9
        for cut in CUTS:
            _, its = p.solve(tol=1e-300, precond=precond, max_iter=cut, refine=-1, allow_not_converged=True)
            assert np.all(its == cut)
            for got, it in zip(p.charges(), want):
                assert np.linalg.norm(got - it[cut][0]) <= bound * np.linalg.norm(it[cut][0])
        p.close()
