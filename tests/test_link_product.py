"""The link product at every right-hand-side width and every row length from
an empty row to several passes of a warp's link slots, with their remainders.

The panels are a built model's, its links are replaced by rows of 0, 1, 2, ...
links to random sources, so that each width meets every remainder. Checked
against the oracle's product with the same coefficients. Mixed precision's
tolerance per value: a charge rounds once, a group's sum of at most four
products four times, and the compensated sums and FP32-pair sweeps stay well
below one more, so 8 half-ulps of FP32 of the sum of the terms' magnitudes
(the oracle's product of the magnitudes) bound it; FP64 rounds once per term of
rows of at most MAX_ROW links and of the sweeps.
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

MAX_ROW = 300


@pytest.fixture(scope="module")
def arrays(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("m") / "crossing.txt")
    geo.crossing_2x2().write(path)
    a = {k: np.array(v) for k, v in fc.Model.build(path, mesh_eps=0.01).arrays.items()}
    n = len(a["node_type"])
    rng = np.random.default_rng(5)
    count = np.arange(n) % (MAX_ROW + 1)
    rng.shuffle(count)
    row = np.repeat(np.arange(n), count)
    src = rng.integers(0, n - 1, len(row))
    a["link_src"] = (src + (src >= row)).astype(np.int32)  # any node but the row's own
    a["link_ptr"] = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    return a


@pytest.fixture(scope="module")
def problems(arrays):
    with fc.Context(0) as ctx:
        out = {}
        for prec in (fc.PREC_MIXED, fc.PREC_FP64):
            p = ctx.problem(fc.Model.from_arrays(arrays), prec)
            p.fill()
            out[prec] = (p, p.coefficients())
        yield out
        for p, _ in out.values():
            p.close()


@pytest.mark.parametrize("precision", [fc.PREC_MIXED, fc.PREC_FP64])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 13, 14, 16, 17, 18, 20, 21, 22, 24, 26, 28, 29, 30, 32])
def test_every_width_and_row_length(arrays, problems, precision, k):
    p, (coef, self_coef) = problems[precision]
    oracle = Oracle(arrays)
    q = np.random.default_rng(k).uniform(-1.0, 1.0, (k, p.n_panels))
    v = p.matvec(q)
    for r in range(k):
        ref = oracle.matvec(q[r], coef, self_coef)
        size = oracle.matvec(np.abs(q[r]), np.abs(coef), np.abs(self_coef))
        bound = 8 * 2.0**-24 if precision == fc.PREC_MIXED else (MAX_ROW + 64) * 2.0**-53
        assert np.all(np.abs(v[r] - ref) <= bound * size), "column %d of %d" % (r, k)
