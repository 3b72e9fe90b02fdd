"""FP64 far-field coefficients against the oracle's reference-order formulas:
every distance band in random mixtures (full and part-full evaluation queues),
conductor and dielectric evaluation panels, geometry from nanometres to tens of
kilometres.

Both sides evaluate the same few tens of FP64 operations in another order, on
differences of absolute coordinates of size R: a value at distance r is within
64 (1 + R / r) units of 2^-53 of its scale, 1/r for a potential and 1/r^2 for a
field (over 4 pi eps0).
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

FOUR_PI_E0 = 1.1126500559756e-10


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("m") / "slab.txt")
    geo.Crossing(k=2, length=10.0, pitch=3.0, gap=1.0, eps_r=3.9, slab=(4.0, 1.0, 3.9, 15.0)).write(path)
    return {k: np.array(v) for k, v in fc.Model.build(path, mesh_eps=1e-4).arrays.items()}


@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e4])
@pytest.mark.parametrize("links", [1, 33, 20000])
def test_far_bands(built, scale, links):
    a = dict(built)
    for name, power in (("node_vertices", 1), ("node_centroid", 1), ("node_area", 2), ("node_maxside", 1)):
        a[name] = (a[name].astype(np.float64) * scale**power).astype(a[name].dtype)
    n = len(a["node_type"])
    rng = np.random.default_rng(links)
    row, src = rng.integers(0, n, (2, 40 * links))
    cent = a["node_centroid"].astype(np.float64)
    dist = np.linalg.norm(cent[row] - cent[src], axis=1)
    rho = dist / np.maximum(a["node_maxside"][row], a["node_maxside"][src])
    far = rho > 1.001
    row, src, dist, rho = row[far][:links], src[far][:links], dist[far][:links], rho[far][:links]
    order = np.argsort(row, kind="stable")
    row, src, dist, rho = row[order], src[order], dist[order], rho[order]
    a["link_src"] = src.astype(np.int32)
    a["link_ptr"] = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int64)
    ref, _ = Oracle(a).fill()
    with fc.Context(0) as ctx:
        p = ctx.problem(fc.Model.from_arrays(a), fc.PREC_FP64)
        p.fill()
        got, _ = p.coefficients()
        p.close()
    field = (a["node_type"][row] & fc.IS_DIEL) != 0
    if links > 1000:
        for lo, hi in ((1, 2), (2, 4), (4, 10), (10, 1e30)):  # every band, both kinds
            for kind in (False, True):
                assert np.any((rho > lo) & (rho < hi) & (field == kind))
    size = np.abs(cent).max()
    bound = 64 * 2.0**-53 * (1 + size / dist) / np.where(field, dist**2, dist) / FOUR_PI_E0
    assert np.all(np.abs(got - ref) <= bound)
