"""FP64 far-field potentials are not biased: their relative errors against the
same quadratures in extended precision, averaged over thousands of links of a
band, stay below half a unit of 2^-53. The rounding of a link's own operations
averages out (a few units a link, some 1/sqrt(5000) of that in the mean) on
source triangles of random shape and direction; what is left is the rounding of
the constants that every link shares: the weights 1/3 and 1/6 as doubles (half a
unit low) against 1 / (4 pi eps0 points) rounded once (0.6 units low, 0.3 high
for the point formula)."""

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

pytestmark = pytest.mark.gpu

X = np.longdouble
FOUR_PI_E0 = 1.1126500559756e-10
A, B, C = 0.659027622374092, 0.231933368553031, 0.109039009072877
RULES = {  # band: points (px, py) and their weight
    1: ([(A, B), (A, C), (B, A), (B, C), (C, A), (C, B)], 1 / 6),
    2: ([(0, 0.5), (0.5, 0), (0.5, 0.5)], 1 / 3),
    3: ([(4 / 6, 1 / 6), (1 / 6, 4 / 6), (1 / 6, 1 / 6)], 1 / 3),
}


def dot(a, b):
    return (a * b).sum(axis=1)


def potentials(r, v, points, weight):
    """the quadrature of 1/|p - r| over triangles v (float sides), over their area"""
    s1, s2, s3 = ((v[:, 3:6] - v[:, 0:3]).astype(X), (v[:, 6:9] - v[:, 3:6]).astype(X), (v[:, 0:3] - v[:, 6:9]).astype(X))
    z = np.cross(s1, s2)
    mn, m1 = np.sqrt(dot(z, z)), np.sqrt(dot(s1, s1))
    x = s1 / m1[:, None]
    y = np.cross(x, z / mn[:, None])
    x02, y12 = -dot(s3, x), -dot(s3, y)
    jacobian = (x02 - m1) * y12 - y12 * x02
    total = 0
    for px, py in points:
        t = X(1) - X(px) - X(py)
        p = v[:, 0:3].astype(X) + s1 * X(px) + (x * x02[:, None] + y * y12[:, None]) * t
        total = total + X(weight) / np.sqrt(dot(p - r, p - r))
    return total * (jacobian / 2) / (mn / 2) / X(FOUR_PI_E0)


@pytest.mark.parametrize("band,lo,hi", [(1, 1.0, 2.0), (2, 2.0, 4.0), (3, 4.0, 10.0), (4, 10.0, 1e30)])
def test_unbiased(tmp_path, band, lo, hi):
    path = str(tmp_path / "in.txt")
    geo.Crossing(k=2, length=10.0, pitch=3.0, gap=1.0).write(path)
    a = {k: np.array(v) for k, v in fc.Model.build(path, mesh_eps=1e-3).arrays.items()}
    n = len(a["node_type"])
    rng = np.random.default_rng(band)
    cent = a["node_centroid"].reshape(n, 3)
    frame = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    corner = np.array([[1, 0, 0], [-0.5, 0.75**0.5, 0], [-0.5, -(0.75**0.5), 0]]) + rng.uniform(-0.2, 0.2, (n, 3, 3))
    a["node_vertices"] = (cent[:, None] + 0.5 * a["node_maxside"][:, None, None] * corner @ frame).astype(np.float32)
    row, src = rng.integers(0, n, (2, 400000))
    rho = np.linalg.norm(cent[row].astype(float) - cent[src], axis=1) / np.maximum(a["node_maxside"][row], a["node_maxside"][src])
    keep = np.flatnonzero((rho > 1.001 * lo) & (rho < 0.999 * hi))[:20000]
    assert len(keep) > 5000
    row, src = row[keep], src[keep]
    order = np.argsort(row, kind="stable")
    row, src = row[order], src[order]
    a["link_src"] = src.astype(np.int32)
    a["link_ptr"] = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int64)
    with fc.Context(0) as ctx:
        p = ctx.problem(fc.Model.from_arrays(a), fc.PREC_FP64)
        p.fill()
        got, _ = p.coefficients()
        p.close()
    if band == 4:  # the point formula at the float difference of the centroids
        d = (cent[row] - cent[src]).astype(X)
        want = 1 / (X(FOUR_PI_E0) * np.sqrt(dot(d, d)))
    else:
        want = potentials(cent[row].astype(X), a["node_vertices"].reshape(n, 9)[src], *RULES[band])
    error = (got.astype(X) - want) / want
    assert np.abs(error).max() < 1e-12  # the same bands and formulas
    assert abs(float(error.mean())) < 0.5 * 2.0**-53
