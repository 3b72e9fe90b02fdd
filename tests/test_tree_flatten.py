"""Models flattened on the device (hierarchies of 8192 elements and more)
against the host builder: many conductors, one conductor, conductors of one
panel (bisected first), dielectric interfaces, lopsided trees whose depth is
several times that of a balanced one, and sizes on both sides of the line.
The arrays have to be the host builder's, bit for bit; and a file job, whose
model never leaves the device, has to give the capacitances of a problem made
from the host's arrays."""

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

pytestmark = pytest.mark.gpu


def quad(name, x, y, z, a, b):
    return "Q %s %g %g %g %g %g %g %g %g %g %g %g %g\n" % (name, x, y, z, x + a, y, z, x + a, y + b, z, x, y + b, z)


def write(shape, path):
    if shape == "crossing":
        geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(path)
    elif shape == "slab":
        geo.Crossing(k=2, length=10.0, pitch=3.0, gap=1.0, eps_r=3.9, slab=(4.0, 1.0, 3.9, 15.0)).write(path)
    else:
        with open(path, "w") as f:
            f.write("0 %s\n" % shape)
            if shape == "one panel each":
                for k in range(4):
                    f.write(quad("p%d" % k, 0.3 * k, 0, 0.25 * k, 1 + k, 1))
            elif shape == "one conductor":
                f.write(quad("p", 0, 0, 0, 1, 1) + quad("p", 0, 0, 0.5, 1, 2))
            else:  # "lopsided": panels that halve towards the origin
                for k in range(24):
                    f.write(quad("a", 2.0 ** -k, 0, 0, 2.0 ** -(k + 1), 2.0 ** -(k + 1)))
                    f.write(quad("b", 2.0 ** -k, 0, 0.3, 2.0 ** -(k + 1), 2.0 ** -(k + 1)))


SHAPES = [("crossing", (1e-2, 4e-3, 6e-4)), ("slab", (1e-4,)), ("one panel each", (1e-2, 2e-3)),
          ("one conductor", (3e-3, 2e-3)), ("lopsided", (1e-2,))]


@pytest.mark.parametrize("shape,mesh", [(s, m) for s, ms in SHAPES for m in ms])
def test_same_arrays_as_the_host(tmp_path, shape, mesh):
    path = str(tmp_path / "in.txt")
    write(shape, path)
    host = fc.Model.build(path, mesh_eps=mesh)
    with fc.Context(0) as ctx:
        dev = fc.Model.build(path, mesh_eps=mesh, ctx=ctx)
    assert dev.names == host.names
    for name in host.arrays:
        assert np.array_equal(dev.arrays[name], host.arrays[name]), name
    for key in ("max_level", "max_mesh_eps", "n_links"):
        assert dev.info[key] == host.info[key], key


@pytest.mark.parametrize("precision", [fc.PREC_MIXED, fc.PREC_FP64])
@pytest.mark.parametrize("shape,mesh", [("crossing", 1e-2), ("crossing", 1e-3), ("slab", 1e-4)])
def test_file_job_of_a_device_model(tmp_path, shape, mesh, precision):
    path = str(tmp_path / "in.txt")
    write(shape, path)
    host = fc.Model.build(path, mesh_eps=mesh)
    with fc.Context(0) as ctx, ctx.server(slots=2) as srv:
        want, steps = srv.submit(host, precision, tol=1e-4).result()
        jobs = [srv.submit_file(path, precision, tol=1e-4, mesh_eps=mesh) for _ in range(3)]
        for j in jobs:
            got, it = j.result()
            assert np.array_equal(got, want) and np.array_equal(it, steps)
            assert j.info["n_panels"] == host.n_panels and j.info["n_links"] == host.n_links
        assert srv.stats()["in_use"] == 0
