"""Device mesh refinement and link construction against the host builder at
sizes around the groups of levels that run without the host: from models whose
refinement fits one group to frontiers larger than a group allows, with the
FP32 pre-test and without it, in vacuum and with a dielectric interface. The
arrays have to be the host builder's, bit for bit."""

import os

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

pytestmark = pytest.mark.gpu


def write(shape, path):
    if shape == "vacuum":
        geo.crossing_2x2().write(path)
    else:
        geo.Crossing(k=2, length=10.0, pitch=3.0, gap=1.0, eps_r=3.9, slab=(4.0, 1.0, 3.9, 15.0)).write(path)


@pytest.mark.parametrize("fp64_only", [False, True])
@pytest.mark.parametrize("shape,mesh", [("vacuum", m) for m in (0.3, 0.05, 0.01, 4e-3, 1.5e-3, 6e-4)] +
                         [("slab", m) for m in (1e-2, 1e-3, 2e-4, 6e-5)])
def test_same_arrays_as_the_host(tmp_path, monkeypatch, shape, mesh, fp64_only):
    path = str(tmp_path / "in.txt")
    write(shape, path)
    host = fc.Model.build(path, mesh_eps=mesh)
    if fp64_only:
        monkeypatch.setenv("FCG_MESH_FP64", "1")
    with fc.Context(0) as ctx:
        dev = fc.Model.build(path, mesh_eps=mesh, ctx=ctx)
    assert dev.names == host.names
    for name in host.arrays:
        assert np.array_equal(dev.arrays[name], host.arrays[name]), name
    for key in ("max_level", "max_mesh_eps", "n_links"):
        assert dev.info[key] == host.info[key], key
