"""Device memory of a model's construction, as the high-water mark of the
device's memory pool. The peak is the links' placement: every pair test of the
traversal then holds its two elements (8 bytes), its place in the next level
(4), its link count (8) and half of an emitted pair (4). Beside these 24 bytes
a test, the levels may have 32 MB of unused room (48 with what small groups of
levels are given at once), and the hierarchy holds about 300 bytes a node."""

import ctypes as C

import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CUmemPool_attribute


class Pool:
    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, self.pool = C.c_int(), C.c_void_p()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetMemPool(C.byref(self.pool), dev) == 0

    def get(self, attribute):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, attribute, C.byref(v)) == 0
        return v.value

    def reset_high(self):
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(C.c_uint64(0))) == 0


def build_peak(path, **options):
    """bytes held at the most, pair tests and nodes of a build on the device"""
    with fc.Context(0) as ctx:
        pool = Pool()
        base = pool.get(USED_CURRENT)
        pool.reset_high()
        m = fc.Model.build(path, ctx=ctx, **options)
        peak = pool.get(USED_HIGH) - base
        nc = len(m.arrays["cond_is_diel"])
        roots = nc * (nc - 1) // 2 + m.n_panels - nc  # the conductors' pairs and every split's
        return peak, m.n_links - roots, m.n_nodes


@pytest.mark.parametrize("mesh,eps_ratio", [(1e-3, 1.0), (3e-4, 1.0), (1e-3, 0.2)])
def test_traversal(tmp_path, mesh, eps_ratio):
    path = str(tmp_path / "in.txt")
    geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(path)
    peak, tests, nodes = build_peak(path, mesh_eps=mesh, eps_ratio=eps_ratio)
    # and the elements' arrays, which grow by 2^20 elements or to twice their size
    elements = 96 * max(2 * nodes, nodes + (1 << 20))
    assert peak <= 24 * tests + (48 << 20) + 300 * nodes + elements


@pytest.mark.parametrize("mesh,eps_ratio", [(1e-3, 1.0), (6e-4, 1.0), (1e-3, 0.2)])
def test_elements_beside_the_links(tmp_path, mesh, eps_ratio):
    """the refined elements' room for growth (100 MB and more) is gone by then"""
    path = str(tmp_path / "in.txt")
    geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(path)
    peak, tests, nodes = build_peak(path, mesh_eps=mesh, eps_ratio=eps_ratio)
    assert peak <= 24 * tests + (48 << 20) + 300 * nodes
