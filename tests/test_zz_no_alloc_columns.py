"""The no-allocation product runs the kernels of the ordinary one at every
number of right-hand sides, padded ones among them: the same bits, per call and
recorded into a graph."""

import numpy as np
import pytest

import fastercap_gb300 as fc
from conftest import load_golden, model_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fc.PREC_FP64, fc.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 32])
def test_same_bits_as_the_allocating_product(precision, k):
    torch = pytest.importorskip("torch")
    with fc.Context(0) as ctx:
        s = torch.cuda.Stream()
        p = ctx.problem(fc.Model.from_arrays(model_arrays(load_golden("random3"))), precision, stream=s.cuda_stream)
        p.fill()
        q = torch.tensor(np.random.default_rng(k).uniform(-1, 1, (k, p.n_panels)), dtype=torch.float64, device="cuda")
        want, got = torch.empty_like(q), torch.full_like(q, float("nan"))
        torch.cuda.synchronize()
        p.matvec_device(q.data_ptr(), want.data_ptr(), k)
        assert p.matvec_device_noalloc(q.data_ptr(), got.data_ptr(), k) == fc.NORMAL_END, fc.last_error()
        assert torch.equal(got, want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            assert p.matvec_device_noalloc(q.data_ptr(), got.data_ptr(), k) == fc.NORMAL_END, fc.last_error()
        got.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        p.close()


def test_scratch_holds_the_padded_columns_only(tmp_path):
    """FP64, six columns of a model whose eight would not fit: accepted."""
    torch = pytest.importorskip("torch")
    from fastercap_gb300 import geometry as geo
    path = str(tmp_path / "in.txt")
    geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(path)
    with fc.Context(0) as ctx:
        m = fc.Model.build(path, mesh_eps=4.2e-4, eps_ratio=100.0, ctx=ctx)
        assert m.n_nodes * 6 * 24 <= (32 << 20) - 3 * 256 and m.n_nodes * 8 * 24 > 32 << 20
        p = ctx.problem(m, fc.PREC_FP64)
        p.fill()
        q = torch.tensor(np.random.default_rng(1).uniform(-1, 1, (6, p.n_panels)), dtype=torch.float64, device="cuda")
        want, got = torch.empty_like(q), torch.full_like(q, float("nan"))
        torch.cuda.synchronize()
        p.matvec_device(q.data_ptr(), want.data_ptr(), 6)
        assert p.matvec_device_noalloc(q.data_ptr(), got.data_ptr(), 6) == fc.NORMAL_END, fc.last_error()
        assert torch.equal(got, want)
        assert p.matvec_device_noalloc(q.data_ptr(), got.data_ptr(), 8) == fc.OUT_OF_MEMORY
        p.close()
