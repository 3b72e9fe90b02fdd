"""A file job that waits for admission holds its link sources in device memory
(4 bytes a link, before any footprint is counted) and no more: its node arrays,
102 bytes a node, wait in host memory. Admitted later, it gives the bits it
gives alone."""

import time

import numpy as np
import pytest

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo
from test_build_memory import USED_CURRENT, Pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fc.PREC_MIXED, fc.PREC_FP64])
def test_waiting_job(tmp_path, precision):
    small, large = str(tmp_path / "small.txt"), str(tmp_path / "large.txt")
    geo.crossing_2x2().write(small)
    geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(large)
    options = dict(precision=precision, tol=1e-2, mesh_eps=4.2e-4, eps_ratio=100.0)  # many nodes, few links
    with fc.Context(0) as ctx:
        pool = Pool()
        with ctx.server(slots=1) as srv:
            alone, steps = srv.submit_file(large, **options).result()
        base = pool.get(USED_CURRENT)
        with ctx.server(slots=2, memory_budget=1) as srv:
            # a solve that goes on until it is cancelled
            first = srv.submit(fc.Model.build(small, mesh_eps=0.01), fc.PREC_FP64, tol=1e-300, refine=1 << 20)
            while not first.poll()["state"] == fc.JOB_RUNNING:
                time.sleep(0.001)
            job = srv.submit_file(large, **options)
            deadline = time.time() + 30
            while job.poll()["build_ms"] == 0 and time.time() < deadline:
                time.sleep(0.001)
            time.sleep(0.5)
            info, held = job.poll(), pool.get(USED_CURRENT) - base
            assert first.poll()["state"] == fc.JOB_RUNNING and info["state"] == fc.JOB_RUNNING
            assert srv.stats()["in_use"] == first.poll()["footprint_bytes"]  # the job waits
            first.cancel()
            cap, its = job.result()
            with pytest.raises(fc.FCError):
                first.result()
            own = first.info["device_bytes"]
        assert info["n_panels"] > 90000 and held >= 4 * info["n_links"]
        # pool blocks are multiples of 512 bytes
        assert held <= own + 4 * info["n_links"] + (1 << 20)
        assert np.array_equal(cap, alone) and np.array_equal(its, steps)


@pytest.mark.parametrize("mesh", [1e-2, 1e-3])
def test_jobs_one_at_a_time(tmp_path, mesh):
    """every job but the first waits, on both sides of the device flattening's line"""
    path = str(tmp_path / "in.txt")
    geo.Crossing(k=8, length=30.0, pitch=3.0, gap=1.0).write(path)
    with fc.Context(0) as ctx:
        with ctx.server(slots=1) as srv:
            alone, steps = srv.submit_file(path, fc.PREC_MIXED, tol=1e-3, mesh_eps=mesh).result()
        with ctx.server(slots=4, memory_budget=1) as srv:
            jobs = [srv.submit_file(path, fc.PREC_MIXED, tol=1e-3, mesh_eps=mesh) for _ in range(6)]
            jobs[-1].cancel()
            for j in jobs[:-1]:
                cap, its = j.result()
                assert np.array_equal(cap, alone) and np.array_equal(its, steps)
            assert srv.stats()["in_use"] == 0
