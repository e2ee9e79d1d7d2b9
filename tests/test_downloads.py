"""Point read-back: several jobs' fields in one call equal each job's own, bit
for bit, on every path (device conversion in one group, in several, and host
conversion), with chunk and thread boundaries inside the jobs."""
import os
import threading

import numpy as np
import pytest

from mpm_3d_b200 import inputs
from mpm_3d_b200.native import POINT_FIELDS, GPUBatch, GPUExplicitUSL, MpmGpuError
from util import bits_equal

pytestmark = pytest.mark.gpu

GENERAL = [f for f in POINT_FIELDS if f not in ("L", "gammap", "gammap_dot")]


def _cloud(dim, n_points, seed, material="IsotropicLinearElasticity"):
    """n_points points at random in the inner part of a 48^dim grid."""
    rng = np.random.default_rng(seed)
    x, v = np.zeros((n_points, 3)), np.zeros((n_points, 3))
    x[:, :dim] = rng.uniform(0.2, 0.8, (n_points, dim))
    v[:, :dim] = rng.uniform(-1.0, 1.0, (n_points, dim))
    vol = (1.0 / 96) ** dim
    body = inputs.Body("cloud", np.full(n_points, 1000 * vol), np.full(n_points, vol), x, v,
                       np.ones(n_points, np.int32), material_class=material)
    return inputs.Case("cloud", dim, (1.0,) * dim, (48,) * dim, 1e-6, 100, [body])


# x, T: 0.8 and 2.3 M values in all, i.e. one and three chunks of 2^20
SIZES = (1, 7, 4096, 33, 200_000, 27_001, 2, 25_000)


@pytest.mark.parametrize("dim,mode", [(3, "fp64"), (3, "mixed"), (2, "fp64")])
def test_many_jobs_equal_each_job(dim, mode):
    batch = GPUBatch(dim=dim, mode=mode)
    ids = [batch.add(_cloud(dim, n, 100 + n)) for n in SIZES]
    batch.step(3)
    order = ids[::-1] + ids[2:4]    # any order, and a job twice
    for f in GENERAL:
        alone = {j: batch.points(j, 0, f) for j in ids}
        for threads in (1, 3, 64):
            for got, j in zip(batch.points_many(order, 0, f, threads=threads), order):
                assert bits_equal(got, alone[j]), f"{f}, {threads} threads, job {j}"
    assert batch.points_many([], 0, "x") == []
    # the same in groups of one or a few jobs, and converted on the host: with
    # 16 MB each job fits and all together do not, with 1 MB the largest does
    # not, and with 0 none does
    for limit in (16 << 20, 1 << 20, 0):
        for f in GENERAL:
            alone = {j: batch.points(j, 0, f) for j in ids}
            batch.set_download_limit(limit)
            for threads in (1, 3):
                for got, j in zip(batch.points_many(order, 0, f, threads=threads), order):
                    assert bits_equal(got, alone[j]), f"{f}, limit {limit}, {threads} threads, job {j}"
            for j in ids:
                assert bits_equal(batch.points(j, 0, f), alone[j]), f"{f}, limit {limit}, job {j} alone"
            batch.set_download_limit(-1)
    batch.close()


def test_fields_of_debug_and_granular_bodies():
    batch = GPUBatch(dim=3, mode="fp64", keep_debug=True)
    sand = inputs.sand_column(3, n_cells=12, steps=30)
    job = batch.add(sand)
    batch.step(20)
    for f in ("L", "gammap", "gammap_dot", "T"):
        device = batch.points(job, 0, f)
        assert np.abs(device).max() > 0.0
        batch.set_download_limit(0)
        assert bits_equal(batch.points(job, 0, f), device), f
        batch.set_download_limit(-1)
    batch.close()


def test_download_is_refused_while_the_stream_is_captured():
    """The call waits for its copies, so a captured stream cannot serve it: an
    error, nothing queued, and the capture stays valid."""
    torch = pytest.importorskip("torch")
    sim = GPUExplicitUSL(inputs.two_body_collision_3d(16, steps=2, gap=0.01))
    sim.step(1)
    want = sim.points(0, "x")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(sim.stream())):
        graph.capture_begin()
        try:
            for f in ("x", "T", "b"):
                with pytest.raises(MpmGpuError, match="captured"):
                    sim.points(0, f)
        finally:
            graph.capture_end()
    del graph
    assert bits_equal(sim.points(0, "x"), want)
    sim.close()


def test_download_threads_are_bounded():
    """However many threads a caller asks for, at most 8 copy a field out (the
    caller's own is one of them)."""
    batch = GPUBatch(dim=3, mode="fp64")
    job = batch.add(_cloud(3, 600_000, 1))
    batch.step(1)
    batch.synchronize()
    tasks = lambda: len(os.listdir("/proc/self/task"))
    seen, stop = [], threading.Event()

    def watch():
        while not stop.is_set():
            seen.append(tasks())

    watcher = threading.Thread(target=watch)
    watcher.start()
    batch.points_many([job], 0, "T", threads=1)   # what the first call of a process starts
    before = tasks()
    seen.clear()
    for _ in range(3):
        batch.points_many([job], 0, "T", threads=64)
    stop.set()
    watcher.join()
    batch.close()
    assert max(seen) <= before + 7, f"{max(seen) - before} threads beside the caller"
