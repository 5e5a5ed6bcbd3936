"""The step kernels' L2 prefetch (csrc/lbm_device.cuh, prefetch_rows) on lattices large enough to take it.

A prefetch changes no value, so a lattice that takes it equals the same lattice in z-slabs, which are
too small for it, bit for bit, at odd extents (rows and directions that start at any byte, a last row
without a successor); the FP16 two-cell kernel equals the one-cell kernel, which has none; and the
reverse sweep over frames that take it does not depend on the checkpoint interval."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_slabs import sliced, whole

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice, storage, shape", [("d3q19", "fp32", (131, 97, 150)), ("d3q27", "fp32", (133, 100, 96)),
                                                     ("d3q19", "fp64", (90, 97, 105)), ("d3q27", "fp64", (77, 78, 105)),
                                                     ("d3q19", "fp32", (33, 250, 230))])  # rows too short for it
def test_prefetch_equals_slabs(engine, lattice, storage, shape):
    cs = engine
    nx, ny, nz = shape
    q, es = {"d3q19": 19, "d3q27": 27}[lattice], {"fp32": 4, "fp64": 8}[storage]
    assert q * es * nx * ny * nz > 126 << 20  # the whole lattice takes the prefetch, thirds of it do not
    rng = np.random.default_rng(1)
    flags = (rng.uniform(size=(nz, ny, nx)) < 0.05).astype(np.uint8).reshape(-1)
    cfg = cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.6, lattice=lattice, storage=storage, collision="trt")
    a = whole(cs, cfg, {"flags": flags}, 3)
    b = sliced(cfg, {"flags": flags}, 3, 3)
    assert np.array_equal(a[0], b[0])
    for u, v in zip(a[2], b[2]):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("shape", [(140, 139, 190), (1002, 60, 62)])
def test_prefetch_in_the_two_cell_kernel(engine, shape):
    cs = engine
    assert 38 * np.prod(shape) > 126 << 20
    out = []
    for variant in (0, 1):
        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=shape[0], ny=shape[1], nz=shape[2], tau=0.6,
                                                           storage="fp16s")) as s:
            s.set_launch_shape(0, 0, variant)
            s.initialize_taylor_green(0.04)
            s.step(4)
            out.append(s.logical_populations())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("lattice, storage", [("d3q19", "fp32"), ("d3q27", "fp16s")])
def test_prefetch_in_the_reverse_sweep(engine, lattice, storage):
    cs = engine
    nx, ny, nz = 131, 75, 62  # frames of 8 bytes past a multiple of 16, rows of more than 512 bytes
    n = nx * ny * nz
    rng = np.random.default_rng(2)
    ns = rng.uniform(0, 0.2, n).astype(np.float32)
    seeds = [rng.normal(size=n).astype(np.float32) for _ in range(3)]
    got = []
    for interval in (6, 4):
        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.7, lattice=lattice, storage=storage,
                                                           collision="trt")) as s:
            s.set_solid_fraction(ns)
            s.initialize_taylor_green(0.04)
            s.adjoint_forward(6, interval)
            got.append(s.adjoint_backward(*seeds))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
