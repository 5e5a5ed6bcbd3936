"""Particles that gather in few cells (csrc/resident.cu, cell_group): the lanes of a warp that share a cell add
their sum once.  Results against the float32 restatement for groups of every size within a warp, and the
time of a gathered cloud against a scattered one."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_resident import device_read

pytestmark = pytest.mark.gpu

COUNT = 3 * 32 + 13  # a last warp of 13 lanes


def cells_of(kind, shape, rng):
    """Cell of each particle: which lanes of a warp share one."""
    nx, ny, nz = shape
    one = {"even": (2, 1, 1), "odd": (3, 1, 1), "last": (nx - 1, ny - 1, nz - 1), "next-to-last": (nx - 2, 0, nz - 1)}
    if kind in one:
        return np.tile(one[kind], (COUNT, 1))
    if kind == "stray":  # one lane of each warp elsewhere, the first lane among them
        c = np.tile((2, 1, 1), (COUNT, 1))
        c[[0, 45, 95, 100]] = (4, 2, 0)
        return c
    if kind == "interleaved":  # groups of 1, 2, 3, ... lanes, interleaved
        sizes = np.repeat(np.arange(15), np.arange(1, 16))[:COUNT]
        rng.shuffle(sizes)
        return np.stack([sizes % nx, sizes // nx % ny, np.zeros_like(sizes)], 1)
    return np.stack([rng.integers(0, e, COUNT) for e in (3, 2, 1)], 1)  # random over six cells


@pytest.mark.parametrize("shape", [(12, 5, 4), (11, 5, 4)], ids=["even-nx", "odd-nx"])
@pytest.mark.parametrize("kind", ["even", "odd", "last", "next-to-last", "stray", "interleaved", "random"])
def test_shared_cells_spread_the_same_force(engine, oracle_mod, shape, kind):
    """Every particle is slower than the flow in each component, so a cell's terms have one sign
    and n additions in any order lie within n ulps of their sum: 2 n 2^-24 between two orders."""
    from cfd_solvers_b200.multiphysics import ParticleVector3, ResidentParticles3D

    cs, O = engine, oracle_mod
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(7)
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.7)) as flow:
        flow.initialize_fields(np.ones(n), *(rng.uniform(0.02, 0.1, n) for _ in range(3)))
        macro, f = flow.refresh_device_macroscopic(), flow.compute_macroscopic()
        force = flow.device_local_acceleration(clear=True)
        flow.wait()
        rec = np.zeros((COUNT, 8))
        rec[:, :3] = cells_of(kind, shape, rng) + rng.uniform(0.01, 0.99, (COUNT, 3))
        rec[:, 3:6] = rng.uniform(-0.1, -0.02, (COUNT, 3))
        rec[:, 6], rec[:, 7] = rng.uniform(0.5, 2, COUNT), rng.uniform(0.3, 3, COUNT)
        with ResidentParticles3D(flow, COUNT) as parts:
            parts.upload(rec)
            parts.advance(macro, force, 0.5, True, ParticleVector3(0.0, -2e-4, 0.0))
            st, acc = O.particles_advance(rec.T.astype(np.float32), (f.ux, f.uy, f.uz), [np.zeros(n, np.float32)] * 3,
                                          nx, ny, nz, 0.5, True, (0.0, -2e-4, 0.0))
            assert np.array_equal(parts.download_records()[:, :6].T.astype(np.float32), st[:6])
            for ptr, e in zip((force.ax, force.ay, force.az), acc):
                assert np.all(np.abs(device_read(ptr, n) - e) <= 2 * COUNT * 2.0 ** -24 * np.abs(e))


@pytest.mark.parametrize("nx", [128, 127])
def test_gathered_particles_do_not_queue(engine, nx):
    """2^18 particles at random over two or eight cells: warps hold every cell, so a sum for warps
    in one cell alone does not apply, and an addition per particle queues at the cells' addresses."""
    import torch
    from cfd_solvers_b200.multiphysics import ParticleVector3, ResidentParticles3D

    cs = engine
    count, shape = 1 << 18, (nx, 128, 128)
    rng = np.random.default_rng(1)
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=128, nz=128, tau=0.7)) as flow:
        flow.initialize_uniform()
        macro = flow.refresh_device_macroscopic()
        force = flow.device_local_acceleration(clear=True)
        stream = torch.cuda.ExternalStream(flow.stream())
        with ResidentParticles3D(flow, count) as parts:

            def time_of(positions):
                rec = np.zeros((count, 8))
                rec[:, :3], rec[:, 6], rec[:, 7] = positions, 1.0, 1e6
                parts.upload(rec)
                best = np.inf
                for _ in range(6):  # the first as warm-up
                    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    a.record(stream)
                    for _ in range(10):
                        parts.advance(macro, force, 1e-6, True, ParticleVector3(0, 0, 0))
                    b.record(stream)
                    flow.wait()
                    best = min(best, a.elapsed_time(b))
                return best

            scattered = time_of(rng.uniform(0, 1, (count, 3)) * shape)
            for k in (2, 8):
                cells = np.stack([rng.integers(0, e - 1, k) for e in shape], 1)
                gathered = time_of(cells[rng.integers(0, k, count)] + rng.uniform(0.1, 0.9, (count, 3)))
                assert gathered < 3 * scattered, (k, gathered, scattered)  # B200: at most 1.7; 4.5 and 17 without groups
