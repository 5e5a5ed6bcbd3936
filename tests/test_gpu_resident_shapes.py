"""The vector forms of the resident kernels at the sizes where they can go wrong (csrc/resident.cu, csrc/thermal.cu):
rows of whole and part blocks of four-cell groups, rows that take the one-cell kernels, cell counts that
take or refuse the four-cell thermal kernels, even and odd rows for the particles' joint accesses.  Every
result equals its float32 restatement (oracle) bit for bit; the spread force, whose order of additions
is not fixed, to 1e-6 of its largest value."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_resident import device_read, device_write

pytestmark = pytest.mark.gpu

SHAPES = [(4, 3, 3), (36, 9, 5), (132, 5, 3), (516, 3, 3), (15, 8, 3), (9, 5, 3), (6, 6, 5)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_resident_kernels_on_every_row_form(engine, oracle_mod, shape):
    from cfd_solvers_b200.multiphysics import (ParticleVector3, ResidentFlowDiagnostics3D, ResidentFreeSurface3D,
                                               ResidentParticles3D, ResidentThermalD3Q7)

    cs, O = engine, oracle_mod
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(5)
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.7)) as flow:
        flow.initialize_fields(np.ones(n), *(rng.uniform(-0.1, 0.1, n) for _ in range(3)))
        macro, f = flow.refresh_device_macroscopic(), flow.compute_macroscopic()
        u = (f.ux, f.uy, f.uz)
        force = flow.device_local_acceleration(clear=True)
        flow.wait()
        a0 = [rng.uniform(-1e-4, 1e-4, n).astype(np.float32) for _ in range(3)]
        for ptr, v in zip((force.ax, force.ay, force.az), a0):
            device_write(ptr, v)
        with ResidentThermalD3Q7(flow, 0.03) as th:
            t0 = rng.uniform(290, 310, n).astype(np.float32)
            th.initialize_field(t0)
            th.step(macro, 2)
            g = (np.array([0.25] + [0.125] * 6, np.float32)[:, None] * t0[None, :]).astype(np.float32)
            g = O.thermal_d3q7_step(g, u, nx, ny, nz, 0.03, 2).reshape(7, -1)
            t = np.zeros(n, np.float32)
            for d in range(7):
                t = t + g[d]
            assert np.array_equal(th.temperature(), t)
            th.add_boussinesq_acceleration(force, 300.0, 3e-3, ParticleVector3(0.5, -1.0, 0.25))
            flow.wait()
            scale = np.float32(-3e-3) * (t - np.float32(300.0))
            a0 = [(a + scale * np.float32(w)).astype(np.float32) for a, w in zip(a0, (0.5, -1.0, 0.25))]
            for ptr, e in zip((force.ax, force.ay, force.az), a0):
                assert np.array_equal(device_read(ptr, n), e)
        with ResidentFreeSurface3D(flow) as fs, ResidentFlowDiagnostics3D(flow) as dg:
            phi = rng.uniform(0, 1, n).astype(np.float32)
            fs.initialize_field(phi)
            fs.advect(macro, 0.7)
            phi = O.fill_advect(phi, u, nx, ny, nz, 0.7)
            assert np.array_equal(fs.fill(), phi)
            fs.add_surface_tension_acceleration(force, 0.072, 1.25)
            flow.wait()
            *normals, k = O.fill_geometry(phi, nx, ny, nz)
            geo = fs.geometry()
            for name, v in zip(("normal_x", "normal_y", "normal_z", "curvature"), (*normals, k)):
                assert np.array_equal(geo[name], v)
            a0 = list(O.surface_tension(phi, k, a0, nx, ny, nz, 0.072, 1.25))
            for ptr, e in zip((force.ax, force.ay, force.az), a0):
                assert np.array_equal(device_read(ptr, n), e)
            q = dg.q_criterion(macro)
            flow.wait()
            assert np.array_equal(device_read(q, n), O.resident_q(u, nx, ny, nz))
        # particles: on cell corners, in the last column, row and plane, past the faces, and at random
        pos = [(0, 0, 0), (nx - 1, ny - 1, nz - 1), (nx - 0.25, 0.5, nz - 0.5), (1.0, ny, -1e-9), (2.5 - 3 * nx, 0.75, 1.25)]
        rec = np.zeros((64, 8))
        rec[:, :3] = rng.uniform(0, 1, (64, 3)) * shape
        rec[:5, :3] = pos
        rec[:, 3:6] = rng.normal(0, 0.02, (64, 3))
        rec[:, 6], rec[:, 7] = rng.uniform(0.5, 2, 64), rng.uniform(0.3, 3, 64)
        with ResidentParticles3D(flow, 64) as parts:
            parts.upload(rec)
            parts.advance(macro, force, 0.5, True, ParticleVector3(0.0, -2e-4, 0.0))
            st, acc = O.particles_advance(rec.T.astype(np.float32), u, a0, nx, ny, nz, 0.5, True, (0.0, -2e-4, 0.0))
            assert np.array_equal(parts.download_records()[:, :6].T.astype(np.float32), st[:6])
            for ptr, e in zip((force.ax, force.ay, force.az), acc):
                assert np.abs(device_read(ptr, n) - e).max() <= 1e-6 * np.abs(e).max()
