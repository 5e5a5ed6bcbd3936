"""Setting a lattice up and reading its sums on the device (csrc/capi.cu, csrc/lbm_device.cuh).

* k_init writes every slot, so an initialisation needs no cleared lattice: wall cells zero the slots
  that no fluid cell's wall link seeds.
* Flags and initial fields in device memory are read in place, host ones are staged, alike; the
  moving-wall scan runs in the preparation kernel.
* The FP64 sums spread rows over a block's y threads and are combined by the last block.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Raw:
    def __init__(self, pointer, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (pointer, False), "version": 3,
                                         "strides": None}


def raw(solver, typestr):
    import torch

    ptr, size = solver.raw_populations()
    count = size // int(typestr[-1])
    return torch.as_tensor(_Raw(ptr, (count,), typestr), device="cuda")


def random_flags(shape, seed):
    f = (np.random.default_rng(seed).uniform(size=shape) < 0.3).astype(np.uint8)
    return f.reshape(-1)


@pytest.mark.parametrize("lattice", ["d3q19", "d3q27"])
@pytest.mark.parametrize("storage, typestr", [("fp32", "<f4"), ("fp16s", "<f2"), ("fp64", "<f8")])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 7, 3), (33, 9, 10)], ids=str)
def test_init_writes_every_slot(engine, lattice, storage, typestr, shape):
    import torch

    cs = engine
    nx, ny, nz = shape
    images = []
    for dirty in (float("nan"), 0.0):
        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, lattice=lattice, storage=storage)) as s:
            for flags in (None, random_flags((nz, ny, nx), 4)):
                if flags is not None:
                    s.set_flags(flags)
                raw(s, typestr).fill_(dirty)
                torch.cuda.synchronize()
                s.initialize_uniform(1.02, 0.01, -0.02, 0.03)
                s.wait()
                images.append(raw(s, typestr).cpu().numpy().copy())
    assert np.isfinite(images[0]).all() and np.isfinite(images[1]).all()
    # the image over a cleared lattice is the one a memset before the kernel gave
    assert images[0].tobytes() == images[2].tobytes() and images[1].tobytes() == images[3].tobytes()


@pytest.mark.parametrize("offset", [0, 1, 3])
def test_device_flags_and_fields_equal_host_ones(engine, offset):
    import torch

    cs = engine
    nx, ny, nz = 17, 6, 5
    n = nx * ny * nz
    flags = random_flags((nz, ny, nx), 9)
    rng = np.random.default_rng(1)
    fields = np.concatenate([rng.uniform(0.9, 1.1, n), rng.uniform(-0.05, 0.05, 3 * n)]).astype(np.float32)
    out = []
    for device in (False, True):
        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz)) as s:
            if device:
                f = torch.zeros(n + offset, dtype=torch.uint8, device="cuda")[offset:]
                f.copy_(torch.from_numpy(flags))
                # a float view at `offset` bytes past an aligned address: staged unless aligned
                u = torch.zeros(16 * n + 16, dtype=torch.uint8, device="cuda")
                u[offset:offset + 16 * n] = torch.from_numpy(fields.view(np.uint8)).cuda()
                torch.cuda.synchronize()
                s.set_flags(f)
                s.library.call("cfdx_lbm_init_fields", s.handle, ctypes.c_void_p(u.data_ptr() + offset), 1)
            else:
                s.set_flags(flags)
                s.initialize_fields(*fields.reshape(4, n))
            s.step(3)
            out.append(s.logical_populations())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("value, moving", [(1, False), (2, True), (15, True), (17, True)])
def test_moving_walls_are_found_on_the_device(engine, where, value, moving):
    import torch

    cs = engine
    flags = np.zeros((6, 5, 40), np.uint8)
    flags[5, 4, 39] = value  # the last cell alone; 17 is out of the id range, as the scan has always seen it
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=40, ny=5, nz=6)) as s:
        for _ in range(2):  # and again after flags without one
            s.set_flags(torch.from_numpy(flags.reshape(-1)).cuda() if where == "device" else flags.reshape(-1))
            if moving:
                with pytest.raises(ValueError):
                    s.adjoint_forward(2, 2)
            else:
                s.adjoint_forward(2, 2)
            s.set_flags(np.zeros(flags.size, np.uint8))
            s.adjoint_forward(2, 2)


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (31, 3, 2), (33, 70, 40), (64, 2, 700), (257, 9, 300)], ids=str)
def test_sums_equal_the_fields_sums(engine, storage, shape):
    """Mass, momentum and kinetic energy against FP64 sums of the reported fields: FP64 additions in
    another order differ by at most (cells) ulps of the sum of magnitudes, far inside 1e-10."""
    cs = engine
    nx, ny, nz = shape
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, storage=storage)) as s:
        if nx > 2:
            s.set_flags(random_flags((nz, ny, nx), 2))
        s.initialize_taylor_green(0.05)
        s.step(2)
        rho, ux, uy, uz = (v.astype(np.float64) for v in s.compute_macroscopic())
        want = [rho.sum(), (rho * ux).sum(), (rho * uy).sum(), (rho * uz).sum(),
                0.5 * (rho * (ux * ux + uy * uy + uz * uz)).sum()]
        size = [np.abs(rho).sum(), np.abs(rho * ux).sum(), np.abs(rho * uy).sum(), np.abs(rho * uz).sum(), want[4]]
        first, second = s.reduce(), s.reduce()
        assert first == second  # the counter of finished blocks is back at zero
        got = [first["mass"], *first["momentum"], first["kinetic_energy"]]
        for g, w, m in zip(got, want, size):
            assert abs(g - w) <= 1e-10 * m + 1e-300
        speed = np.sqrt(ux * ux + uy * uy + uz * uz).max()
        assert abs(first["max_speed"] - speed) <= 2e-7 * speed


def test_fields_inside_the_lattice_are_staged(engine):
    """Initial fields that lie in the population buffer itself are copied out before k_init overwrites them."""
    import torch

    cs = engine
    nx, ny, nz = 18, 7, 5
    n = nx * ny * nz
    rng = np.random.default_rng(6)
    fields = np.concatenate([rng.uniform(0.9, 1.1, n), rng.uniform(-0.05, 0.05, 3 * n)]).astype(np.float32)
    out = []
    for inside in (False, True):
        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz)) as s:
            if inside:
                view = raw(s, "<f4")
                view[n:5 * n] = torch.from_numpy(fields).cuda()
                torch.cuda.synchronize()
                s.library.call("cfdx_lbm_init_fields", s.handle, ctypes.c_void_p(view.data_ptr() + 4 * n), 1)
            else:
                s.initialize_fields(*fields.reshape(4, n))
            s.step(2)
            out.append(s.logical_populations())
    assert np.array_equal(out[0], out[1])


def test_flag_staging_retries_when_memory_is_short(engine):
    """Host flags and voxelized bodies are staged from the scratch pool: a first attempt that runs out of
    memory returns the pool's idle memory and tries again, as every other allocation does."""
    cs = engine
    lib = cs.load()
    nx, ny, nz = 17, 6, 5
    flags = random_flags((nz, ny, nx), 9)
    triangles = np.array([[[0.1, 0.1, 0.1], [0.9, 0.1, 0.1], [0.1, 0.9, 0.1]]])

    def retries():
        count = ctypes.c_ulonglong(0)
        lib.raw.cfdx_debug_retry_allocations(-1, ctypes.byref(count))
        return count.value

    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz)) as s:
        s.set_flags(np.zeros(flags.size, np.uint8))  # holds its flag and wall-link fields from here on
        want = None
        for hook in (0, 1):
            before = retries()
            lib.raw.cfdx_debug_retry_allocations(hook, None)
            try:
                s.set_flags(flags)
                s.initialize_uniform(1.0, 0.02, 0.0, 0.0)
                s.step(2)
                got = s.logical_populations()
                assert retries() == before + hook
                lib.raw.cfdx_debug_retry_allocations(hook, None)
                s.set_solid_surface(triangles)
                assert retries() == before + 2 * hook
            finally:
                lib.raw.cfdx_debug_retry_allocations(0, None)
            want = got if want is None else want
            assert np.array_equal(got, want)


def test_an_allocation_that_fails_leaves_no_error_behind(engine):
    """A lattice larger than the device is refused; the launches after it do not report that error again."""
    cs = engine
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=18, ny=7, nz=5)) as s:
        with pytest.raises(MemoryError):
            cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=1500, ny=1500, nz=1500, lattice="d3q27", storage="fp64"))
        s.set_flags(random_flags((5, 7, 18), 3))
        s.initialize_uniform()
        s.step(2)
        assert s.reduce()["nonfinite"] == 0


@pytest.mark.parametrize("lattice, storage, walls, ratio", [("d3q19", "fp32", True, 1.45), ("d3q27", "fp64", False, 1.25)])
def test_sums_run_at_about_the_field_reads_rate(engine, lattice, storage, walls, ratio):
    """The sums and the field read load the same populations.  A reduction whose blocks need a second
    wave (too many registers) or whose loads wait in line (too few) takes 1.66 and 1.44 times as
    long as the read here; in one wave 1.1 and 0.96, the host's share of a call included."""
    import time

    import torch

    cs = engine
    nx, ny, nz = 512, 512, 48
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, lattice=lattice, storage=storage)) as s:
        if walls:
            s.set_flags(cs.cavity_flags(nx, ny, nz))
        s.initialize_taylor_green(0.03)

        def best(call, n=10):
            call()
            times = []
            for _ in range(6):
                torch.cuda.synchronize()
                t = time.perf_counter()
                for _ in range(n):
                    call()
                torch.cuda.synchronize()
                times.append((time.perf_counter() - t) / n)
            return min(times)

        read, sums = best(s.refresh_device_macroscopic), best(s.reduce)
        assert sums < ratio * read, (sums, read)
