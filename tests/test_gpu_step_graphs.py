"""Step loops of 8 or more steps replay a captured CUDA graph of 8 steps (cfdx_lbm_step, csrc/capi.cu).

A graph launches the same kernels with the same argument blocks as the step-by-step loop, so a
run of many steps in one call must equal the same steps taken one call at a time, bit for bit,
for every storage the graph path takes (FP32, FP64; FP16 and slabs keep plain launches), with
walls, moving walls, gray cells, per-cell forces and the paired FP32 kernel, from even and odd
time steps, and for step counts that leave a remainder after the whole graphs.  The graph is
kept on the handle between calls (one per starting parity) and must be captured again whenever
a parameter, a buffer or the kernel choice changes.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(cs, q, storage, kind, variant=0):
    nx, ny, nz = 18, 14, 12
    lattice = {19: "d3q19", 27: "d3q27"}[q]
    s = cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.62, lattice=lattice, storage=storage,
                                                      collision="trt", acceleration_x=2e-5))
    if variant:
        s.set_launch_shape(0, 0, variant)
    if kind in ("cavity", "gray"):
        s.set_flags(cs.cavity_flags(nx, ny, nz))
        s.set_wall_velocity(2, 0.05, 0.0, 0.0)
    if kind == "gray":
        rng = np.random.default_rng(3)
        s.set_solid_fraction(rng.uniform(0, 0.2, nx * ny * nz).astype(np.float32))
        s.set_local_body_acceleration(*(rng.normal(0, 1e-5, nx * ny * nz).astype(np.float32) for _ in range(3)))
    s.initialize_taylor_green(0.03)
    return s


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("storage", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["periodic", "cavity", "gray"])
def test_graph_steps_equal_single_steps(engine, q, storage, kind):
    cs = engine
    with solver(cs, q, storage, kind) as a, solver(cs, q, storage, kind) as b:
        a.step(1)
        b.step(1)  # start both at an odd time step
        a.step(101)  # 12 graph replays of 8 + 5 plain steps
        for _ in range(101):
            b.step(1)
        assert a.time_step() == b.time_step() == 102
        assert np.array_equal(a.logical_populations(), b.logical_populations())
        a.step(64)
        b.step(32)
        b.step(32)
        assert np.array_equal(a.logical_populations(), b.logical_populations())


def test_graph_steps_paired_fp32_kernel(engine):
    cs = engine
    with solver(cs, 19, "fp32", "cavity", variant=2) as a, solver(cs, 19, "fp32", "cavity", variant=1) as b:
        a.step(70)
        for _ in range(70):
            b.step(1)
        assert np.array_equal(a.logical_populations(), b.logical_populations())


def test_cached_graph_follows_changes(engine):
    """Calls that replay the handle's graph, and calls after changes that must not replay it."""
    cs = engine

    def run(s, steps, single):
        if single:
            for _ in range(steps):
                s.step(1)
        else:
            s.step(steps)

    with solver(cs, 19, "fp32", "cavity") as a, solver(cs, 19, "fp32", "cavity") as b:
        plan = [
            (None, 16), (None, 8), (None, 1), (None, 8), (None, 9),   # replays from even and odd steps
            (lambda s: s.set_tau(0.7), 16),
            (lambda s: s.set_wall_velocity(2, 0.02, 0.01, 0.0), 8),
            (lambda s: s.set_launch_shape(0, 0, 2), 16),              # paired kernel
            (lambda s: s.set_launch_shape(0, 0, 1), 8),
            (lambda s: s.set_flags(cs.cavity_flags(18, 14, 12, lid_id=3)), 8),
            (lambda s: s.set_wall_velocity(3, -0.03, 0.0, 0.0), 24),
        ]
        for change, steps in plan:
            for s, single in ((a, False), (b, True)):
                if change:
                    change(s)
                run(s, steps, single)
            assert a.time_step() == b.time_step()
            assert np.array_equal(a.logical_populations(), b.logical_populations())


@pytest.mark.parametrize("q, storage, variant", [(19, "fp32", 0), (19, "fp32", 2), (27, "fp32", 0), (19, "fp64", 0),
                                                 (19, "fp16s", 0), (19, "fp16s", 1), (19, "fp16s", 2), (27, "fp16s", 0),
                                                 (19, "fp16s", 3), (19, "fp16s", 4), (27, "fp16s", 3)])
@pytest.mark.parametrize("kind", ["gray", "cavity", "periodic"])
def test_overlapping_launches_equal_separate_ones(engine, q, storage, variant, kind):
    """Each lattice kernel, in its gray, walled and open form, may be scheduled while the one before
    it drains (programmatic dependent launch): steps, reductions, field reads and setters queued back to back equal the same calls
    with the stream drained after each, bit for bit."""
    cs = engine
    out = []
    for drain in (False, True):
        with solver(cs, q, storage, kind, variant) as s:
            seen = []
            for k in range(12):
                s.step(1 + 9 * (k % 3))
                if drain:
                    s.wait()
                if k % 4 == 1:
                    seen.append(s.reduce())
                if k % 4 == 2:
                    s.refresh_device_macroscopic()
                    s.device_local_acceleration(clear=True)
                if k % 4 == 3:
                    s.set_tau(0.62 + 0.01 * k)
                if drain:
                    s.wait()
            out.append((seen, s.logical_populations()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("q, storage, kind, variant", [(19, "fp32", "periodic", 0), (27, "fp64", "gray", 0),
                                                       (19, "fp32", "cavity", 2), (19, "fp16s", "cavity", 3),
                                                       (19, "fp16s", "periodic", 0), (19, "fp16s", "cavity", 2)])
def test_steps_under_a_callers_capture(engine, q, storage, kind, variant):
    """Dependent launches recorded by a caller's capture of the solver's stream: beside a fork to
    another stream that joins again, a memset and a field read, a replay equals the same calls."""
    import torch

    cs = engine
    out = []
    for captured in (False, True):
        with solver(cs, q, storage, kind, variant) as s:
            s.refresh_device_macroscopic()  # allocates its fields
            s.wait()
            stream, side = torch.cuda.ExternalStream(s.stream()), torch.cuda.Stream()
            buf = torch.zeros(1 << 14, device="cuda")
            torch.cuda.synchronize()

            def calls():
                s.step(2)
                side.wait_stream(stream)
                with torch.cuda.stream(side):
                    buf.add_(1.0)
                stream.wait_stream(side)
                s.step(2)
                buf.zero_()
                s.step(1)
                s.refresh_device_macroscopic()
                s.step(9)

            with torch.cuda.stream(stream):
                if captured:
                    graph = torch.cuda.CUDAGraph()
                    graph.capture_begin(capture_error_mode="thread_local")
                    try:
                        calls()
                    finally:
                        graph.capture_end()
                    graph.replay()
                    torch.cuda.synchronize()
                    del graph
                else:
                    calls()
            torch.cuda.synchronize()
            out.append(s.logical_populations())
    assert np.array_equal(out[0], out[1])
