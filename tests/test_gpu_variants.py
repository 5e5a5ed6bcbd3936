"""The paired-cell step kernel against the one-cell kernel (GPU).

Both variants evaluate the same per-cell collision with the same rounding
(FP16 stores: the same stochastic rounding bits per cell and direction), so
after any number of steps their populations must agree bit for bit.
The cases cover partial warps (nx/2 not a multiple of 32), multi-warp rows,
the x-periodic wrap of shifted word accesses, random walls next to fluid
cells inside one thread's pair, moving walls, gray cells and both parities.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(18, 15, 13), (130, 6, 5), (2, 6, 4), (64, 9, 7)]


def run(cs, variant, q, shape, storage, flags_kind, gray, steps, seed=11, planes=0):
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    storage, _, rounding = storage.partition(":")
    cfg = cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.6, lattice={19: "d3q19", 27: "d3q27"}[q],
                              storage=storage, collision="trt", smagorinsky_les=True, smagorinsky_cs=0.1,
                              acceleration_x=1e-5, fp16_rounding=rounding or "stochastic")
    with cs.EsotericPullCudaSolver(cfg) as s:
        s.set_launch_shape(0, 0, variant)
        s.set_step_planes(planes)
        if flags_kind == "random":
            fl = (rng.random(n) < 0.2).astype(np.uint8)
            fl[rng.random(n) < 0.05] = 3
            s.set_flags(fl)
            s.set_wall_velocity(3, 0.02, -0.01, 0.0)
        elif flags_kind == "cavity":
            s.set_flags(cs.cavity_flags(nx, ny, nz))
            s.set_wall_velocity(2, 0.08, 0.0, 0.0)
        if gray:
            s.set_solid_fraction(rng.uniform(0, 0.2, n).astype(np.float32))
        s.initialize_taylor_green(0.05)
        s.step(steps)
        logical = s.logical_populations()
        red = s.reduce()
        return logical, red


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp16s:nearest"])
@pytest.mark.parametrize("shape", SHAPES, ids=[f"{a}x{b}x{c}" for a, b, c in SHAPES])
@pytest.mark.parametrize("flags_kind, gray", [(None, False), ("random", False), ("cavity", True)])
@pytest.mark.parametrize("steps", [5, 6])
def test_paired_matches_single_bitwise(engine, q, storage, shape, flags_kind, gray, steps):
    a_log, a_red = run(engine, 1, q, shape, storage, flags_kind, gray, steps)
    b_log, b_red = run(engine, 2, q, shape, storage, flags_kind, gray, steps)
    assert np.array_equal(a_log.view(np.uint32), b_log.view(np.uint32))
    assert a_red["mass"] == b_red["mass"]


def test_paired_variant_requires_even_nx(engine):
    cs = engine
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=17, ny=4, nz=4)) as s:
        with pytest.raises(ValueError, match="paired"):
            s.set_launch_shape(0, 0, 2)
        s.set_launch_shape(0, 0, 0)  # automatic falls back to one cell per thread
        s.step(3)


@pytest.mark.parametrize("storage, shape", [("fp16s", (17, 6, 5)), ("fp32", (17, 6, 5)), ("fp64", (16, 6, 5)),
                                            ("fp16s", (16, 6, 5)), ("fp32", (16, 6, 5))])
def test_a_refused_launch_shape_leaves_the_handle_as_it_was(engine, storage, shape):
    """Every setter that chooses the kernel again used to find the refused variant: an odd row in the
    two-cell kernel.  Refused variants and shapes between setters change nothing."""
    cs = engine
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(4)
    flags, ns = (rng.random(n) < 0.1).astype(np.uint8), rng.uniform(0, 0.2, n).astype(np.float32)
    refused = [(0, 0, 5), (0, 0, -1), (48, 1, 0), (256, 1, 0), (64, 0, 0)]
    if nx % 2 or storage == "fp64":
        refused += [(0, 0, 2), (32, 4, 2)]
    else:
        refused += [(16, 4, 2)]  # the two-cell kernels take whole warps along x
    refused += [(0, 0, 3), (0, 0, 4)] if nx % 2 or storage != "fp16s" else [(32, 1, 3)]
    out = []
    for refuse in (False, True):
        def tries(s):
            for bx, by, variant in refused if refuse else []:
                with pytest.raises(ValueError):
                    s.set_launch_shape(bx, by, variant)

        with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.6, storage=storage)) as s:
            tries(s)
            s.initialize_taylor_green(0.05)
            s.step(2)
            s.set_flags(flags)
            s.step(2)
            tries(s)
            s.set_solid_fraction(ns)
            s.step(3)
            out.append(s.logical_populations())
    assert np.array_equal(out[0], out[1])


# The wall-aware FP16 pair kernel (variants 3 and 4) marches along z; plane
# counts that do not divide nz leave a short last chunk, and rows of 256 cells
# span more than one warp.  The pipelined form (variant 3) reads flags three
# and wall-link masks two planes ahead: runs of 1, 2 and 3 planes per thread
# end its look-ahead at every depth.
W2_SHAPES = SHAPES + [(256, 5, 9)]


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("storage", ["fp16s", "fp16s:nearest"])
@pytest.mark.parametrize("shape", W2_SHAPES, ids=[f"{a}x{b}x{c}" for a, b, c in W2_SHAPES])
@pytest.mark.parametrize("flags_kind, gray", [(None, False), ("random", False), ("random", True),
                                              ("cavity", False), ("cavity", True)])
@pytest.mark.parametrize("variant, planes", [(3, 0), (3, 1), (3, 2), (3, 3), (4, 1), (4, 5)])
def test_wall_aware_pairs_match_single_bitwise(engine, q, storage, shape, flags_kind, gray, variant, planes):
    steps = 5
    a_log, a_red = run(engine, 1, q, shape, storage, flags_kind, gray, steps)
    b_log, b_red = run(engine, variant, q, shape, storage, flags_kind, gray, steps, planes=planes)
    assert np.array_equal(a_log.view(np.uint32), b_log.view(np.uint32))
    assert a_red["mass"] == b_red["mass"]


# Marches of four planes and more, the lengths that large lattices take: only from the fourth plane
# on does the pipelined form store all four slots of its flag ring and fetch wall-link masks
# three planes ahead over the stage it has just read.  Whole chunks and short last ones.
LONG_SHAPES = [(18, 7, 17), (130, 6, 8), (256, 5, 21)]


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("storage", ["fp16s", "fp16s:nearest"])
@pytest.mark.parametrize("shape", LONG_SHAPES, ids=[f"{a}x{b}x{c}" for a, b, c in LONG_SHAPES])
@pytest.mark.parametrize("flags_kind, gray", [(None, False), ("random", False), ("random", True), ("cavity", False)])
@pytest.mark.parametrize("variant, planes", [(3, 4), (3, 5), (3, 8), (3, 21), (4, 4)])
def test_wall_aware_pairs_in_long_marches(engine, q, storage, shape, flags_kind, gray, variant, planes):
    a_log, a_red = run(engine, 1, q, shape, storage, flags_kind, gray, 5)
    b_log, b_red = run(engine, variant, q, shape, storage, flags_kind, gray, 5, planes=planes)
    assert np.array_equal(a_log.view(np.uint32), b_log.view(np.uint32))
    assert a_red["mass"] == b_red["mass"]


# Above 2^20 cells a walled D3Q19 FP16 lattice takes the pair kernel, with the planes per thread that
# the rule picks for its size (four on the last shape).
@pytest.mark.parametrize("shape", [(104, 102, 100), (300, 60, 60), (256, 160, 128)], ids=str)
@pytest.mark.parametrize("flags_kind", ["random", "cavity"])
def test_automatic_choice_above_the_border_matches_single_bitwise(engine, shape, flags_kind):
    assert np.prod(shape) >= 1 << 20
    a_log, a_red = run(engine, 1, 19, shape, "fp16s", flags_kind, False, 3)
    b_log, b_red = run(engine, 0, 19, shape, "fp16s", flags_kind, False, 3)
    assert np.array_equal(a_log.view(np.uint32), b_log.view(np.uint32))
    assert a_red["mass"] == b_red["mass"]


def test_wall_aware_pairs_need_fp16_and_even_nx(engine):
    cs = engine
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=16, ny=4, nz=4)) as s:
        with pytest.raises(ValueError, match="wall-aware"):
            s.set_launch_shape(0, 0, 3)
        with pytest.raises(ValueError, match="planes"):
            s.set_step_planes(-1)
    with cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(nx=17, ny=4, nz=4, storage="fp16s")) as s:
        with pytest.raises(ValueError, match="wall-aware"):
            s.set_launch_shape(0, 0, 4)
