"""FP16 runs keep their bits from one version of the engine to the next (GPU).

A moment summed in another order rounds differently now and then, FP16 storage turns that into
another stored half, and a run restarted from an older checkpoint leaves the trajectory it had
(relative 1e-4 in a few hundred steps of a Smagorinsky cavity).  So the order of the FP16
collision's sums is part of the results: SHA-256 digests of the populations, recorded on a B200
from the engine as it was before its collision was first reordered, over both lattices, every
branch of the FP16 collision (Smagorinsky, per-cell force, gray cells, both collisions and
roundings), scales that are not powers of two, odd and even rows, and a walled lattice above the
size from which the pair kernel is chosen.  Initial fields come from the host, so only the engine's
own arithmetic is in the digest."""
from __future__ import annotations

import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLED, OPEN = (33, 17, 13), (64, 18, 12)
CASES = {
    "cavity-les-19": (19, WALLED, dict(collision="trt", les=True, walls="cavity")),
    "cavity-les-27": (27, WALLED, dict(collision="trt", les=True, walls="cavity")),
    "cavity-les-nearest-27": (27, OPEN, dict(collision="bgk", les=True, walls="cavity", rounding="nearest")),
    "random-les-force-19": (19, OPEN, dict(collision="trt", les=True, walls="random", force=True)),
    "random-les-force-27": (27, OPEN, dict(collision="trt", les=True, walls="random", force=True)),
    "gray-force-19": (19, WALLED, dict(collision="trt", walls="random", force=True, gray=True)),
    "gray-force-27": (27, WALLED, dict(collision="trt", walls="random", force=True, gray=True)),
    "open-bgk-19": (19, OPEN, dict(collision="bgk")),
    "open-les-19": (19, OPEN, dict(collision="trt", les=True)),
    "open-bgk-27": (27, WALLED, dict(collision="bgk")),
    "scaled-les-19": (19, OPEN, dict(collision="trt", les=True, walls="cavity", scaled=True)),
    "scaled-les-27": (27, WALLED, dict(collision="trt", les=True, walls="cavity", scaled=True)),
    "pairs-les-19": (19, (104, 104, 100), dict(collision="trt", les=True, walls="cavity", steps=12)),
    "adjoint-19": (19, WALLED, dict(collision="trt", walls="random", gray=True, adjoint=True)),
    "adjoint-27": (27, OPEN, dict(collision="bgk", walls="random", gray=True, adjoint=True)),
}
DIGESTS = {
    "cavity-les-19": "06f59257059f9979ebdfa8c57e154fab9eccefb9d697f99a99ddbe79bf88d497",
    "cavity-les-27": "5ea2309a86905d736ef116cee071be5d7852e27b2e97aefc6e9a13e524423498",
    "cavity-les-nearest-27": "01075bc756a2234b5756c97b86acbbf073a8ce6774713d5292c945edf8a808a5",
    "random-les-force-19": "ebd82534e357c2806b6335f9373c07b766d2441d898e9b9b0b291c780e972893",
    "random-les-force-27": "403db113eb6f3e1901683816977ff8629c21899af4dfd97b76bf3cdac75be11e",
    "gray-force-19": "e152cc6b31be49bd951868422fe645481915231f7f2f91549084a8f4df7f7f17",
    "gray-force-27": "d6be400357ffc2b91114efc63f648fc792523bbb4d55ae36c941a0d531539ab1",
    "open-bgk-19": "033ab978ba95593590db976fa58072ffeb20381df5e74e84f8ca1b1a4557c9d4",
    "open-les-19": "0e7cb5c4fd08a0cfb041b4e4b364afd75774231297d34de3729925d7dd04ca37",
    "open-bgk-27": "97bba7128b5d4c5e7dbe01cec2705031e7afd54e13c7490bcd3c2d461608b22e",
    "scaled-les-19": "3283e705d5eeef670576950206902442f8b0f6cd37f532d81bffc795ea936eaa",
    "scaled-les-27": "47a0315f5b2d6f5af7d79f0f42040e4694afcb1cf48c0140787e48f2dc2b1ebe",
    "pairs-les-19": "2333142c65ae83e07df7bece47ed9ca1e4e4bd55b058852f3f6faeda5057e85e",
    "adjoint-19": "56f5701ab956362ce914d74fd2bd831cc00a42fb53dddc21f99310bfe5f1473a",
    "adjoint-27": "aa35b869b6dc57dba9cf51990e6c5a6a308035b0ac6faa9c5afd7f8d7c5978f5",
}


def digest(cs, name):
    q, (nx, ny, nz), c = CASES[name]
    n = nx * ny * nz
    rng = np.random.default_rng(20 + q)
    cfg = cs.InPlaceLbmConfig(nx=nx, ny=ny, nz=nz, tau=0.55, lattice={19: "d3q19", 27: "d3q27"}[q], storage="fp16s",
                              collision=c["collision"], smagorinsky_les=c.get("les", False), smagorinsky_cs=0.1,
                              fp16_rounding=c.get("rounding", "stochastic"))
    with cs.EsotericPullCudaSolver(cfg) as s:
        if c.get("scaled"):
            s.set_storage_scale(rng.uniform(5.0, 90.0, 4).astype(np.float32)[scale_class(q)])
        if c.get("walls") == "cavity":
            s.set_flags(cs.cavity_flags(nx, ny, nz))
            s.set_wall_velocity(2, 0.08, 0.0, 0.02)
        elif c.get("walls") == "random":
            s.set_flags((rng.random(n) < 0.15).astype(np.uint8))
        if c.get("gray"):
            s.set_solid_fraction(rng.uniform(0, 0.2, n).astype(np.float32))
        if c.get("force"):
            s.set_local_body_acceleration(*(rng.normal(0, 1e-4, n).astype(np.float32) for _ in range(3)))
        s.initialize_fields(rng.uniform(0.95, 1.05, n).astype(np.float32),
                            *(rng.uniform(-0.06, 0.06, n).astype(np.float32) for _ in range(3)))
        h = hashlib.sha256()
        if c.get("adjoint"):
            s.adjoint_forward(11, 4)
            grad, _ = s.adjoint_backward(*(rng.normal(size=n).astype(np.float32) for _ in range(3)))
            h.update(np.ascontiguousarray(grad).tobytes())
        else:
            s.step(c.get("steps", 40))
        h.update(np.ascontiguousarray(s.logical_populations()).tobytes())
        return h.hexdigest()


def scale_class(q):
    """Weight class (number of nonzero components) of each direction, in the engine's order."""
    return np.array([0] + [1] * 6 + [2] * 12 + ([3] * 8 if q == 27 else []))


@pytest.mark.parametrize("name", list(CASES))
def test_populations_keep_their_bits(engine, name):
    assert digest(engine, name) == DIGESTS[name]
