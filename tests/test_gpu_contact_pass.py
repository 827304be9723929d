"""The fluid side of the fluid/rigid contact as its own pass (near-sphere bit
table, searches by warp) against the staged step, whose force pass walks the
rigid grid for every particle inside the bodies' AABB: the same bits, over the
search half-widths, contact distances from a fraction of a rigid cell to
several, origins up to where every cell counts as near, and body counts up to
more than one scene."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, _ffi, build
from fluidgrid_gb300.scenes import H, SPACING, SceneSpec, Body, lattice, box_surface, sphere_surface, \
    random_quaternion

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def scene(seed, origin, rel, radius, nbodies):
    rng = np.random.default_rng(seed)
    o = np.asarray(origin, np.float64)
    pos = lattice(18, 9, 17, SPACING, o + SPACING, 0.05 * H, rng)
    bodies = []
    for b in range(nbodies):
        c = tuple(float(x) for x in o + (0.15 + 0.13 * b, 0.17, 0.2))
        loc = box_surface(0.12, 301, rng) if b % 2 == 0 else sphere_surface(0.07, 97)
        bodies.append(Body(local=loc, mass=4.0, position=c, orientation=random_quaternion(rng)))
    return SceneSpec(pos=pos, vel=np.c_[rng.normal(0, 0.3, (len(pos), 3)), np.zeros(len(pos))].astype(np.float32),
                     box_min=tuple(o), box_max=tuple(o + 1.0), buckets=(32, 16, 8), bodies=bodies,
                     rb_buckets=(31, 7, 11), f2r_rel=(rel, rel, rel), fluid_radius=radius)


def run(specs, staged):
    w = World(specs)
    w.set_option("autotune_period", 0)
    for _ in range(2):
        if staged:
            for name in ("neighbourhood", "density", "rb_grid", "rb_from_fluid", "rb_from_rb", "forces", "body_sums",
                         "body_integrate", "integrate"):
                flags = _ffi.RUN_WITH_CONTACT if name == "forces" else 0
                _ffi.check(w.L.fg_world_run_stage(w.h, _ffi.RUN[name], flags), name)
        else:
            w.step(1)
    out = w.download() + (w.read("BODY_X"),)
    w.close()
    return out


@pytest.mark.parametrize("origin", [(0.0, 0.0, 0.0), (-3.0, 2.0, -0.4), (70000.0, 0.0, 0.0)])
@pytest.mark.parametrize("rel,radius,nbodies", [(0, 0.25 * H, 1), (2, 0.25 * H, 2), (3, 0.8 * H, 1),
                                                (2, 0.02 * H, 2)])
def test_contact_pass_equals_inline_walk(origin, rel, radius, nbodies):
    specs = [scene(3, origin, rel, radius, nbodies), scene(4, (0.1, 0.1, 0.1), 2, 0.25 * H, 1),
             scene(5, origin, rel, radius, 0)]
    a, b = run(specs, False), run(specs, True)
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.uint8), y.view(np.uint8))
    if rel == 2 and radius == 0.25 * H:
        still = [scene(3, origin, rel, 0.0, 0), specs[1], specs[2]]
        n = len(specs[0].pos)
        assert not np.array_equal(run(still, False)[1][:n], a[1][:n]), "some particles must be in contact"
