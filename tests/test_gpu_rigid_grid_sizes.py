"""The rigid-sphere grid over scene sizes: one CTA per scene up to 4,096
spheres (a radix sort of 1 to 128 warps' pairs, two or more passes by the
bucket count), the general sort beyond; against a stable key sort.  A full
step, whose rigid grid and contact run beside the fluid's, against the same
stages one after another."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, _ffi, build
from fluidgrid_gb300.scenes import H, SPACING, SceneSpec, Body, lattice, random_quaternion

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def scene(seed, spheres, buckets, rb_rb=False):
    rng = np.random.default_rng(seed)
    pos = lattice(10, 6, 9, SPACING, (SPACING, SPACING, SPACING), 0.05 * H, rng)
    bodies = []
    for b, n in enumerate(spheres):
        loc = np.zeros((n, 4), np.float32)
        loc[:, :3] = rng.uniform(-0.1, 0.1, (n, 3))
        bodies.append(Body(local=loc, mass=4.0, position=(0.2 + 0.15 * b, 0.2, 0.2),
                           orientation=random_quaternion(rng)))
    return SceneSpec(pos=pos, box_min=(0, 0, 0), box_max=(1, 1, 1), buckets=(32, 16, 8), bodies=bodies,
                     rb_buckets=buckets, rb_rb=rb_rb)


@pytest.mark.parametrize("buckets", [(1, 1, 1), (16, 16, 1), (257, 1, 1), (64, 64, 64)])
@pytest.mark.parametrize("counts", [(1,), (33, 127), (129, 0, 1023, 31), (1025, 4095), (4096, 2048), (4097, 5),
                                    (9000, 12000)])
def test_rigid_grid_equals_a_stable_sort(counts, buckets):
    specs = [scene(7 + s, (c,) if c else (), buckets) for s, c in enumerate(counts)]
    w = World(specs)
    w.step(1)
    w.sync()
    g = {k: w.read(k) for k in ("RB_KEYS_UNSORTED", "RB_KEYS", "RB_IDS", "RB_START", "RB_END", "RB_SPOS", "RB_WORLD")}
    w.close()
    order = np.argsort(g["RB_KEYS_UNSORTED"], kind="stable")
    keys = g["RB_KEYS_UNSORTED"][order]
    assert np.array_equal(g["RB_KEYS"], keys)
    assert np.array_equal(g["RB_IDS"], order)
    assert np.array_equal(g["RB_SPOS"].view(np.uint32), g["RB_WORLD"][order].view(np.uint32))
    used, first, n = np.unique(keys, return_index=True, return_counts=True)
    start = np.full(len(g["RB_START"]), 0xffffffff, np.uint32)
    start[used] = first
    assert np.array_equal(g["RB_START"], start)
    assert np.array_equal(g["RB_END"][used], first + n)


@pytest.mark.parametrize("counts", [(4000, 300), (5000, 300)])
def test_forked_step_equals_the_stages(counts):
    specs = [scene(3, counts, (64, 64, 64), True), scene(4, (700,), (16, 16, 16))]
    out = []
    for staged in (False, True):
        w = World(specs)
        w.set_option("autotune_period", 0)
        for _ in range(3):
            if staged:
                for name in ("neighbourhood", "density", "rb_grid", "rb_from_fluid", "rb_from_rb", "forces",
                             "body_sums", "body_integrate", "integrate"):
                    flags = _ffi.RUN_WITH_CONTACT if name == "forces" else 0
                    _ffi.check(w.L.fg_world_run_stage(w.h, _ffi.RUN[name], flags), name)
            else:
                w.step(1)
        out.append(w.download() + (w.read("BODY_X"), w.read("BODY_L"), w.read("RB_FORCE")))
        w.close()
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    assert np.abs(out[0][4][:, :3]).max() > 0
