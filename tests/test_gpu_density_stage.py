"""The density pass, which stages each cell's candidates by warp, against the
FP64 oracle and across target counts: around the edges of a warp's range and of
a work item, cells with one target and with more than a warp's, cells that
straddle ranges, cells wider than the kernel radius, buckets shared by many
cells, more groups than a warp stages (the walk by thread), a far origin with
unusual neighbour roundings; and the same bits for a scene alone and beside
others, whose sizes choose the warps' ranges."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, build
from fluidgrid_gb300.scenes import H, SceneSpec
from oracle import oracle as O
import helpers as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def cloud(n, spacing, seed, buckets=(64, 16, 16), cell=None, origin=0.3):
    """n particles in a cube at a mean distance of `spacing` kernel radii."""
    rng = np.random.default_rng(seed)
    side = spacing * H * n ** (1.0 / 3.0)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = origin + rng.uniform(0, side, (n, 3))
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.normal(0, 0.3, (n, 3))
    return SceneSpec(pos=pos, vel=vel, box_min=(origin - 1,) * 3, box_max=(origin + 5,) * 3, buckets=buckets,
                     cell=cell)


SCENES = {
    "one": cloud(1, 0.5, 1), "31": cloud(31, 0.2, 2), "33": cloud(33, 0.2, 3), "127": cloud(127, 0.4, 4),
    "129": cloud(129, 0.4, 5), "one_cell_1000": cloud(1000, 0.02, 6), "compressed": cloud(5003, 0.25, 7),
    "usual": cloud(20011, 0.5, 8), "spray": cloud(3001, 1.7, 9), "few_buckets": cloud(4001, 0.5, 10, (7, 3, 1)),
    "wide_cells": cloud(3001, 0.4, 11, cell=(2 * H, 1.3 * H, H)), "far": cloud(3001, 0.5, 12, origin=9000.0),
}


def density(specs):
    w = World(specs)
    w.set_option("autotune_period", 0)
    w.step(1)
    w.sync()
    out = w.read("DP"), w.read("VEL")
    lay = [w.layout(s) for s in range(len(specs))]
    w.close()
    return out, lay


@pytest.mark.parametrize("name", list(SCENES))
def test_density_against_fp64(name):
    spec = SCENES[name]
    (dp, _), _ = density([spec])
    ref = T.oracle_grid(spec, spec.pos, spec.vel)
    d64, _ = O.density(ref["spos"], ref["start"], ref["end"], ref["p"], O.kernels_cache(spec.h), spec.gas, spec.rest,
                       spec.mass, f64=True)
    assert (np.abs(dp[:, 0] - d64[:, 0]) / d64[:, 0]).max() <= 1e-5


def test_same_bits_alone_and_mixed():
    specs = [SCENES[k] for k in ("129", "compressed", "spray", "usual", "one", "few_buckets")]
    mixed, lay = density(specs * 6)
    for k, spec in enumerate(specs):
        alone, _ = density([spec])
        for copy in (k, k + 5 * len(specs)):
            b, n = lay[copy]["pbase"], lay[copy]["n"]
            for a, m in zip(alone, mixed):
                assert np.array_equal(a.view(np.uint32), m[b:b + n].view(np.uint32)), (k, copy)
