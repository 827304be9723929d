"""Small worlds join the steps of one call in one graph launch: the same bits
and the same kernel counts as steps one at a time, with and without bodies,
across target-order refreshes and list capacity checks; a chosen
graph_steps = 1 keeps the steps apart."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, build
from fluidgrid_gb300.scenes import H, SPACING, SceneSpec, Body, lattice, box_surface, random_quaternion

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def scene(nbodies):
    rng = np.random.default_rng(11)
    pos = lattice(12, 8, 10, SPACING, (SPACING, SPACING, SPACING), 0.05 * H, rng)
    bodies = [Body(local=box_surface(0.12, 301, rng), mass=4.0, position=(0.25, 0.22, 0.2),
                   orientation=random_quaternion(rng)) for _ in range(nbodies)]
    return SceneSpec(pos=pos, box_min=(0, 0, 0), box_max=(1, 1, 1), buckets=(32, 16, 8), bodies=bodies,
                     rb_buckets=(16, 16, 16))


@pytest.mark.parametrize("nbodies", [0, 1])
@pytest.mark.parametrize("calls", [(1,) * 20 + (40,), (7,) * 9, (3,) * 21, (2,) * 31, (64,)])
def test_joined_steps_equal_single_steps(calls, nbodies):
    out = []
    for chosen in (True, False):
        w = World([scene(nbodies)])
        w.set_option("autotune_period", 0)
        w.set_option("order_period", 9)
        if chosen:
            w.set_option("graph_steps", 1)
        k0 = w.kernel_launches()
        for k in calls:
            w.step(k)
        state = w.download() + ((w.read("BODY_X"), w.read("BODY_Q")) if nbodies else ())
        out.append((w.kernel_launches() - k0, state))
        assert w.get_option("graph_steps") == 1
        w.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
