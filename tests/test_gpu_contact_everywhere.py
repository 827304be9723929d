"""The contact pass where nearly all of a CTA's particles are near a sphere
(walked by thread at half-widths of up to 1 and of 3 and more) against the
staged step, which walks for every particle: the same bits, alone and beside a
scene of surfaces of the same or another half-width."""
import numpy as np
import pytest

from fluidgrid_gb300 import build
from fluidgrid_gb300.scenes import H, Body
import test_gpu_contact_pass as C

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def porous(rel, m):
    spec = C.scene(7, (0.0, 0.0, 0.0), rel, 0.25 * H, 0)
    spec.pos, spec.vel = spec.pos[:2625], spec.vel[:2625]  # an odd number of work items
    rng = np.random.default_rng(m)
    lo, hi = spec.pos[:, :3].min(0), spec.pos[:, :3].max(0)
    loc = np.zeros((m, 4), np.float32)
    loc[:, :3] = rng.uniform(lo - hi, hi - lo, (m, 3)) / 2
    spec.bodies.append(Body(local=loc, mass=50.0, position=tuple(float(x) for x in (lo + hi) / 2),
                            orientation=(0.0, 0.0, 0.0, 1.0)))
    return spec


@pytest.mark.parametrize("rel", [0, 1, 2, 3, 8])
@pytest.mark.parametrize("m", [40, 600, 700])
def test_contact_everywhere_equals_inline_walk(rel, m):
    surfaces = [C.scene(3, (0.1, 0.1, 0.1), r, 0.25 * H, 1) for r in (1, 2)]
    for specs in ([porous(rel, m)], [surfaces[1], porous(rel, m)], [porous(rel, m), surfaces[0]]):
        a, b = C.run(specs, False), C.run(specs, True)
        for x, y in zip(a, b):
            assert np.array_equal(x.view(np.uint8), y.view(np.uint8))
