"""The host memory that a server keeps for its next requests goes with the
server, though a result of its lives on."""
import gc
import os

import numpy as np
import pytest

from fluidgrid_gb300 import Server, build
from fluidgrid_gb300.scenes import H, SceneSpec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def resident():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


def scene(n):
    i = np.arange(n)
    nx = int(round(n ** (1 / 3))) + 1
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = np.stack([i % nx, i // (nx * nx), i // nx % nx], 1) * (0.5 * H) + 0.1
    return SceneSpec(pos=pos, box_min=(0,) * 3, box_max=(0.2 + nx * 0.5 * H,) * 3, buckets=(1 << 20, 1, 1))


def test_spare_memory_goes_with_the_server():
    """Three requests of 2.2 million particles: 211 MB of arrays (each its own
    mapping), all of them given back to the server and kept."""
    srv = Server(budget_bytes=32 << 30, max_particles=2_500_000)
    small, spec = scene(1000), scene(2_200_000)
    ids = [srv.submit(small, 1)] + [srv.submit(spec, 1) for _ in range(3)]
    while not all(srv.done(i) for i in ids):
        srv.step()
    kept = srv.result(ids[0])
    for i in ids[1:]:
        srv.result(i)
    gc.collect()
    before, want = resident(), kept[0].copy()
    srv.close()
    assert before - resident() > 150e6
    assert np.array_equal(kept[0], want)
