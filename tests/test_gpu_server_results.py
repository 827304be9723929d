"""Results of the server as arrays of their own: the same values as a copied
result, valid after the server is gone, not written by later requests that
reuse host memory, given back from any thread; bodies' motion across
re-layouts as in a world of its own."""
import gc
import threading

import numpy as np
import pytest

from fluidgrid_gb300 import Server, World, build
from fluidgrid_gb300.scenes import H, SPACING, SceneSpec, Body, lattice, box_surface, random_quaternion

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def scene(seed, nx, nbodies, vel=True):
    rng = np.random.default_rng(seed)
    pos = lattice(nx, 7, 9, SPACING, (SPACING, SPACING, SPACING), 0.05 * H, rng)
    v = np.zeros_like(pos)
    v[:, :3] = rng.normal(0, 0.3, (len(pos), 3))
    bodies = [Body(local=box_surface(0.1, 200 + 31 * b, rng), mass=4.0, position=(0.2 + 0.1 * b, 0.25, 0.2),
                   orientation=random_quaternion(rng)) for b in range(nbodies)]
    return SceneSpec(pos=pos, vel=v if vel else None, box_min=(0, 0, 0), box_max=(1, 1, 1), buckets=(32, 16, 8),
                     bodies=bodies, rb_buckets=(16, 16, 16))


def alone(spec, steps):
    w = World([spec])
    w.step(steps)
    out = w.download()
    w.close()
    return out


def test_results_are_arrays_of_their_own():
    jobs = [(scene(1, 8, 1), 1), (scene(2, 13, 0, vel=False), 3), (scene(3, 8, 2), 2), (scene(4, 9, 1), 4)]
    want = [alone(s, k) for s, k in jobs]
    srv = Server(budget_bytes=8 << 30)
    held = []
    for _ in range(3):
        ids = [srv.submit(s, k) for s, k in jobs]
        while not all(srv.done(i) for i in ids):
            srv.step()
        for i in ids:
            copy = srv.result(i, release=False)
            own = srv.result(i)
            for a, b in zip(copy, own):
                assert b.dtype == np.float32 and b.flags.writeable and b.flags.c_contiguous
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
            held.append(own)
            with pytest.raises(Exception):
                srv.request(i)
        if len(held) == 4:
            held[1] = None  # goes back to the server; the next requests may use it
    srv.close()
    del srv
    gc.collect()
    for k, own in enumerate(held):
        if own is not None:
            for a, b in zip(want[k % 4], own):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k
                b += 1.0
    ts = [threading.Thread(target=held.__setitem__, args=(k, None)) for k in range(len(held))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()


def test_scene_without_particles():
    srv = Server(budget_bytes=8 << 30)
    s = scene(5, 8, 1)
    empty = SceneSpec(pos=np.zeros((0, 4), np.float32), box_min=(0, 0, 0), box_max=(1, 1, 1), buckets=(32, 16, 8),
                      bodies=s.bodies, rb_buckets=(16, 16, 16))
    ids = [srv.submit(empty, 1), srv.submit(s, 2)]
    while not all(srv.done(i) for i in ids):
        srv.step()
    a = srv.result(ids[0])
    assert a[0].shape == a[1].shape == (0, 4)
    for x, y in zip(alone(s, 2), srv.result(ids[1])):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    srv.close()
