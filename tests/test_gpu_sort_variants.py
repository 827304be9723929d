"""The world's sorts above the size that one launch sorts (65,536 pairs): three
kernels a pass out of place from implied ids, one kernel a pass, and counting,
over the digit widths (odd and even numbers of passes) and over particles in
order, at random and all in few cells; keys and ids against a stable sort.  The
target order, sorted the same way, changes no bit of a step."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, build
from fluidgrid_gb300.scenes import H, SceneSpec

pytestmark = pytest.mark.gpu
N = 70_001


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def scene(form):
    rng = np.random.default_rng(5)
    nx = 42
    i = np.arange(N)
    pos = np.ones((N, 4), np.float32)
    pos[:, :3] = np.stack([i % nx, i // (nx * nx), i // nx % nx], 1) * (0.5 * H) + 0.1
    if form == "random":
        pos = rng.permutation(pos)
    if form == "few_cells":
        pos[:, :3] = 0.1 + 40.0 * H * rng.integers(0, 12, (N, 1)) + rng.uniform(0, 2e4 * H, (N, 3)) * (i % 3 == 0)[:, None]
    vel = np.zeros((N, 4), np.float32)
    vel[:, :3] = rng.normal(0, 0.05, (N, 3))
    return SceneSpec(pos=pos, vel=vel, box_min=(0,) * 3, box_max=(2000,) * 3, buckets=(1 << 17, 1, 1))


def stepped(form, variant, bits, order=2, stages=None):
    w = World([scene(form)])
    w.set_option("autotune_period", 0)
    w.set_option("one_pass_sort", variant)
    w.set_option("digit_bits", bits)
    w.set_option("target_order", order)
    if stages is not None:
        w.set_stages(stages)
    w.step(1)
    out = {k: w.read(k) for k in ("KEYS_UNSORTED", "KEYS", "IDS", "VEL")}
    w.close()
    return out


@pytest.mark.parametrize("bits", range(1, 9))
@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("form", ["lattice", "random", "few_cells"])
def test_keys_and_ids_are_the_stable_order(form, variant, bits):
    HASH_AND_SORT = 3  # the grid's first two stages: few_cells has more pairs than a test should add up
    g = stepped(form, variant, bits, stages=HASH_AND_SORT if form == "few_cells" else None)
    order = np.argsort(g["KEYS_UNSORTED"], kind="stable")
    assert np.array_equal(g["KEYS"], g["KEYS_UNSORTED"][order]), "keys"
    assert np.array_equal(g["IDS"], order.astype(np.uint32)), "ids"


@pytest.mark.parametrize("bits", [1, 3, 5, 8])
def test_the_target_order_changes_no_bit(bits):
    a, b = stepped("random", 2, bits, order=0), stepped("random", 2, bits, order=2)
    assert np.array_equal(a["VEL"].view(np.uint32), b["VEL"].view(np.uint32))


@pytest.mark.parametrize("n,tuned", [(20_011, False), (N, True)])
def test_the_tuner_tries_digit_widths_where_a_sort_goes_by_them(n, tuned):
    spec = scene("lattice")
    spec.pos, spec.vel = spec.pos[:n].copy(), spec.vel[:n].copy()
    w = World([spec])
    w.set_option("one_pass_sort", 0)
    w.set_option("digit_bits", 5)
    w.set_option("autotune_tiles", 2)  # the digit width only: 6 to 8
    w.set_option("autotune_period", 4)
    w.step(12)
    assert (w.get_option("digit_bits") != 5) == tuned
    w.close()
