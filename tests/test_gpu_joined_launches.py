"""That small worlds do join the steps of a call, and where they do not: the
graph launches of steps of which no order refresh or capacity check falls
between, joined by fours and twos once a single step has been replayed 16
times; one a step with graph_steps = 1 chosen, above the size limit, and in
calls of one step."""
import numpy as np
import pytest

from fluidgrid_gb300 import World, build
import test_gpu_joined_steps as J
import test_gpu_sort_variants as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def launches(spec, calls, chosen=None):
    w = World([spec])
    w.set_option("autotune_period", 0)
    w.set_option("order_period", 0)   # one refresh, at step 0
    w.set_option("list_autogrow", 0)  # no capacity checks
    if chosen:
        w.set_option("graph_steps", chosen)
    for k in calls:
        w.step(k)
    n = w.graph_launches()
    w.close()
    return n


def test_steps_are_joined():
    spec = J.scene(0)
    # step 0 builds the graph, 16 replays follow; then 47 steps: 11 of four, one of two, one alone
    assert launches(spec, (64,)) == 17 + 13
    assert launches(spec, (17, 2, 2, 3, 1)) == 17 + 1 + 1 + 2 + 1
    assert launches(J.scene(1), (64,)) == 17 + 13


def test_steps_are_not_joined():
    assert launches(J.scene(0), (64,), chosen=1) == 64
    assert launches(J.scene(0), (1,) * 40) == 40
    big = S.scene("lattice")
    big.pos, big.vel = np.tile(big.pos, (2, 1))[:98_305].copy(), np.tile(big.vel, (2, 1))[:98_305].copy()
    big.pos[S.N:, 1] += 3.0
    assert launches(big, (40,)) == 40


def test_chosen_joins_stay():
    # the refresh's step, seven of eight, and seven left over
    assert launches(J.scene(0), (64,), chosen=8) == 1 + 7 + 7
