"""gSPHCalculateForcesWithSRB with spheres all through the fluid, so that nearly
every particle is near one: static, dynamic and both grids, half-widths 0 to 4,
passes of few and of many warps, sparse and dense targets, against the oracle;
and no more than a small multiple of the time without spheres.  Bar as for the
other launcher tests: 2e-4 of max(|F|, median |F|)."""
import numpy as np
import pytest

from fluidgrid_gb300 import _ffi, build
from fluidgrid_gb300._ffi import float3, int3
from fluidgrid_gb300.scenes import H
from oracle import oracle as O
import helpers as T
import test_gpu_dispersed as D
from test_gpu_reference_api import _sphere_grid, dev, f4, host, p, u32

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
RB = 0.5 * H
FORMS = {"few": (3001, (0.5,)), "many": (D.WIDE + 33, (0.5, 1.5))}


@pytest.fixture(scope="module")
def L():
    build.build()
    return _ffi.load()


def spheres(spec, m, seed):
    rng = np.random.default_rng(seed)
    lo, hi = spec.pos[:, :3].min(0), spec.pos[:, :3].max(0)
    at = np.zeros((m, 4), np.float32)
    at[:, :3] = rng.uniform(lo, hi, (m, 3))
    return at


class Case:
    def __init__(self, L, spec, rel, static, dynamic, m, rnb, cell=RB):
        zero, turn = np.zeros((1, 4), np.float32), np.array([[0, 0, 0, 1]], np.float32)
        dp, self.ref, self.kc = D.launcher_density(spec)
        self.L, self.spec, self.dp, self.rel, self.rnb, self.cell = L, spec, dp, rel, rnb, cell
        self.use = static, dynamic
        self.grids = [_sphere_grid(L, spheres(spec, m, k), zero, turn, rnb, cell) for k in range(2)]
        self.bvel = np.array([[0.3, -0.2, 0.1, 0.0]], np.float32)
        self.t = [dev(x) for x in (self.ref["spos"], self.ref["svel"], dp, spec.vel, self.bvel)]
        self.u = [dev(self.ref[k].view(np.int32)) for k in ("start", "end", "ids")]
        self.none = f4(1), u32(8)

    def __call__(self):
        s, (pos, svel, dp, vel, bvel), (start, end, ids) = self.spec, self.t, self.u
        nf, nu = self.none
        args = []
        for g, use, v in zip(self.grids, self.use, (None, bvel)):
            args += [p(g["pos"] if use else nf)] + ([p(v)] if v is not None else [])
            args += [p(g["start"] if use else nu), p(g["end"] if use else nu), self.rnb if use else 8]
        self.L.gSPHCalculateForcesWithSRB(p(pos), p(svel), p(nf), p(vel), p(dp), p(ids), p(start), p(end), s.n, s.mass,
                                          s.visc, s.fluid_radius, int3(*(self.rel,) * 3), RB,
                                          float3(*(self.cell,) * 3), s.ck, s.ckd, *args, *self.use)
        return vel

    def oracle(self):
        s, ref = self.spec, self.ref
        cp = O.contact_params(s.fluid_radius, RB, s.ck, s.ckd, (self.cell,) * 3, (self.rel,) * 3, 0.003)
        grids = [O.contact_grid(g["ref_pos"], v, g["ref_start"], g["ref_end"], self.rnb) if use else None
                 for g, use, v in zip(self.grids, self.use, (None, self.bvel))]
        return O.forces(ref["spos"], ref["svel"], self.dp, ref["start"], ref["end"], ref["ids"], s.mass, s.visc,
                        ref["p"], self.kc, newvel_init=s.vel, contact=(cp, *grids))


@pytest.mark.parametrize("use", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("form,rel,m,rnb", [("few", 0, 301, 4096), ("few", 1, 2003, 4199), ("few", 2, 2003, 997),
                                            ("few", 4, 301, 4096), ("many", 1, 5003, 4199), ("many", 2, 5003, 8192)])
def test_contact_everywhere(L, form, rel, m, rnb, use):
    n, parts = FORMS[form]
    spec = D.cloud(n, parts, 21)
    c = Case(L, spec, rel, use[0], use[1], m, rnb)
    got = host(c())
    assert L.fgc_last_status() == 0
    F, Fr = T.force_from_vel(got, spec.vel, spec.dt), T.force_from_vel(c.oracle(), spec.vel, spec.dt)
    mag = np.linalg.norm(Fr, axis=1)
    assert (np.linalg.norm(F - Fr, axis=1) / np.maximum(mag, np.median(mag))).max() <= 2e-4
    plain = D.force_launcher(spec, c.dp, c.ref)
    plain[1]()
    assert (host(plain[0]) != got).any(1).sum() > 100, "many particles must be in contact"


def test_spheres_all_through_the_fluid_cost_little(L):
    """4,096 spheres among 262,144 particles: the searches inside the force pass
    made it 3.7 times the pass without spheres, as a pass of their own 2.1."""
    spec = D.cloud(262_144, (0.5,), 22, (1 << 19, 1, 1))
    c = Case(L, spec, 2, True, False, 4096, 32768)
    plain = D.force_launcher(spec, c.dp, c.ref)[1]
    assert D.milliseconds(c) <= 2.9 * D.milliseconds(plain)
