"""gCalcMassDensity and gSPHCalculateForces (no lists: the force launcher
searches by warp) against the oracle over the clouds of the density pass's
test: warp-range edges, single and overfull cells, sprays, shared buckets, wide
cells, a far origin; and an index range whose tables hold more particles than
are asked for.  Bars as for the other launcher tests: density 1e-5 of FP64,
forces 2e-4 of max(|F|, median |F|)."""
import ctypes

import numpy as np
import pytest

from fluidgrid_gb300 import _ffi, build
from oracle import oracle as O
import helpers as T
import test_gpu_density_stage as D

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def p(t):
    return ctypes.c_void_p(t.data_ptr())


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("part", [1.0, 0.6])
@pytest.mark.parametrize("name", list(D.SCENES))
def test_launchers_match_oracle(name, part):
    build.build()
    L = _ffi.load()
    spec = D.SCENES[name]
    ref = T.oracle_grid(spec, spec.pos, spec.vel)
    kc = O.kernels_cache(spec.h)
    L.gInitializeCommonFluidParams(spec.common_params())
    L.gInitializeKernelParams(_ffi.fgr_kernels_cache(kc.kPoly6, kc.kSpikyGradient, kc.kViscosityLaplacian))
    n = max(1, int(spec.n * part))
    opos, ovel = dev(ref["spos"]), dev(ref["svel"])
    start, end = dev(ref["start"].view(np.int32)), dev(ref["end"].view(np.int32))
    ids, key = dev(ref["ids"].view(np.int32)), dev(ref["skeys"].view(np.int32))
    dp = torch.full((spec.n, 2), -7.0, device="cuda")
    L.gCalcMassDensity(p(opos), p(dp), p(key), p(start), p(end), spec.n, spec.gas, spec.rest, spec.mass)
    full = dp.cpu().numpy()
    d64, _ = O.density(ref["spos"], ref["start"], ref["end"], ref["p"], kc, spec.gas, spec.rest, spec.mass, f64=True)
    assert (np.abs(full[:, 0] - d64[:, 0]) / d64[:, 0]).max() <= 1e-5
    some = torch.full((spec.n, 2), -7.0, device="cuda")
    L.gCalcMassDensity(p(opos), p(some), p(key), p(start), p(end), n, spec.gas, spec.rest, spec.mass)
    assert np.array_equal(some.cpu().numpy()[:n], full[:n]) and (some.cpu().numpy()[n:] == -7.0).all()
    vel, forces = dev(spec.vel), torch.zeros(4, device="cuda")
    L.gSPHCalculateForces(p(opos), p(ovel), p(forces), p(dp), p(start), p(end), p(vel), p(ids), n, spec.mass,
                          spec.visc)
    assert L.fgc_last_status() == 0
    nv = O.forces(ref["spos"], ref["svel"], full, ref["start"], ref["end"], ref["ids"], spec.mass, spec.visc,
                  ref["p"], kc, newvel_init=spec.vel)
    got = vel.cpu().numpy()
    done = ref["ids"][:n]
    F = T.force_from_vel(got, spec.vel, spec.dt)[done]
    Fr = T.force_from_vel(nv, spec.vel, spec.dt)[done]
    mag = np.linalg.norm(Fr, axis=1)
    assert (np.linalg.norm(F - Fr, axis=1) / np.maximum(mag, np.median(mag))).max() <= 2e-4
    rest = ref["ids"][n:]
    assert np.array_equal(got[rest], spec.vel[rest])
