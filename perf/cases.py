"""The work that users of this framework have it do, as cases to time.

Kinds:
  world      one scene in a World (the whole-step API), advanced some steps
             from a given state, as a rollout, a frame of substeps or one
             step of a long run
  batched    many uneven scenes in one World
  host       a host program that owns the state: upload, step, download
  launchers  the reference's doTimeStep order through its own launcher names
  two_way    the reference's two-way fluid/rigid order through its launchers
  served     requests through the continuous-batching Server
  sort       the allocation-free key/index sort

A scene is a jittered block of particles `pack` kernel radii apart in a walled
box (0.5: the spacing that scenes start from; 0.32: the compressed state in
which they spend most of a run, ~110 neighbours in range instead of ~30), with
velocities of a moving fluid and rigid boxes cut by its surface; it starts a
little off the walls, as one that an emitter dropped.  A world's
state is written back to the given one at the start of each pass, through its
device buffers, so that every pass does the same work.
"""
import ctypes
import math

import numpy as np
import torch

from fluidgrid_gb300 import Server, World, _ffi
from fluidgrid_gb300.scenes import Body, SceneSpec

H = 0.0457
CLEAR = 0.1  # the block's distance from the walls at the start
F32 = np.float32


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: a preview or control-loop scene, a few substeps a frame
        {"name": "world_4k", "kind": "world", "n": 4099, "pack": 0.5, "table": 16, "bodies": 0, "spheres": 0,
         "steps": 4},
        # the small dam break: 16,384 particles, 64^3 buckets
        {"name": "dam_break_16k", "kind": "world", "n": 16384, "pack": 0.5, "table": 16, "bodies": 0, "spheres": 0,
         "steps": 4},
        # the headline workload's sizes as the block starts to fall
        {"name": "dam_break_rigid_1m", "kind": "world", "n": 1048576, "pack": 0.5, "table": 2, "bodies": 1,
         "spheres": 4096, "steps": 1},
        # the same in its compressed phase, where most of a long run's time goes
        {"name": "compressed_rigid_1m", "kind": "world", "n": 1000003, "pack": 0.32, "table": 2, "bodies": 1,
         "spheres": 4096, "steps": 1},
        # the largest scene: 4M particles, eight bodies with contact between them
        {"name": "jet_4m", "kind": "world", "n": 4194304, "pack": 0.5, "table": 1, "bodies": 8, "spheres": 4096,
         "steps": 1},
        # uneven independent scenes in shared launches, replayed two steps a graph
        {"name": "batched_32", "kind": "batched", "count": 32, "nmin": 2048, "nmax": 65536, "pack": 0.45, "steps": 2},
        # a host loop that owns the state and reads it back every step
        {"name": "host_loop_262k", "kind": "host", "n": 262144, "pack": 0.45, "table": 2, "bodies": 0,
         "spheres": 0},
        # reference host code with its launchers swapped in: a mid-size fluid, odd sizes
        {"name": "launchers_33k", "kind": "launchers", "n": 33333, "pack": 0.5, "table": 3},
        # and a large one, partly compressed
        {"name": "launchers_1m", "kind": "launchers", "n": 1048576, "pack": 0.4, "table": 2},
        # the same host code with two-way rigid coupling
        {"name": "two_way_262k", "kind": "two_way", "n": 262144, "pack": 0.5, "table": 2, "bodies": 4,
         "spheres": 2048},
        # a burst of requests through the server, until the last result is back
        {"name": "served_12", "kind": "served", "count": 12, "nmin": 4096, "nmax": 131072, "pack": 0.5, "steps": 3},
        # grid keys sorted by a caller that must not allocate
        {"name": "sort_700k", "kind": "sort", "n": 700001, "bits": 21},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["world", "world", "world", "batched", "host", "launchers", "launchers", "two_way", "served",
                       "sort"])
    pack = round(rng.uniform(0.32, 0.5), 3)
    if kind == "world":
        pairs = 4.2 / pack ** 3
        n = min(_log(rng, 2048, 4000000), int(1.6e8 / pairs))
        bodies = max(0, rng.randint(-2, 4))
        return {"kind": kind, "n": n, "pack": pack, "table": rng.choice([1, 2, 3, 4, 16 if n < 300000 else 2]),
                "bodies": bodies, "spheres": _log(rng, 512, 4096) if bodies else 0,
                "steps": 1 if bodies else rng.randint(1, 4 if n < 20000 else 2 if n * pairs < 8e7 else 1)}
    if kind == "batched":
        return {"kind": kind, "count": rng.randint(8, 48), "nmin": 2048, "nmax": _log(rng, 16384, 65536),
                "pack": round(rng.uniform(0.4, 0.5), 3), "steps": rng.randint(1, 2)}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 16384, 1048576), "pack": pack, "table": rng.choice([1, 2, 4]),
                "bodies": rng.randint(0, 2), "spheres": _log(rng, 512, 4096)}
    if kind == "launchers":
        n = min(_log(rng, 4096, 1048576), int(6e7 * pack ** 3 / 4.2))
        return {"kind": kind, "n": n, "pack": pack, "table": rng.choice([1, 2, 3, 4])}
    if kind == "two_way":
        return {"kind": kind, "n": _log(rng, 16384, 400000), "pack": pack, "table": rng.choice([1, 2, 3]),
                "bodies": rng.randint(1, 8), "spheres": _log(rng, 512, 4096)}
    if kind == "served":
        return {"kind": kind, "count": rng.randint(4, 16), "nmin": 4096, "nmax": _log(rng, 32768, 131072),
                "pack": round(rng.uniform(0.45, 0.5), 3), "steps": rng.randint(2, 3)}
    return {"kind": kind, "n": _log(rng, 4096, 1048576), "bits": rng.randint(12, 32)}


# ------------------------------------------------------------------ inputs

def _next_pow2(v):
    p = 1
    while p < v:
        p <<= 1
    return p


def _buckets(n, table):
    """`table` buckets per particle: a power of two, or (table 3) an odd product."""
    if table == 3:
        s = max(17, int(round((3.0 * n) ** (1.0 / 3.0)))) | 1
        return (s, s + 2, s)
    return (_next_pow2(max(n, 4096)) * table, 1, 1)


def _surface(side, count, g):
    """`count` points on the faces of a cube, evenly over the faces."""
    u = torch.rand(count, 2, generator=g, device="cuda", dtype=torch.float64) - 0.5
    face = torch.arange(count, device="cuda") % 6
    p = torch.empty(count, 3, device="cuda", dtype=torch.float64)
    for a in range(3):
        o = [x for x in range(3) if x != a]
        for s in range(2):
            m = face == 2 * a + s
            p[m, a] = s - 0.5
            p[m, o[0]] = u[m, 0]
            p[m, o[1]] = u[m, 1]
    out = np.zeros((count, 4), F32)
    out[:, :3] = (p * side).cpu().numpy()
    return out


def _scene(g, n, pack, buckets, bodies=0, spheres=0, rb_rb=False):
    """A SceneSpec with its state as host arrays."""
    sp = pack * H
    nx = max(4, int(round((2.0 * n) ** (1.0 / 3.0))))
    ny = max(2, -(-n // (nx * nx)))
    i = torch.arange(n, device="cuda")
    cell = torch.stack([i % nx, i // (nx * nx), (i // nx) % nx], 1).double()
    jit = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) - 0.5
    pos = torch.ones(n, 4, device="cuda")
    pos[:, :3] = (cell * sp + CLEAR + jit * (0.2 * sp)).float()
    vel = torch.zeros(n, 4, device="cuda")
    vel[:, :3] = 0.2 * torch.randn(n, 3, generator=g, device="cuda")
    ext = [nx * sp, ny * sp, nx * sp]
    box = (ext[0] * 1.4142 + 2 * CLEAR, max(2 * ext[1], ext[1] + 0.8) + 2 * CLEAR, ext[2] * 1.4142 + 2 * CLEAR)
    r = torch.rand(bodies, 3, generator=g, device="cuda").cpu().numpy().astype(float) if bodies else []
    q = torch.randn(bodies, 4, generator=g, device="cuda").cpu().numpy().astype(float) if bodies else []
    out = []
    for b in range(bodies):
        side = min(0.2 + 0.2 * r[b][1], 0.5 * ext[0])
        c = (CLEAR + ext[0] * (0.2 + 0.6 * r[b][0]), CLEAR + ext[1], CLEAR + ext[2] * (0.2 + 0.6 * r[b][2]))
        quat = [float(F32(x)) for x in q[b] / np.linalg.norm(q[b])]
        out.append(Body(local=_surface(side, spheres, g), mass=50.0 * (side / 0.4) ** 3, position=c,
                        orientation=tuple(quat)))
    return SceneSpec(pos=pos.cpu().numpy(), vel=vel.cpu().numpy(), box_min=(0.0, 0.0, 0.0),
                     box_max=tuple(float(F32(x)) for x in box), buckets=buckets, bodies=out,
                     rb_buckets=(32, 32, 32), rb_rb=rb_rb)


def _specs(case, seed):
    """The case's scenes; the same for prepare() and exact()."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = case["kind"]
    if k in ("batched", "served"):
        rng = np.random.default_rng(77)  # sizes belong to the case, values to the seed
        out = []
        for s in range(case["count"]):
            n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
            bodies = s % 2 if k == "batched" else int(rng.integers(0, 3))
            out.append(_scene(g, n, case["pack"], _buckets(n, 4), bodies, 512 if k == "batched" else 1024))
        return out
    return [_scene(g, case["n"], case["pack"], _buckets(case["n"], case["table"]), case.get("bodies", 0),
                   case.get("spheres", 0), rb_rb=(k == "world" and case["bodies"] > 1))]


def _request_steps(case):
    return [max(1, case["steps"] - s % 3) for s in range(case["count"])]


# ------------------------------------------------------------- the states

class _Mem:
    """A device buffer of a world as torch sees it; the world lives as long as its views."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


_streams = []


def _stream():
    """The program's one stream: its worlds step in turn, none beside another."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _buffer(w, name):
    ptr, nbytes = w.buffer(name)
    if not nbytes:
        return None
    wide = name in ("BODY_X", "BODY_V", "BODY_Q", "BODY_L")
    t = torch.as_tensor(_Mem(w, ptr, nbytes // (8 if wide else 4), "<f8" if wide else "<f4"), device="cuda")
    return t.view(-1, 4)


_BODY_STATE = ("BODY_X", "BODY_V", "BODY_Q", "BODY_L", "BODY_XF", "BODY_VF", "BODY_QF")


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _f4(n):
    return torch.zeros((n, 4), dtype=torch.float32, device="cuda")


def _u32(n):
    return torch.zeros(n, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    k = case["kind"]
    if k == "sort":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        keys = torch.randint(0, 1 << case["bits"], (n,), generator=g, device="cuda")
        keys = torch.where(keys > 0x7fffffff, keys - (1 << 32), keys).to(torch.int32)
        return {"kind": k, "L": _ffi.load(), "in": keys, "ids": torch.arange(n, dtype=torch.int32, device="cuda"),
                "keys": torch.empty_like(keys), "vals": _u32(n), "n": n, "bits": case["bits"]}
    specs = _specs(case, seed)
    if k == "served":
        return {"kind": k, "server": Server(pipeline_depth=2), "specs": specs, "steps": _request_steps(case)}
    if k in ("launchers", "two_way"):
        return _prepare_launchers(k, specs[0])
    stream = _stream()
    w = World(specs, stream=stream.cuda_stream)
    if k == "batched":
        w.set_option("graph_steps", case["steps"])
    names = (() if k == "host" else ("POS", "VEL")) + (_BODY_STATE if w.nbodies else ())
    live = [_buffer(w, b) for b in names]
    s = {"kind": k, "world": w, "stream": stream, "live": live, "start": [t.clone() for t in live],
         "out": dict(zip(names, live))}
    if k == "host":
        s["bufs"] = [torch.empty((w.n, 4), dtype=torch.float32, pin_memory=True).numpy() for _ in range(4)]
        s["bufs"][0][:] = specs[0].pos
        s["bufs"][1][:] = specs[0].vel
    else:
        s["steps"] = case["steps"]
    torch.cuda.synchronize()
    return s


def _prepare_launchers(kind, spec):
    L = _ffi.load()
    n, nb = spec.n, spec.nbuckets
    kc = _kernels(spec.h)
    L.gInitializeCommonFluidParams(spec.common_params())
    L.gInitializeKernelParams(_ffi.fgr_kernels_cache(*kc))
    s = {"kind": kind, "L": L, "spec": spec, "n": n, "nb": nb, "cell": _ffi.float3(*spec.cell_size),
         "pos0": torch.from_numpy(spec.pos).cuda(), "vel0": torch.from_numpy(spec.vel).cuda(),
         "pos": _f4(n), "vel": _f4(n), "opos": _f4(n), "ovel": _f4(n), "forces": _f4(1),
         "dp": torch.zeros((n, 2), dtype=torch.float32, device="cuda"),
         "key": _u32(n), "pid": _u32(n), "start": _u32(nb), "end": _u32(nb)}
    if kind == "two_way":
        B = len(spec.bodies)
        loc = np.concatenate([np.c_[b.local[:, :3], np.full(len(b.local), i, F32)]
                              for i, b in enumerate(spec.bodies)]).astype(F32)
        m, rnb = len(loc), int(np.prod(spec.rb_buckets))
        state = np.zeros((6, B, 4), F32)  # position, velocity, angular momentum, orientation, force, torque
        for i, b in enumerate(spec.bodies):
            state[0, i, :3] = b.position
            state[3, i] = b.orientation
        counts = [len(b.local) for b in spec.bodies]
        offs = np.cumsum([0] + counts)
        flags = np.zeros(m, np.int32)
        flags[offs[:-1]] = 1
        inv = np.zeros((B, 12), F32)
        inv[:, [0, 5, 10]] = 0.00125
        cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        s.update(B=B, m=m, rnb=rnb, loc=cuda(loc), body0=cuda(state), body=cuda(state), flags=cuda(flags),
                 last=cuda((offs[1:] - 1).astype(np.int32)), inv=cuda(inv), inertia=cuda(np.zeros((B, 12), F32)),
                 mass=cuda(np.array([b.mass for b in spec.bodies], F32)), rkey=_u32(m), rid=_u32(m), rworld=_f4(m),
                 rsorted=_f4(m), rstart=_u32(rnb), rend=_u32(rnb), F=_f4(m), T=_f4(m), bkey=_u32(m), bidx=_u32(m),
                 Fs=_f4(m), Ts=_f4(m), Fscan=_f4(m), Tscan=_f4(m), none_f=_f4(1), none_u=_u32(8))
    return s


# ------------------------------------------------------------------- a pass

def run(state):
    return _RUN[state["kind"]](state)


def _run_world(s):
    w = s["world"]
    with torch.cuda.stream(s["stream"]):
        for live, start in zip(s["live"], s["start"]):
            live.copy_(start)
        w.step(s["steps"])
    # the bodies' FP32 state is what the contact kernels read
    return {k: v for k, v in s["out"].items() if k in ("POS", "VEL", "BODY_XF", "BODY_VF", "BODY_QF")}


def _run_host(s):
    hp, hv, op, ov = s["bufs"]
    with torch.cuda.stream(s["stream"]):
        for live, start in zip(s["live"], s["start"]):
            live.copy_(start)
        s["world"].e2e_steps(1, hp, hv, op, ov)
    return [op, ov]


def _run_served(s):
    srv = s["server"]
    ids = [srv.submit(spec, k) for spec, k in zip(s["specs"], s["steps"])]
    waiting = set(ids)
    while waiting:
        srv.step()
        waiting = {i for i in waiting if not srv.done(i)}
    return [srv.result(i) for i in ids]


def _run_sort(s):
    s["keys"].copy_(s["in"])
    s["vals"].copy_(s["ids"])
    _ffi.check(s["L"].fg_sort_pairs_noalloc(_p(s["keys"]), _p(s["vals"]), s["bits"], s["n"], None),
               "fg_sort_pairs_noalloc")
    return [s["keys"], s["vals"]]


def _grid_and_density(s):
    L, spec, n, nb = s["L"], s["spec"], s["n"], s["nb"]
    s["pos"].copy_(s["pos0"])
    s["vel"].copy_(s["vel0"])
    L.gCalcHashKey(_p(s["key"]), _p(s["pid"]), _p(s["pos"]), n, nb, s["cell"])
    L.gSort(_p(s["key"]), _p(s["pid"]), n)
    L.gFindCellOffsetOrderingPosVel(_p(s["start"]), _p(s["end"]), _p(s["key"]), _p(s["pid"]), _p(s["pos"]),
                                    _p(s["opos"]), _p(s["vel"]), _p(s["ovel"]), n, nb)
    L.gCalcMassDensity(_p(s["opos"]), _p(s["dp"]), _p(s["key"]), _p(s["start"]), _p(s["end"]), n, spec.gas,
                       spec.rest, spec.mass)


def _integrate(s):
    s["L"].gSPHIntegrate(_p(s["pos"]), _p(s["vel"]), _p(s["forces"]), s["n"], _p(s["dp"]), _p(s["start"]),
                         _p(s["end"]))


def _run_launchers(s):
    L, spec, n = s["L"], s["spec"], s["n"]
    _grid_and_density(s)
    L.gSPHCalculateForces(_p(s["opos"]), _p(s["ovel"]), _p(s["forces"]), _p(s["dp"]), _p(s["start"]), _p(s["end"]),
                          _p(s["vel"]), _p(s["pid"]), n, spec.mass, spec.visc)
    _integrate(s)
    return {k: s[k] for k in ("pos", "vel", "dp", "key", "pid", "start")}


def _run_two_way(s):
    L, spec, n, m, B, rnb, nb = s["L"], s["spec"], s["n"], s["m"], s["B"], s["rnb"], s["nb"]
    s["body"].copy_(s["body0"])
    x, v, am, q, F, T = s["body"]
    r = spec.rb_radius
    rcell = _ffi.float3(r, r, r)
    _grid_and_density(s)
    L.gCalcHashKeyWithOffset(_p(s["rkey"]), _p(s["rid"]), _p(x), _p(q), _p(s["loc"]), _p(s["rworld"]), m, rcell, rnb)
    L.fgc_sort_pairs(_p(s["rkey"]), _p(s["rid"]), int(math.ceil(math.log2(rnb))), m)
    L.gFindCellOffsetOrderingPos(_p(s["rstart"]), _p(s["rend"]), _p(s["rkey"]), _p(s["rid"]), _p(s["rworld"]),
                                 _p(s["rsorted"]), m, rnb)
    L.gCalculateRigidBodyForcesFromFluids(_p(s["rsorted"]), _p(v), _p(x), _p(s["F"]), _p(s["T"]), _p(s["rstart"]),
                                          _p(s["rend"]), m, rcell, r, rnb, _p(s["opos"]), _p(s["ovel"]),
                                          _p(s["start"]), _p(s["end"]), spec.fluid_radius, s["cell"], nb,
                                          _ffi.int3(*spec.r2f_rel), spec.ck, spec.ckd)
    L.gSPHCalculateForcesWithSRB(_p(s["opos"]), _p(s["ovel"]), _p(s["forces"]), _p(s["vel"]), _p(s["dp"]),
                                 _p(s["pid"]), _p(s["start"]), _p(s["end"]), n, spec.mass, spec.visc,
                                 spec.fluid_radius, _ffi.int3(*spec.f2r_rel), r, rcell, spec.ck, spec.ckd,
                                 _p(s["none_f"]), _p(s["none_u"]), _p(s["none_u"]), 8, _p(s["rsorted"]), _p(v),
                                 _p(s["rstart"]), _p(s["rend"]), rnb, False, True)
    L.gCopyRBDataToParticle(_p(s["bkey"]), _p(s["bidx"]), _p(s["F"]), m)
    L.fgc_sort_pairs(_p(s["bkey"]), _p(s["bidx"]), 8, m)
    L.gReorderForceTorque(_p(s["Fs"]), _p(s["Ts"]), _p(s["F"]), _p(s["T"]), _p(s["bidx"]), m)
    L.fgc_segmented_scan_float4(_p(s["Fscan"]), _p(s["Fs"]), _p(s["flags"]), m)
    L.fgc_segmented_scan_float4(_p(s["Tscan"]), _p(s["Ts"]), _p(s["flags"]), m)
    L.gAddForceTorque(_p(s["Fscan"]), _p(s["Tscan"]), _p(s["Fs"]), _p(F), _p(T), _p(s["last"]), B)
    L.gIntegrateRB(_p(x), _p(s["mass"]), _p(v), _p(F), B, spec.dt, _ffi.float4(*spec.rb_gravity),
                   _ffi.float3(*spec.box_min), _ffi.float3(*spec.box_max), _p(am), _p(T), _p(s["inertia"]), _p(q),
                   _p(s["inv"]), spec.rb_vlimit)
    _integrate(s)
    return {"pos": s["pos"], "vel": s["vel"], "dp": s["dp"], "key": s["key"], "pid": s["pid"],
            "sphere_force": s["F"], "sphere_torque": s["T"], "body": s["body"]}


_RUN = {"world": _run_world, "batched": _run_world, "host": _run_host, "served": _run_served, "sort": _run_sort,
        "launchers": _run_launchers, "two_way": _run_two_way}


# -------------------------------------------------------------------- work

def work(case):
    k = case["kind"]
    if k == "sort":
        return {"bytes": 16.0 * case["n"], "flops": 0.0}
    if k in ("batched", "served"):
        rng = np.random.default_rng(77)
        sizes = []
        for s in range(case["count"]):
            sizes.append(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]))))
            if k == "served":
                rng.integers(0, 3)
        steps = _request_steps(case) if k == "served" else [case["steps"]] * case["count"]
        n, ns = sum(sizes), sum(a * b for a, b in zip(sizes, steps))
    else:
        n = case["n"]
        ns = n * case.get("steps", 1)
    # positions and velocities in and out; each pair in range: its density
    # term (11 operations) and its force term (38)
    pairs = 4.0 / 3.0 * math.pi / case["pack"] ** 3
    return {"bytes": 64.0 * n, "flops": ns * pairs * 49.0}


# --------------------------------------------------- the same in 64 bits

PX, PY, PZ = 73856093, 19349663, 83492791
EMPTY = 0xffffffff


def _kernels(h):
    h, pi = float(F32(h)), float(F32(3.14159265))
    return 315.0 / (64.0 * pi * h ** 9), -45.0 / (pi * h ** 6), 45.0 / (pi * h ** 6)


def _axis(p, cell, o):
    """Cell index along one axis of the FP32 coordinate p + o cells, as the hash rounds it."""
    c = torch.tensor(F32(cell), device="cuda")
    off = torch.tensor(F32(F32(cell) * F32(o)), device="cuda")
    return (((p + off) if o else p) + torch.tensor(F32(5000.0), device="cuda")).div(c).to(torch.int32).long()


def _bucket(p32, cell, nb, o=(0, 0, 0)):
    k = [(_axis(p32[:, a], cell[a], o[a]) * c) & EMPTY for a, c in enumerate((PX, PY, PZ))]
    return (k[0] ^ k[1] ^ k[2]) % nb


class _Grid:
    """Points sorted by bucket, and the buckets' ranges; pos32: the coordinates that are hashed."""

    def __init__(self, pos, cell, nb, pos32=None):
        self.cell, self.nb = cell, nb
        self.key, self.order = torch.sort(_bucket(pos.float() if pos32 is None else pos32, cell, nb), stable=True)
        self.pos = pos[self.order]
        self.count = torch.bincount(self.key, minlength=nb)
        self.start = torch.cumsum(self.count, 0) - self.count

    def visit(self, q, rel, fn):
        """fn(candidate indices, whether each is one) over the buckets around the points q."""
        q32 = q.float()
        for z in range(-rel[2], rel[2] + 1):
            for y in range(-rel[1], rel[1] + 1):
                for x in range(-rel[0], rel[0] + 1):
                    b = _bucket(q32, self.cell, self.nb, (x, y, z))
                    st, n = self.start[b], self.count[b]
                    for k in range(int(n.max()) if len(n) else 0):
                        m = k < n
                        fn(torch.where(m, st + k, 0), m)


def _contact(q, vq, body_q, grid, v, body, rel, mind, k, kd):
    """Spring and damper contact of the points q with the grid's points (not with those of their own body)."""
    acc = torch.zeros_like(q)

    def one(j, m):
        r = grid.pos[j] - q
        lg = r.norm(dim=1)
        m = m & (lg < mind)
        if body_q is not None:
            m = m & (body[j] != body_q)
        nrm = r / torch.where(m, lg, 1.0)[:, None]
        c = k * lg - kd * (nrm * (v[j] - vq)).sum(1)
        acc.add_(torch.where(m, c, 0.0)[:, None] * nrm)

    grid.visit(q, rel, one)
    return acc


def _f(x):
    return float(F32(x))


class _Sim:
    """One scene advanced in 64 bits (cells and buckets from FP32 coordinates, as the path defines them)."""

    def __init__(self, spec):
        self.s = spec
        self.pos = torch.from_numpy(spec.pos).cuda().double()[:, :3]
        self.vel = torch.from_numpy(spec.vel).cuda().double()[:, :3]
        B = len(spec.bodies)
        d = lambda a, k: torch.tensor(np.asarray(a, np.float64).reshape(B, k), device="cuda")  # noqa: E731
        self.x = d([[_f(c) for c in b.position] for b in spec.bodies], 3)
        self.q = d([[_f(c) for c in b.orientation] for b in spec.bodies], 4)
        self.v = torch.zeros(B, 4, device="cuda", dtype=torch.float64)
        self.L = torch.zeros(B, 4, device="cuda", dtype=torch.float64)
        if B:
            self.local = torch.from_numpy(np.concatenate([b.local[:, :3] for b in spec.bodies])).cuda().double()
            self.body = torch.from_numpy(np.repeat(np.arange(B), [len(b.local) for b in spec.bodies])).cuda()
        self.sphere_force = self.sphere_torque = None

    def step(self):
        s = self.s
        h, h2, dt = _f(s.h), _f(F32(s.h) * F32(s.h)), _f(s.dt)
        poly, spiky, lap = _kernels(s.h)
        mass, gas, rest = _f(s.mass), _f(s.gas), _f(s.rest)
        g = _Grid(self.pos, s.cell_size, s.nbuckets)
        P, V = g.pos, self.vel[g.order]
        w = torch.zeros(len(P), device="cuda", dtype=torch.float64)

        def density(j, m):
            r2 = (P - P[j]).square().sum(1)
            w.add_(torch.where(m & (r2 <= h2), h2 - r2, 0.0) ** 3)

        g.visit(P, (1, 1, 1), density)
        rho = mass * poly * w
        press = gas * (rho - rest)
        rho = rho.clamp(min=1.0)
        self.dp = torch.stack([rho, press], 1)
        acc = torch.zeros_like(P)
        me = torch.arange(len(P), device="cuda")

        def force(j, m):
            d = P - P[j]
            l2 = d.square().sum(1)
            m = m & (l2 <= h2) & (j != me)
            l = torch.where(m, l2, 1.0).sqrt()
            a = torch.where(m, (h - l) / (rho * rho[j]), 0.0)
            acc.add_((-spiky * (h - l) * (press + press[j]) / l * a)[:, None] * d)
            acc.add_((lap * _f(s.visc) * a)[:, None] * (V[j] - V))

        g.visit(P, (1, 1, 1), force)
        F = acc * mass + torch.tensor([_f(c) for c in s.gravity], device="cuda", dtype=torch.float64)
        if s.bodies:
            sph = self.spheres(torch.float64)
            rg = _Grid(sph, (s.rb_radius,) * 3, int(np.prod(s.rb_buckets)), self.spheres(torch.float32))
            sv, sb = self.v[self.body][:, :3], self.body
            near = _f(s.fluid_radius) + _f(s.rb_radius) + _f(0.003)
            lo, hi = sph.min(0).values - near, sph.max(0).values + near
            hit = torch.nonzero(((P >= lo) & (P <= hi)).all(1))[:, 0]
            F[hit] += _contact(P[hit], V[hit], None, rg, sv[rg.order], None, s.f2r_rel, near, _f(s.ck), _f(s.ckd))
            self.bodies(sph, sv, sb, g, V, rg)
        F += self.walls(P, V)
        sp = F.norm(dim=1)
        F = torch.where(sp > s.vlimit, s.vlimit / sp, 1.0)[:, None] * F
        self.vel = torch.empty_like(V)
        self.vel[g.order] = V + F * dt
        self.pos = self.pos + self.vel * dt

    def walls(self, P, V):
        s = self.s
        F = torch.zeros_like(P)
        for a in range(3):
            for sign, edge in ((1.0, s.box_min[a]), (-1.0, s.box_max[a])):
                d = _f(0.003043174) - sign * (P[:, a] - _f(edge))
                F[:, a] += torch.where(d > _f(0.00001), sign * (20000.0 * d - 256.0 * sign * V[:, a]), 0.0)
        return F

    def spheres(self, dtype):
        """conj(q) p q + centre; in FP32 as the grid hashes it, each operation rounded."""
        q, p = self.q[self.body].to(dtype), self.local.to(dtype)
        p = torch.cat([p, torch.zeros_like(p[:, :1])], 1)
        conj = torch.cat([-q[:, :3], q[:, 3:]], 1)
        return self._product(self._product(conj, p), q)[:, :3] + self.x[self.body].to(dtype)

    @staticmethod
    def _product(a, b):
        ax, ay, az, aw = a.unbind(1)
        bx, by, bz, bw = b.unbind(1)
        return torch.stack([(aw * bx + bw * ax) + (ay * bz - az * by), (aw * by + bw * ay) + (az * bx - ax * bz),
                            (aw * bz + bw * az) + (ax * by - ay * bx), aw * bw - ((ax * bx + ay * by) + az * bz)], 1)

    def bodies(self, sph, sv, sb, g, V, rg):
        s = self.s
        B = len(s.bodies)
        mind = _f(s.rb_radius) + _f(s.fluid_radius) + _f(0.0001)
        f = _contact(sph, sv, None, g, V, None, s.r2f_rel, mind, _f(s.ck), _f(s.ckd))
        if s.rb_rb:
            mind = 2 * _f(s.rb_radius) + _f(0.001)
            f = f + _contact(sph, sv, sb, rg, sv[rg.order], sb[rg.order], (1, 1, 1), mind, _f(s.rbrb_k), _f(s.rbrb_kd))
        t = torch.linalg.cross(sph - self.x[sb], f)
        idx = sb.double()[:, None]
        self.sphere_force, self.sphere_torque = torch.cat([f, idx], 1)[rg.order], torch.cat([t, idx], 1)[rg.order]
        z = torch.zeros(B, 4, device="cuda", dtype=torch.float64)
        F, T = z.index_add(0, sb, torch.cat([f, idx], 1)), z.index_add(0, sb, torch.cat([t, idx], 1))
        self.F, self.T = F, T
        sp = F.norm(dim=1)
        F = torch.where(sp > s.rb_vlimit, s.rb_vlimit / sp, 1.0)[:, None] * F
        dt = _f(s.dt)
        m = torch.tensor([[_f(b.mass)] for b in s.bodies], device="cuda", dtype=torch.float64)
        grav = torch.tensor([_f(c) for c in s.rb_gravity], device="cuda", dtype=torch.float64)
        self.v = self.v + (F + grav) / m * dt * dt
        x = self.x + self.v[:, :3] * dt
        self.L = (self.L + T * dt) * _f(0.9)
        inv = _f(0.00125)  # times the identity: R I R^T L = inv L
        om = torch.cat([inv * self.L[:, :3], torch.zeros_like(self.L[:, :1])], 1)
        om = 0.5 * self._product(om, self.q)
        q = self.q + self._product(om * dt * _f(0.1), self.q)
        self.q = q / q.norm(dim=1, keepdim=True)
        v = self.v.clone()
        for a in (1, 0, 2):
            lo, hi = _f(s.box_min[a]), _f(s.box_max[a])
            out = x[:, a] < lo if a == 1 else (x[:, a] <= lo) | (x[:, a] >= hi)
            x[:, a] = x[:, a].clamp(min=lo) if a == 1 else x[:, a].clamp(lo, hi)
            v[:, a] = torch.where(out, _f(-0.7) * v[:, a], v[:, a])
        self.x, self.v = x, v

    def state(self):
        n, o = len(self.pos), {"device": "cuda", "dtype": torch.float64}
        return torch.cat([self.pos, torch.ones(n, 1, **o)], 1), torch.cat([self.vel, torch.zeros(n, 1, **o)], 1)


def _x4(sim):
    return torch.cat([sim.x, torch.zeros_like(sim.x[:, :1])], 1)


def exact(case, seed):
    k = case["kind"]
    if k == "sort":
        return None
    sims = [_Sim(s) for s in _specs(case, seed)]
    steps = _request_steps(case) if k == "served" else [case.get("steps", 1)] * len(sims)
    for sim, ns in zip(sims, steps):
        for _ in range(ns):
            sim.step()
    if k == "served":
        return [sim.state() for sim in sims]
    if k == "host":
        return list(sims[0].state())
    if k in ("world", "batched"):
        st = [sim.state() for sim in sims]
        out = {"POS": torch.cat([a for a, _ in st]), "VEL": torch.cat([b for _, b in st])}
        rb = [sim for sim in sims if sim.s.bodies]
        if rb:
            out.update(BODY_XF=torch.cat([_x4(b) for b in rb]), BODY_VF=torch.cat([b.v for b in rb]),
                       BODY_QF=torch.cat([b.q for b in rb]))
        return out
    sim = sims[0]
    pos, vel = sim.state()
    out = {"pos": pos, "vel": vel, "dp": sim.dp, "key": None, "pid": None}
    if k == "launchers":
        return dict(out, start=None)
    body = torch.stack([_x4(sim), sim.v, sim.L, sim.q, sim.F, sim.T])
    return dict(out, sphere_force=sim.sphere_force, sphere_torque=sim.sphere_torque, body=body)
