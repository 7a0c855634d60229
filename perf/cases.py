"""What the framework's users have it do, as cases that can be timed and checked.

Each case is one pass of a user's program through the public entry points
(snow_gb300.api, and the C ABI's device sort), at sizes and with the options
that the scene generators, tests and benchmark of this repository use. Inputs
are made from a seed with torch on the GPU and handed over as pinned host
arrays, which is what the upload and download entry points take.

Kinds of pass:
  scene      a program that runs one simulation after another in a resident
             scene: discard the pending grid sums, upload an initial state,
             init, step, download the particle state
  live       a viewer: one step of a running scene, then its state
  monitor    as `scene`, but stepping one by one with the bulk statistics of
             every step read while the next one runs
  batch      many scenes of uneven size advanced together, then downloaded
  serve      simulation jobs submitted to the server, waited for and fetched
  reference  the shaders' own arithmetic on their std140 buffers
  sort       the binning sort on device buffers of the caller
"""
import ctypes as C
import math

import numpy as np
import torch

from snow_gb300 import api, native as N, scenes

DEV = "cuda" if torch.cuda.is_available() else "cpu"
CRIT = dict(poisson=0.2, crit_compression=2.5e-2, crit_stretch=7.5e-3)


# ---- the cases -----------------------------------------------------------------
def listed():
    return [
        # the smallest call: a small scene in a viewer, one step and its particles per frame
        dict(name="viewer 4k", kind="live", shape="snowball", n=4096, edge=32, dt=1e-4, steps=1, warm=False),
        # the binning sort as an engine that owns its device memory calls it, at its largest
        dict(name="sort 262144", kind="sort", n=262144, bits=24),
        # a snowball hitting the ground, 100 steps: the small plain simulation
        dict(name="snowball 32k", kind="scene", shape="snowball", n=32768, edge=64, dt=1e-4, steps=100, warm=False),
        # the same arithmetic as the shaders', for programs that compare with them
        dict(name="reference 32k", kind="reference", shape="snowball", n=32768, edge=64, dt=1e-4, steps=20, warm=False),
        # watching a run: statistics after every step
        dict(name="monitored 262k", kind="monitor", shape="two", n=262144, edge=160, dt=2e-5, steps=32, warm=True),
        # a long time step (half a cell per step): particles are re-binned all the time
        dict(name="long steps 300k", kind="scene", shape="two", n=300007, edge=200, dt=5e-4, steps=20, warm=True),
        # stiff material and a rough velocity field with the semi-implicit update
        dict(name="semi-implicit 131k", kind="scene", shape="jitter", n=131072, edge=128, dt=5e-4, steps=8, warm=False, beta=1.0),
        # many uneven scenes at once, as a parameter study does
        dict(name="batch 24", kind="batch", scenes=24, n_min=10000, n_max=500000, dt=1e-4, steps=40),
        # jobs of uneven size and length arriving at the server together
        dict(name="serve 10", kind="serve", scenes=10, n_min=20000, n_max=200000, dt=1e-4, steps_min=50, steps_max=150),
        # the ordinary large scene: two snowballs in the middle of their collision
        dict(name="two snowballs 1M", kind="scene", shape="two", n=1 << 20, edge=256, dt=2e-5, steps=50, warm=True),
        # a block dropped onto a sphere in a large, mostly empty grid
        dict(name="block on sphere 1.5M", kind="scene", shape="block", n=1500001, edge=384, dt=2e-5, steps=24, warm=False),
        # the largest scene
        dict(name="two snowballs 16M", kind="scene", shape="two", n=1 << 24, edge=512, dt=2e-5, steps=12, warm=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _odd(rng, lo, hi):
    return int(_log(rng, lo, hi)) | 1


def _edge_for(n, rng, two):
    """A grid that holds the shape with room to move, as the generators match
    it: about five radii, not always a multiple of the block size."""
    r = (3.0 * n / 8.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
    e = (7.0 if two else 5.0) * r * rng.uniform(1.0, 1.3)
    return max(32, min(512, int(e)))


def draw(rng):
    kind = rng.choice(["live", "scene", "scene", "scene", "scene", "scene", "monitor", "batch", "serve", "reference",
                       "sort", "implicit"])
    if kind == "sort":
        return dict(kind="sort", n=_odd(rng, 1000, 262143), bits=rng.randint(9, 32))
    if kind == "live":
        n = _odd(rng, 1000, 60000)
        return dict(kind="live", shape="snowball", n=n, edge=_edge_for(n, rng, False), dt=_log(rng, 2e-5, 2e-4),
                    steps=rng.randint(1, 4), warm=rng.random() < 0.5)
    if kind == "reference":
        n = _odd(rng, 2000, 60000)
        return dict(kind="reference", shape="snowball", n=n, edge=max(48, min(96, _edge_for(n, rng, False))), dt=1e-4,
                    steps=rng.randint(2, 20), warm=False)
    if kind == "batch":
        return dict(kind="batch", scenes=rng.randint(2, 24), n_min=10000, n_max=_odd(rng, 60000, 500000), dt=1e-4,
                    steps=rng.randint(10, 40))
    if kind == "serve":
        return dict(kind="serve", scenes=rng.randint(2, 10), n_min=20000, n_max=_odd(rng, 40000, 200000), dt=1e-4,
                    steps_min=20, steps_max=rng.randint(50, 150))
    if kind == "implicit":
        n = _odd(rng, 20000, 260000)
        return dict(kind="scene", shape="jitter", n=n, edge=_edge_for(n, rng, True), dt=5e-4, steps=rng.randint(2, 8),
                    warm=False, beta=rng.choice([0.5, 1.0]))
    if kind == "monitor":
        n = _odd(rng, 50000, 500000)
        return dict(kind="monitor", shape="two", n=n, edge=_edge_for(n, rng, True), dt=2e-5, steps=rng.randint(8, 32),
                    warm=True)
    shape = rng.choice(["snowball", "two", "two", "block"])
    n = _odd(rng, 8000, 8000000)
    edge = _edge_for(n, rng, shape != "snowball")
    # up to half a cell per step at the shapes' 5 m/s (2 m/s for the others)
    dt = _log(rng, 0.02, 0.5) / edge / (5.0 if shape == "two" else 2.0)
    dt = min(dt, 0.4 / edge / math.sqrt(1.4e5 / 400.0))
    return dict(kind="scene", shape=shape, n=n, edge=edge, dt=dt, steps=rng.randint(8, 60 if n < 1500000 else 12),
                warm=rng.random() < 0.6)


# ---- inputs -----------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _fill(kind, center, n, h, g, aspect=(1.0, 1.0, 1.0)):
    """n points of a jittered lattice (8 per cell, +-h/8) nearest to `center`
    in the norm of a sphere or of a box with the given aspect."""
    asp = torch.tensor(aspect, dtype=torch.float64, device=DEV)
    cells = n / 8.0
    if kind == "sphere":
        half = torch.full((3,), (3.0 * cells / (4.0 * math.pi)) ** (1.0 / 3.0) * 1.05 + 2, dtype=torch.float64)
    else:
        half = torch.tensor(aspect, dtype=torch.float64) * (cells / float(np.prod(aspect))) ** (1.0 / 3.0) / 2 * 1.05 + 2
    axes = []
    for k in range(3):
        lo, hi = math.floor((center[k] - float(half[k]) * h) / h), math.ceil((center[k] + float(half[k]) * h) / h)
        axes.append((torch.arange(2 * lo, 2 * hi, device=DEV, dtype=torch.float64) + 0.5) * (h / 2))
    p = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    p += (torch.rand(p.shape, generator=g, device=DEV, dtype=torch.float64) - 0.5) * (h / 4)
    d = (p - torch.tensor(center, dtype=torch.float64, device=DEV)) / asp
    key = d.square().sum(1) if kind == "sphere" else d.abs().amax(1)
    keep = torch.sort(torch.topk(key, n, largest=False, sorted=False).indices).values
    return p[keep].to(torch.float32)


def _walls(edge):
    h = 1.0 / edge
    return scenes.walls((0.0, 0.0, 0.0), (edge,) * 3, h)


def _uniform(g, lo, hi, n=1):
    r = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo
    return [float(x) for x in r]


def _shape(case, g):
    """(positions, velocities, colliders) of a single scene, float32 on the GPU."""
    n, edge = case["n"], case["edge"]
    h, coll = 1.0 / edge, _walls(edge)
    cells = n / 8.0
    off = _uniform(g, -0.4 * h, 0.4 * h, 3)
    if case["shape"] == "snowball":  # just above the ground, falling
        r = (3.0 * cells / (4.0 * math.pi)) ** (1.0 / 3.0) * h
        x = _fill("sphere", (0.5 + off[0], 5.0 * h + r + off[1], 0.5 + off[2]), n, h, g)
        v = torch.tensor([0.0, -2.0, 0.0], device=DEV).repeat(n, 1)
    elif case["shape"] in ("two", "jitter"):  # touching, head-on at 5 m/s each
        r = (3.0 * cells / 2 / (4.0 * math.pi)) ** (1.0 / 3.0) * h
        gap = 0.5 * h + r
        a = _fill("sphere", (0.5 - gap + off[0], 0.5 + off[1], 0.5), n // 2, h, g)
        b = _fill("sphere", (0.5 + gap + off[0], 0.5 + off[2], 0.5), n - n // 2, h, g)
        x = torch.cat([a, b])
        v = torch.zeros_like(x)
        v[: len(a), 0], v[len(a):, 0] = 5.0, -5.0
        if case["shape"] == "jitter":
            v += torch.randn(v.shape, generator=g, device=DEV)
    else:  # a block on a sphere collider, moving down
        aspect = (0.6, 0.3, 0.6)
        x = _fill("box", (0.5 + off[0], 0.6 + off[1], 0.5 + off[2]), n, h, g, aspect)
        lo, hi = x.amin(0).tolist(), x.amax(0).tolist()
        r = 0.25 * (hi[0] - lo[0])
        coll.append(scenes.Collider(pos=(0.5, lo[1] - r, 0.5), type=scenes.COLLIDER_SPHERE, radius=float(r)))
        v = torch.tensor([0.0, -2.0, 0.0], device=DEV).repeat(n, 1)
    return x, v, coll


def _deformation(x, g):
    """Smooth deformation gradients of a run that is under way: F_E within a
    per cent or so of a rotation, F_P with determinants about one."""
    ph = torch.rand(2, 9, generator=g, device=DEV, dtype=torch.float64) * 2 * math.pi
    kw = (torch.rand(2, 9, 3, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * 60
    eye = torch.eye(3, device=DEV).reshape(9)
    fe, fp = (torch.sin(x @ kw[i].T.float() + ph[i].float()) for i in range(2))
    return eye + 4e-3 * fe, eye + 2e-2 * fp


def _host(t):
    """A pinned host array with t's values."""
    if t is None:
        return None
    if DEV == "cpu":
        return t.numpy()
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def _scene(case, x, v, coll, young, hardening):
    edge = case["edge"]
    h = 1.0 / edge
    n = len(x)
    s = scenes.Scene(grid_pos=(0.0, 0.0, 0.0), grid_dim=(edge,) * 3, grid_spacing=h, young=young, hardening=hardening,
                     dt=case["dt"], steps=case["steps"], colliders=coll, implicit_beta=float(case.get("beta", 0.0)), **CRIT)
    m = torch.full((n,), scenes.SNOW_DENSITY * h ** 3 / 8.0, device=DEV)
    s.x, s.v, s.m = _host(x), _host(v), _host(m)
    return s


def _single(case, seed):
    """(scene, FE, FP) of a one-scene case."""
    g = _gen(seed)
    x, v, coll = _shape(case, g)
    fe = fp = None
    if case["warm"]:
        fe, fp = (_host(t) for t in _deformation(x, g))
        v = v + 0.05 * torch.sin(x.flip(1) * 40.0)
    stiff = case["shape"] == "jitter"
    return _scene(case, x, v, coll, 1.4e7 if stiff else 1.4e5, 10.0), fe, fp


def _many(case, seed):
    """The scenes of a batch or the jobs of a server: sizes and materials are
    the case's own (the same for every seed), shapes and motion the seed's."""
    rs = np.random.RandomState(12345 + case["scenes"])
    out = []
    for i in range(case["scenes"]):
        n = int(round(math.exp(rs.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        kind = "sphere" if rs.rand() < 0.5 else "box"
        r = (3.0 * n / 8.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
        edge = min(192, max(64, int(math.ceil(5.0 * r / 32) * 32)))
        young, hard = float(rs.uniform(4.8e4, 1.4e5)), float(rs.uniform(5.0, 10.0))
        steps = case["steps"] if "steps" in case else int(rs.randint(case["steps_min"], case["steps_max"] + 1))
        g = _gen(seed * 1009 + i)
        h = 1.0 / edge
        x = _fill(kind, [0.5 + t for t in _uniform(g, -0.05, 0.05, 3)], n, h, g)
        d = torch.randn(3, generator=g, device=DEV)
        v = (d / d.norm() * _uniform(g, 0.5, 4.0)[0]).repeat(n, 1)
        out.append(_scene(dict(edge=edge, dt=case["dt"], steps=steps), x, v, _walls(edge), young, hard))
    return out


def _outputs(n):
    """Preallocated pinned arrays of the particle state."""
    def a(*shape):
        return torch.empty(shape, dtype=torch.float32, pin_memory=DEV != "cpu").numpy()
    return dict(x=a(n, 3), v=a(n, 3), FE=a(n, 3, 3), Jp=a(n), volume=a(n))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = _gen(seed)
        top = (1 << case["bits"]) - 1
        keys = torch.randint(0, top + 1, (case["n"],), generator=g, device=DEV, dtype=torch.int64)
        # cell keys come in runs: several particles of a cell, cells near each other
        keys = (keys // 64 * 64 + torch.arange(case["n"], device=DEV) % 64) & top
        keys = torch.where(keys > 0x7FFFFFFF, keys - (1 << 32), keys).to(torch.int32)
        return dict(kind=kind, n=case["n"], bits=case["bits"], keys=keys, out=torch.empty_like(keys),
                    perm=torch.empty_like(keys), L=N.load())
    if kind == "serve":
        jobs = _many(case, seed)
        return dict(kind=kind, jobs=jobs, srv=api.Server(hbm_budget=64 << 30), n=[s.n for s in jobs])
    if kind == "batch":
        sc = _many(case, seed)
        ctx = api.Context(0)
        sims = [api.SimScene(ctx, s).upload().init() for s in sc]
        out = _outputs(sum(s.n for s in sc))
        at = np.cumsum([0] + [s.n for s in sc])
        parts = [{k: a[at[i]:at[i + 1]] for k, a in out.items()} for i in range(len(sc))]
        return dict(kind=kind, ctx=ctx, sims=sims, batch=api.Batch(ctx, sims), parts=parts, out=out, steps=case["steps"],
                    dts=[s.dt for s in sc])
    s, fe, fp = _single(case, seed)
    ctx = api.Context(0)
    if kind == "reference":
        return dict(kind=kind, sim=api.SimScene(ctx, s, mode=N.MODE_REFERENCE), bufs=s.std140(), dt=s.dt,
                    steps=case["steps"], ctx=ctx)
    sim = api.SimScene(ctx, s).upload(FE=fe, FP=fp).init()
    return dict(kind=kind, ctx=ctx, sim=sim, fe=fe, fp=fp, out=_outputs(s.n), dt=s.dt, steps=case["steps"])


# ---- one pass -------------------------------------------------------------------
def _stats_row(d):
    return np.concatenate([[d["mass"], d["kinetic_energy"], d["mean_jp"]], d["momentum"], d["center_of_mass"],
                           d["bbox_min"], d["bbox_max"]]).astype(np.float32)


def run(st):
    kind = st["kind"]
    if kind == "sort":
        rc = st["L"].snow_sort_keys_static(st["keys"].data_ptr(), st["out"].data_ptr(), st["perm"].data_ptr(), st["n"],
                                           st["bits"], C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != N.SNOW_OK:
            raise RuntimeError(f"snow_sort_keys_static: {rc}")
        return st["out"], st["perm"]
    if kind == "live":
        return st["sim"].step(st["dt"], st["steps"]).download(out=st["out"])
    if kind == "reference":
        return st["sim"].upload_std140(*st["bufs"]).init().step(st["dt"], st["steps"]).download_std140()
    if kind == "serve":
        srv = st["srv"]
        ids = [srv.submit(s, keep_state=True) for s in st["jobs"]]
        srv.drain()
        for r in srv.poll():
            if r["status"] != N.SNOW_OK:
                raise RuntimeError(f"job {r['id']}: {r['status']}")
        got = [srv.fetch(i, n) for i, n in zip(ids, st["n"])]
        return {k: np.concatenate([r[k] for r in got]) for k in ("x", "v", "FE", "Jp")}
    if kind == "batch":
        for sim in st["sims"]:
            sim.dispatch(N.K_G_RESET)
            sim.upload().init()
        st["batch"].step(st["steps"], st["dts"])
        for sim, part in zip(st["sims"], st["parts"]):
            sim.download(out=part)
        return st["out"]
    sim, dt = st["sim"], st["dt"]
    sim.dispatch(N.K_G_RESET)
    sim.upload(FE=st["fe"], FP=st["fp"]).init()
    if kind == "scene":
        return sim.step(dt, st["steps"]).download(out=st["out"])
    rows = []
    for i in range(st["steps"]):  # step i's statistics are read while step i + 1 runs
        sim.step(dt, 1).stats_enqueue(i % 2)
        if i:
            rows.append(_stats_row(st["ctx"].stats_read((i - 1) % 2)))
    rows.append(_stats_row(st["ctx"].stats_read((st["steps"] - 1) % 2)))
    return dict(sim.download(out=st["out"]), stats=np.stack(rows))


# ---- what a pass cannot do without ------------------------------------------------
# Per particle and step: position, mass, velocity, volume, F_E and J_p read and
# written once. Operations: about 4,200 per particle and step (64 stencil nodes
# gathered and scattered, one eigen-solve); those of the semi-implicit
# iterations, whose number depends on the state, are not counted.
_STATE, _FLOPS = 72, 4200


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return dict(bytes=16.0 * case["n"], flops=0.0)  # keys read; keys and permutation written
    if kind in ("batch", "serve"):
        rs = np.random.RandomState(12345 + case["scenes"])
        tot = steps = 0.0
        for _ in range(case["scenes"]):
            n = int(round(math.exp(rs.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
            rs.rand(), rs.uniform(), rs.uniform()
            k = case["steps"] if "steps" in case else int(rs.randint(case["steps_min"], case["steps_max"] + 1))
            tot += n
            steps += n * k
        return dict(bytes=2.0 * _STATE * steps + (28.0 + 68.0) * tot, flops=_FLOPS * steps)
    n, k = case["n"], case["steps"]
    io = 68.0 * n  # the state downloaded
    if kind != "live":
        io += (100.0 if case["warm"] else 28.0) * n  # and uploaded
    return dict(bytes=2.0 * _STATE * n * k + io, flops=float(_FLOPS) * n * k)


# ---- the same in 64 bits ----------------------------------------------------------
def _f32(v):
    return float(np.float32(v))


def _eig(s):
    """Cyclic Jacobi on symmetric 3x3 matrices given as six vectors
    (00, 11, 22, 01, 02, 12): eigenvalues and the columns of V."""
    a = [[s[0], s[3], s[4]], [s[3], s[1], s[5]], [s[4], s[5], s[2]]]
    one, zero = torch.ones_like(s[0]), torch.zeros_like(s[0])
    V = [[one if r == c else zero for c in range(3)] for r in range(3)]
    for _ in range(6):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq = a[p][q]
            tiny = apq.abs() < 1e-300
            th = (a[q][q] - a[p][p]) / (2 * torch.where(tiny, one, apq))
            t = torch.where(th >= 0, 1.0, -1.0) / (th.abs() + torch.sqrt(th * th + 1))
            t = torch.where(tiny, zero, t)
            c = 1 / torch.sqrt(t * t + 1)
            sn = t * c
            a[p][p], a[q][q] = a[p][p] - t * apq, a[q][q] + t * apq
            a[p][q] = a[q][p] = zero
            arp, arq = a[r][p], a[r][q]
            a[r][p] = a[p][r] = c * arp - sn * arq
            a[r][q] = a[q][r] = sn * arp + c * arq
            for k in range(3):
                V[k][p], V[k][q] = c * V[k][p] - sn * V[k][q], sn * V[k][p] + c * V[k][q]
    return [a[0][0], a[1][1], a[2][2]], V


def _spd(F):
    """sigma (N x 3) and V (N x 3 x 3) of F = W diag(sigma) V^T."""
    S = F.transpose(1, 2) @ F
    lam, V = _eig([S[:, 0, 0], S[:, 1, 1], S[:, 2, 2], S[:, 0, 1], S[:, 0, 2], S[:, 1, 2]])
    return torch.stack(lam, 1).clamp_min(1e-300).sqrt(), torch.stack([torch.stack(r, 1) for r in V], 1)


def _det(F):
    return (F[:, 0] * torch.cross(F[:, 1], F[:, 2], dim=1)).sum(1)


def _weights(xg):
    """Base cells and, per axis, the spline's values and derivatives at the
    four stencil nodes base - 1 .. base + 2 (particles lie inside the grid)."""
    base = xg.floor()
    f = xg - base
    u = 1 - f
    w = torch.stack([u ** 3 / 6, 0.5 * f ** 3 - f ** 2 + 2 / 3, 0.5 * u ** 3 - u ** 2 + 2 / 3, f ** 3 / 6], 2)
    d = torch.stack([-0.5 * u ** 2, 1.5 * f ** 2 - 2 * f, -1.5 * u ** 2 + 2 * u, 0.5 * f ** 2], 2)
    return base.long(), w, d


def _collide(x, v, sc, C_):
    """The colliders of scene sc (per row) on points x with velocities v, in
    order: the inward normal part goes, with Coulomb friction."""
    for k in range(C_["type"].shape[1]):
        ty, pos, vel = C_["type"][sc, k], C_["pos"][sc, k], C_["vel"][sc, k]
        nrm, rad, mu = C_["normal"][sc, k], C_["radius"][sc, k], C_["friction"][sc, k]
        d = x - pos
        dist = d.norm(dim=1)
        hit = torch.where(ty == 0, (d * nrm).sum(1) <= 0, (ty == 1) & (dist < rad))
        nn = torch.where((ty == 1)[:, None], d / dist.clamp_min(1e-300)[:, None], nrm)
        rel = v - vel
        vn = (rel * nn).sum(1)
        vt = rel - nn * vn[:, None]
        lt = vt.norm(dim=1)
        stick = lt <= -mu * vn
        slide = vt + (mu * vn / lt.clamp_min(1e-300))[:, None] * vt + vel
        new = torch.where(stick[:, None], vel, slide)
        v = torch.where((hit & (vn < 0))[:, None], new, v)
    return v


class _Exact:
    """Explicit steps of several scenes side by side in 64 bits."""
    CHUNK = 1 << 20

    def __init__(self, scs, fes, fps):
        t64 = lambda a: torch.as_tensor(np.asarray(a), device=DEV, dtype=torch.float64)  # noqa: E731
        self.scs = scs
        self.sc = torch.cat([torch.full((s.n,), i, device=DEV) for i, s in enumerate(scs)])
        self.x, self.v = (torch.cat([t64(getattr(s, k)) for s in scs]) for k in ("x", "v"))
        self.m = torch.cat([t64(s.m) for s in scs])
        eye = lambda n: torch.eye(3, device=DEV, dtype=torch.float64).repeat(n, 1, 1)  # noqa: E731
        self.F = torch.cat([eye(s.n) if f is None else t64(f).reshape(-1, 3, 3) for s, f in zip(scs, fes)])
        self.jp = torch.cat([_det(eye(s.n) if f is None else t64(f).reshape(-1, 3, 3)) for s, f in zip(scs, fps)])
        per = lambda f: torch.tensor([_f32(f(s)) for s in scs], device=DEV, dtype=torch.float64)  # noqa: E731
        nu = per(lambda s: s.poisson)
        E = per(lambda s: s.young)
        self.mu, self.la = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        self.h, self.xi, self.alpha = per(lambda s: s.grid_spacing), per(lambda s: s.hardening), per(lambda s: s.alpha)
        self.lo, self.hi = 1 - per(lambda s: s.crit_compression), 1 + per(lambda s: s.crit_stretch)
        self.dt = per(lambda s: s.dt)
        self.g = torch.tensor([[_f32(c) for c in s.gravity] for s in scs], device=DEV, dtype=torch.float64)
        self.edge = torch.tensor([s.grid_dim[0] for s in scs], device=DEV)
        self.at = torch.tensor(np.cumsum([0] + [s.grid_dim[0] ** 3 for s in scs]), device=DEV)
        nc = max(len(s.colliders) for s in scs)
        pad = [list(s.colliders) + [scenes.Collider(pos=(0.0, 0.0, 0.0), type=-1)] * (nc - len(s.colliders)) for s in scs]
        col = lambda f: torch.tensor([[f(c) for c in row] for row in pad], device=DEV, dtype=torch.float64)  # noqa: E731
        vec = lambda k: col(lambda c: [_f32(t) for t in getattr(c, k)])  # noqa: E731
        self.C = dict(type=col(lambda c: float(c.type)), pos=vec("pos"), vel=vec("vel"), normal=vec("normal"),
                      radius=col(lambda c: _f32(c.radius)), friction=col(lambda c: _f32(c.friction)))
        self.live = torch.arange(len(self.x), device=DEV)
        G = int(self.at[-1])
        mass = torch.zeros(G, device=DEV, dtype=torch.float64)
        for i in self._chunks():
            base, w, _ = self._stencil(i)
            for node, ww, _ in self._nodes(i, base, w, None):
                mass.index_add_(0, node, self.m[i] * ww)
        self.V0 = torch.zeros_like(self.m)
        for i in self._chunks():
            base, w, _ = self._stencil(i)
            rho = torch.zeros(len(i), device=DEV, dtype=torch.float64)
            for node, ww, _ in self._nodes(i, base, w, None):
                rho += mass[node] * ww
            self.V0[i] = self.m[i] * self.h[self.sc[i]] ** 3 / rho

    def _chunks(self):
        return torch.split(self.live, self.CHUNK)

    def _stencil(self, i):
        return _weights(self.x[i] / self.h[self.sc[i]][:, None])

    def _nodes(self, i, base, w, d):
        """(flat node, weight, weight gradient) of the 64 stencil nodes."""
        e, at = self.edge[self.sc[i]], self.at[self.sc[i]]
        for c in range(4):
            for b in range(4):
                wyz = w[:, 1, b] * w[:, 2, c]
                row = at + (base[:, 0] - 1) + e * ((base[:, 1] - 1 + b) + e * (base[:, 2] - 1 + c))
                if d is not None:
                    gy, gz = d[:, 1, b] * w[:, 2, c], w[:, 1, b] * d[:, 2, c]
                for a in range(4):
                    ww = w[:, 0, a] * wyz
                    yield row + a, ww, None if d is None else torch.stack(
                        [d[:, 0, a] * wyz, w[:, 0, a] * gy, w[:, 0, a] * gz], 1)

    def step(self):
        self.C["pos"] = self.C["pos"] + self.C["vel"] * self.dt[:, None, None]
        G = int(self.at[-1])
        acc = torch.zeros(G, 7, device=DEV, dtype=torch.float64)
        for i in self._chunks():
            s, F = self.sc[i], self.F[i]
            sig, V = _spd(F)
            R = F @ (V / sig[:, None, :]) @ V.transpose(1, 2)
            hard = torch.exp(self.xi[s] * (1 - self.jp[i]))
            J = _det(F)
            A = 2 * (self.mu[s] * hard)[:, None, None] * ((F - R) @ F.transpose(1, 2))
            A = A + (self.la[s] * hard * (J - 1) * J)[:, None, None] * torch.eye(3, device=DEV, dtype=torch.float64)
            A = -self.V0[i][:, None, None] * A
            q = torch.cat([self.m[i][:, None], self.m[i][:, None] * self.v[i]], 1)
            base, w, d = self._stencil(i)
            for node, ww, gw in self._nodes(i, base, w, d):
                acc.index_add_(0, node, torch.cat([q * ww[:, None], (A @ gw[:, :, None])[:, :, 0]], 1))
        node = torch.nonzero(acc[:, 0] > 0)[:, 0]
        a = acc[node]
        s = torch.searchsorted(self.at, node, right=True) - 1
        loc, e = node - self.at[s], self.edge[s]
        xi = torch.stack([loc % e, loc // e % e, loc // (e * e)], 1) * self.h[s][:, None]
        old = a[:, 1:4] / a[:, :1]
        vs = old + self.dt[s][:, None] * (a[:, 4:] / a[:, :1] + self.g[s])
        vs = _collide(xi, vs, s, self.C)
        grid = torch.zeros(G, 6, device=DEV, dtype=torch.float64) if len(self.x) < self.CHUNK * 12 else acc[:, :6].zero_()
        grid[node] = torch.cat([vs, vs - self.alpha[s][:, None] * old], 1)
        for i in self._chunks():
            s = self.sc[i]
            base, w, d = self._stencil(i)
            dv = torch.zeros(len(i), 3, device=DEV, dtype=torch.float64)
            L = torch.zeros(len(i), 3, 3, device=DEV, dtype=torch.float64)
            for node, ww, gw in self._nodes(i, base, w, d):
                n6 = grid[node]
                dv += ww[:, None] * n6[:, 3:]
                L += n6[:, :3, None] * gw[:, None, :]
            dt = self.dt[s]
            F = self.F[i] + dt[:, None, None] * (L @ self.F[i])
            sig, V = _spd(F)
            cl = torch.minimum(torch.maximum(sig, self.lo[s][:, None]), self.hi[s][:, None])
            self.F[i] = F @ (V * (cl / sig)[:, None, :]) @ V.transpose(1, 2)
            self.jp[i] = self.jp[i] * (sig / cl).prod(1)
            v = self.alpha[s][:, None] * self.v[i] + dv
            v = _collide(self.x[i], v, s, self.C)
            self.v[i] = v
            self.x[i] = self.x[i] + dt[:, None] * v

    def stats(self):
        m, x, v = self.m, self.x, self.v
        return torch.cat([torch.stack([m.sum(), 0.5 * (m * v.square().sum(1)).sum(), self.jp.mean()]), (m[:, None] * v).sum(0),
                          (m[:, None] * x).sum(0) / m.sum(), x.amin(0), x.amax(0)])

    def state(self):
        return dict(x=self.x, v=self.v, FE=self.F, Jp=self.jp, volume=self.V0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":  # whole numbers: a stable sort of the keys as unsigned numbers
        keys = prepare(case, seed)["keys"].cpu().numpy().view(np.uint32)
        perm = np.argsort(keys, kind="stable")
        return keys[perm].view(np.int32), perm.astype(np.int32)
    if kind == "reference" or case.get("beta"):
        # fixed-point sums that truncate; a solve that stops at its tolerance:
        # neither has a value to more digits than the arithmetic that is asked for
        return None
    if kind in ("batch", "serve"):
        scs = _many(case, seed)
        fes = fps = [None] * len(scs)
    else:
        s, fe, fp = _single(case, seed)
        scs, fes, fps = [s], [fe], [fp]
    ex = _Exact(scs, fes, fps)
    steps = torch.tensor([s.steps for s in scs], device=DEV)
    rows = []
    for k in range(int(steps.max())):
        ex.live = torch.nonzero(steps[ex.sc] > k)[:, 0]
        ex.step()
        if kind == "monitor":
            rows.append(ex.stats())
    out = ex.state()
    if kind == "serve":
        del out["volume"]
    if kind == "monitor":
        out["stats"] = torch.stack(rows)
    return out
