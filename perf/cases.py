"""Performance cases of the DEM step, through the calls a user's program makes.

Every sphere and lattice case is the DEM command (Model.dem) on a model whose
session is in hand, the way a deck runs it; the serving case is Server.serve.
The scenes are those of parmec_gb300.scenes, made from the seed: the hopper
fill, the rotating drum, the shaken boxes of the batch, the spring lattice on
its shaking table (with and without contact between its cubes) and the stream
of excitation-sweep requests.  A pass runs `steps` time steps from where the
state stands and brings the state back to the model's host arrays, as DEM
does; the first pass on a state starts with the reference's half step.

listed() and draw() give the cases, prepare() the state of one, run() a pass,
work() what a pass cannot do without, and exact() the outputs of the first
pass in plain 64-bit torch arithmetic (an independent, vectorised DEM).
"""
import math

import numpy as np
import torch

from parmec_gb300 import abi, batch, scenes, serving
from parmec_gb300.engine import GpuEngine

# contact pairs per sphere of the dense scenes, for work()
PAIRS_PER_SPHERE = 0.93


def listed():
    return [
        # the smallest deck a user runs, and the smallest of a parameter
        # study: launches and latency are all of it
        {"name": "hopper_216", "kind": "hopper", "side": 6, "steps": 300},
        # the CPU-runnable hopper fill of the benchmark, plain FP64
        {"name": "hopper_4096", "kind": "hopper", "side": 16, "steps": 300},
        # the same deck at the scale of boulders, the time step chosen by
        # DEM(adaptive=...): the host reads every step back
        {"name": "hopper_adaptive", "kind": "hopper", "side": 13, "steps": 60, "adaptive": 0.1},
        # the rotating drum, plain FP64: the headline workload at its full size
        {"name": "drum_fp64", "kind": "drum", "spheres": 1048576, "form": "fp64", "steps": 30},
        # the drum in the mixed form, at a ragged size
        {"name": "drum_mixed", "kind": "drum", "spheres": 300007, "form": "mixed", "steps": 60},
        # uneven shaken boxes stepped together, both forms (the batch workload)
        {"name": "batch_mixed", "kind": "batch", "scenes": 64, "form": "mixed", "steps": 40},
        {"name": "batch_fp64", "kind": "batch", "scenes": 12, "form": "fp64", "steps": 40},
        # the spring lattice on its shaking table, springs only
        {"name": "lattice_springs", "kind": "lattice", "side": 96, "contact": False, "steps": 60},
        # the same with contact between the cubes, a small and a larger one
        {"name": "lattice_contact_16", "kind": "lattice", "side": 16, "contact": True, "steps": 12},
        {"name": "lattice_contact_64", "kind": "lattice", "side": 64, "contact": True, "steps": 6},
        # a stream of requests of different sizes and lengths through one pool
        {"name": "serve_mixed", "kind": "serve", "requests": 10, "form": "mixed", "spheres": 16384, "steps": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hopper", "hopper", "adaptive", "drum", "drum", "batch", "lattice", "contact", "serve"])
    if kind == "hopper":
        return {"kind": "hopper", "side": rng.randint(3, 32), "steps": rng.randint(100, 300)}
    if kind == "adaptive":
        return {"kind": "hopper", "side": rng.randint(3, 20), "steps": rng.randint(20, 60),
                "adaptive": rng.choice([0.05, 0.1, 0.2])}
    if kind == "drum":
        return {"kind": "drum", "spheres": _log(rng, 5000, 1000000), "form": rng.choice(["fp64", "mixed"]),
                "steps": rng.randint(10, 30)}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 48), "form": rng.choice(["fp64", "mixed"]),
                "steps": rng.randint(20, 40)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(3, 10), "form": rng.choice(["fp64", "mixed"]),
                "spheres": _log(rng, 2048, 16384), "steps": rng.randint(100, 400)}
    contact = kind == "contact"
    return {"kind": "lattice", "side": _log(rng, 4, 64 if contact else 96), "contact": contact,
            "steps": rng.randint(2, 6) if contact else rng.randint(20, 60)}


# ---------------------------------------------------------------- scenes

def _form(case):
    return abi.PG_FORM_MIXED if case.get("form") == "mixed" else abi.PG_FORM_FP64


def _hopper(case, seed):
    # a lattice dense enough to hold contacts from the start, its outer
    # spheres reaching the walls; with a chosen time step at 100 times the
    # size (the rotational damping ratio of the step estimate grows as 1/r^2
    # and cuts the step of centimetre spheres 10,000 times)
    side, k = case["side"], 100.0 if case.get("adaptive") else 1.0
    return scenes.hopper_fill(side, seed=seed, spacing=k * 0.036, jitter=k * 0.005, rmin=k * 0.01, rmax=k * 0.02,
                              kn=1e9 if case.get("adaptive") else 1e6, box=k * ((side - 1) * 0.036 + 0.04))


def _sizes(count, lo, hi):
    """Sphere counts of a batch or a stream, log-uniform and fixed by the
    case: lattice sides of the scenes."""
    n = scenes.log_uniform(np.random.default_rng(count), lo, hi, count)
    return [max(2, int(round(float(k) ** (1.0 / 3.0)))) for k in n]


def _boxes(case, seed):
    """The batch's shaken boxes: (model, dt, excitation) each."""
    rng = np.random.default_rng(seed)
    return [scenes.shaken_box(side ** 3, seed * 100003 + k, float(rng.uniform(1.0, 20.0)), float(rng.uniform(0.1, 1.0)))
            for k, side in enumerate(_sizes(case["scenes"], 2048, 65536))]


def _requests(case, seed):
    """The stream: half the requests shaken by a sinusoid, half by band noise,
    each for its own number of steps."""
    rng = np.random.default_rng(seed)
    out = []
    for k, side in enumerate(_sizes(case["requests"], 512, case["spheres"])):
        m, dt = scenes.hopper_fill(n_side=side, seed=seed * 1000003 + k, box=max(1.0, side / 16.0))
        a, g0 = rng.uniform(0.1, 1.0) * 9.81, (0.0, 0.0, -9.81)
        if k % 2 == 0:
            exc = batch.sinusoid(g0, (a, 0.0, 0.0), rng.uniform(1.0, 20.0))
        else:
            exc = batch.band_noise(g0, (1.0, 0.0, 0.0), a, 1.0, 20.0, seed=int(rng.integers(1 << 30)))
        out.append(serving.Request(k, 0.0, m, _request_steps(case, k), exc, dt))
    return out


def _request_steps(case, k):
    return case["steps"] * (8 - 3 * k % 5) // 8


def _pool_room(requests):
    """Spheres and scene slots of the pool: fewer than the whole stream, so
    that requests wait for others to finish."""
    sizes = [q.model.parnum for q in requests]
    return max(max(sizes), (6 * sum(sizes)) // 10), max(2, (2 * len(sizes)) // 3)


def prepare(case, seed):
    if case["kind"] == "serve":
        requests = _requests(case, seed)
        room, slots = _pool_room(requests)
        srv = serving.Server(requests[0].model, requests[0].dt, form=_form(case), max_scenes=slots,
                             max_spheres=room, max_scene_extent=4.0)
        return {"server": srv, "requests": requests}
    excitations = None
    engine = GpuEngine(form=_form(case))
    if case["kind"] == "hopper":
        model, dt = _hopper(case, seed)
    elif case["kind"] == "drum":
        model, dt, _ = scenes.drum(case["spheres"], seed=seed)
    elif case["kind"] == "batch":
        made = _boxes(case, seed)
        model, _ = batch.pool([m for m, _, _ in made])
        dt, excitations = made[0][1], [e for _, _, e in made]
    else:
        model, dt = scenes.spring_lattice(case["side"], seed=seed, contact_radius=1e-3 if case["contact"] else 0.0)
    if model.springs_changed:                     # DEM's own order of the springs, before the session sees them
        from parmec_gb300.springs import sort_springs
        sort_springs(model)
        model.springs_changed = False
    model.sort_materials()
    engine.attach(model)
    if excitations is not None:
        for k, e in enumerate(excitations):
            engine.set_scene(k, True, excitation=e, start=0)
    model.engine = engine
    model._dirty = False
    return {"model": model, "dt": dt, "steps": case["steps"], "adaptive": case.get("adaptive", 0.0)}


def run(state):
    if "server" in state:
        results, _ = state["server"].serve(state["requests"], realtime=False)
        results.sort(key=lambda r: r.rid)
        return {"position": np.concatenate([r.position for r in results], axis=1),
                "linear": np.concatenate([r.linear for r in results], axis=1),
                "energy": np.array([r.energy for r in results])}
    m, dt = state["model"], state["dt"]
    m.dem(state["steps"] * dt - 0.5 * dt, dt, interval=1e9, adaptive=state["adaptive"])
    n = m.parnum
    out = {"position": m.P.position[0:3, :n], "linear": m.P.linear[:, :n], "angular": m.P.angular[:, :n],
           "rotation": m.P.rotation[:, :n], "force": m.P.force[:, :n], "torque": m.P.torque[:, :n]}
    if m.sprnum:
        # in the SPRING commands' order
        at = m.S.sprmap[:m.sprnum]
        out["spring_force"] = m.S.sprfrc[0][at]
        out["stroke"] = m.S.stroke[0][at]
    if state["adaptive"]:
        out["time"] = float(m.curtime)
    return out


# ---------------------------------------------------------------- work

def _particle_steps(case):
    """(particles x steps, particles) of a pass."""
    if case["kind"] == "hopper":
        n = case["side"] ** 3
    elif case["kind"] == "drum":
        n = case["spheres"]
    elif case["kind"] == "batch":
        n = sum(side ** 3 for side in _sizes(case["scenes"], 2048, 65536))
    elif case["kind"] == "serve":
        sides = _sizes(case["requests"], 512, case["spheres"])
        return (sum(side ** 3 * _request_steps(case, k) for k, side in enumerate(sides)),
                sum(side ** 3 for side in sides))
    else:
        n = case["side"] ** 2 + 1
    return n * case["steps"], n


def work(case):
    ps, n = _particle_steps(case)
    if case["kind"] == "lattice":
        springs = 3.0 * case["side"] ** 2 * case["steps"]
        nodes = 8.0 * ps
        # particle state read and written and constants; a spring's points,
        # curve, dashpot, stroke and forces; a node's reference point read and
        # its place written; a triangle's vertices
        size = ps * (336 + 172) + springs * (96 + 128 + 32 + 24 + 72) + nodes * 48 + 12.0 * ps * 72
        flops = ps * 330 + springs * 180 + nodes * 21
        if case["contact"]:
            # of the pairs of a packed lattice (16 a triangle) the box and
            # plane tests, and the closest points of one feature pair
            pairs = 16.0 * 12.0 * ps
            size += pairs * (4 + 4)
            flops += pairs * (60 + 120)
        return {"bytes": size + n * 360, "flops": flops}
    c = PAIRS_PER_SPHERE if case["kind"] in ("drum", "hopper") else 0.4
    per = (312 + 28 * c) if case.get("form") == "mixed" else (420 + 56 * c)
    return {"bytes": ps * per + n * 360, "flops": ps * (280 + 130 * c)}


# ---------------------------------------------------------------- the same in plain 64-bit torch

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_device())


def _expmap(o):
    """Rotation matrices (n, 3, 3) of rotation vectors (n, 3), with the
    reference's product O2*O3 in the place of O1*O3 in the second-order term."""
    a2 = (o * o).sum(1)
    a = a2.sqrt()
    small = a2 < 1e-8
    safe = torch.where(small, torch.ones_like(a), a)
    s = torch.where(small, 1 - a2 / 6 + a2 * a2 / 120, torch.sin(safe) / safe)
    c = torch.where(small, 0.5 - a2 / 24 + a2 * a2 / 720, (1 - torch.cos(safe)) / (safe * safe))
    x, y, z = o.unbind(1)
    xy, xz, yz = c * x * y, c * y * z, c * y * z          # xz: the reference's O2*O3
    rows = [1 - c * (z * z + y * y), xy - s * z, xz + s * y,
            xy + s * z, 1 - c * (z * z + x * x), yz - s * x,
            xz - s * y, yz + s * x, 1 - c * (y * y + x * x)]
    return torch.stack(rows, 1).reshape(-1, 3, 3)


def _mv(m, v):
    return (m * v[:, None, :]).sum(2)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


class _Bodies:
    """Particle state and the reference's integration, 64-bit torch."""

    def __init__(self, m):
        P, n = m.P, m.parnum
        self.n = n
        self.x, self.X = _t(P.position[0:3, :n].T), _t(P.position[3:6, :n].T)
        self.v, self.O, self.o = _t(P.linear[:, :n].T), _t(P.angular[0:3, :n].T), _t(P.angular[3:6, :n].T)
        self.L = _t(P.rotation[:, :n].T).reshape(n, 3, 3).transpose(1, 2).contiguous()
        self.J = _t(P.inertia[:, :n].T).reshape(n, 3, 3).transpose(1, 2).contiguous()
        self.I = torch.linalg.inv(self.J)
        self.m = _t(P.mass[:n])
        self.im = 1.0 / self.m
        self.F, self.T = torch.zeros_like(self.x), torch.zeros_like(self.x)

    def half_step(self, h):
        w = 0.5 * h * self.O
        self.L = torch.bmm(self.L, _expmap(w))
        self.o = _mv(self.L, w)
        self.x = self.x + 0.5 * h * self.v

    def advance(self, F, T, h):
        self.F, self.T = F, T
        Tb = _mv(self.L.transpose(1, 2), T)
        B = _mv(_expmap(-0.5 * h * self.O), _mv(self.J, self.O)) + 0.5 * h * Tb
        A = _mv(self.I, B)
        Tb = h * (Tb - _cross(A, _mv(self.J, A)))
        self.O = self.O + _mv(self.I, Tb)
        self.v = self.v + h * self.im[:, None] * F
        self.L = torch.bmm(self.L, _expmap(h * self.O))
        self.o = _mv(self.L, self.O)
        self.x = self.x + h * self.v

    def outputs(self):
        col = lambda a: a.T.contiguous().cpu().numpy()  # noqa: E731
        return {"position": col(self.x), "linear": col(self.v), "angular": col(torch.cat([self.O, self.o], 1)),
                "rotation": col(self.L.transpose(1, 2).reshape(self.n, 9)), "force": col(self.F), "torque": col(self.T)}


def _closest(p, A, B, C):
    """Closest points of triangles (A, B, C) to points p by the regions of the
    (s, t) plane, with the reference's -e/c beyond edge bc where t < 0."""
    e0, e1, v = B - A, C - A, A - p
    dot = lambda q, r: (q * r).sum(1)  # noqa: E731
    a, b, c, d, e = dot(e0, e0), dot(e0, e1), dot(e1, e1), dot(e0, v), dot(e1, v)
    det, s, t = a * c - b * b, b * e - c * d, b * d - a * e
    clamp = lambda q: q.clamp(0.0, 1.0)  # noqa: E731
    sd, te = clamp(-d / a), clamp(-e / c)
    hyp = (c + e - b - d) / (a - 2 * b + c)
    zero = torch.zeros_like(s)
    inside, sn, tn = s + t < det, s < 0, t < 0
    # s + t < det
    s_in = torch.where(sn, torch.where(tn & (d < 0), sd, zero), torch.where(tn, sd, s / det))
    t_in = torch.where(sn, torch.where(tn & (d < 0), zero, te), torch.where(tn, zero, t / det))
    # beyond edge bc
    up, right = (c + e) > (b + d), (a + d) > (b + e)
    h = clamp(hyp)
    s_out = torch.where(sn, torch.where(up, h, zero), torch.where(tn, torch.where(right, h, te), hyp))
    t_out = torch.where(sn, torch.where(up, 1 - h, te), torch.where(tn, torch.where(right, 1 - h, zero), 1 - hyp))
    s, t = torch.where(inside, s_in, s_out), torch.where(inside, t_in, t_out)
    return A + s[:, None] * e0 + t[:, None] * e1


def _sphere_pairs(x, r, scene, skin):
    """Index pairs i < j of spheres of one scene closer than r_i + r_j + skin."""
    cell = float(2 * r.max() + skin)
    lo = x.min(0).values
    u = ((x - lo) / cell).floor().long() + 1
    dim = u.max(0).values + 2
    key = ((scene * dim[2] + u[:, 2]) * dim[1] + u[:, 1]) * dim[0] + u[:, 0]
    order = torch.argsort(key)
    sk = key[order]
    out_i, out_j = [], []
    ids = torch.arange(len(x), device=x.device)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            k = key + (dz * dim[1] + dy) * dim[0]
            # a row of three cells is one range of sorted keys
            b, e = torch.searchsorted(sk, k - 1), torch.searchsorted(sk, k + 1, right=True)
            width = int((e - b).max())
            for w in range(width):
                ok = b + w < e
                i = ids[ok]
                j = order[(b + w)[ok]]
                keep = (i < j) & (scene[i] == scene[j])
                i, j = i[keep], j[keep]
                q = x[i] - x[j]
                near = (q * q).sum(1) < (r[i] + r[j] + skin) ** 2
                out_i.append(i[near])
                out_j.append(j[near])
    i, j = torch.cat(out_i), torch.cat(out_j)
    at = torch.argsort(i * len(x) + j)
    return i[at], j[at]


def _wall_pairs(x, r, scene, tri, tscene, skin):
    """Sphere-triangle index pairs whose boxes come within the skin."""
    lo, hi = tri.min(1).values, tri.max(1).values                       # (T, 3)
    # the spheres near the outside of some triangle's box, in chunks of triangles
    out_i, out_t = [], []
    reach = (r + skin)[:, None]
    # spheres well inside every scene's walls meet none: tested against 64
    # triangles at a time
    for t0 in range(0, len(tri), 64):
        l, h, ts = lo[t0:t0 + 64], hi[t0:t0 + 64], tscene[t0:t0 + 64]
        cl, ch = l.min(0).values, h.max(0).values
        some = ((x + reach >= cl) & (x - reach <= ch)).all(1).nonzero()[:, 0]
        for s0 in range(0, len(some), 1 << 18):
            i = some[s0:s0 + (1 << 18)]
            near = ((x[i, None, :] + reach[i, None] >= l[None]) & (x[i, None, :] - reach[i, None] <= h[None])).all(2)
            near &= scene[i][:, None] == ts[None]
            a, b = near.nonzero(as_tuple=True)
            out_i.append(i[a])
            out_t.append(b + t0)
    return torch.cat(out_i), torch.cat(out_t)


class _Granular:
    """Sphere-sphere and sphere-triangle contacts with the granular law."""

    def __init__(self, m, pscene=None, tscene=None):
        n, nt = m.parnum, m.trinum
        self.r = _t(m.E.radii[0, :n])
        self.tri = _t(m.Tr.tri[:, :nt].T).reshape(nt, 3, 3)
        self.moving = _t(m.Tr.triobs[:nt] <= -2, torch.bool)
        self.point = _t(m.O.obspnt[:, 0]) if m.obsnum else torch.zeros(3, dtype=torch.float64, device=_device())
        self.omega = None                        # angular velocity of the one moving obstacle
        ip = m.iparam[0]
        self.kn, self.damper, self.mus, self.mud, self.kskn = ip[0], ip[1], ip[2], ip[3], ip[6]
        zs = lambda k: torch.zeros(k, dtype=torch.long, device=_device())  # noqa: E731
        self.scene = zs(n) if pscene is None else _t(pscene, torch.long)
        self.tscene = zs(nt) if tscene is None else _t(tscene, torch.long)
        self.skin = 0.2 * float(self.r.min())
        self.ref = None
        self.key = torch.zeros(0, dtype=torch.long, device=_device())
        self.state = torch.zeros(0, 3, dtype=torch.float64, device=_device())
        self.on = torch.zeros(0, dtype=torch.bool, device=_device())

    def _search(self, b):
        i, j = _sphere_pairs(b.x, self.r, self.scene, self.skin)
        wi, wt = _wall_pairs(b.x, self.r, self.scene, self.tri, self.tscene, self.skin)
        self.np = len(i)
        key = torch.cat([i * b.n + j, b.n * b.n + wi * len(self.tri) + wt])
        key, at = torch.sort(key)
        i, j = torch.cat([i, wi]), torch.cat([j, wt])
        state = torch.zeros(len(key), 3, dtype=torch.float64, device=b.x.device)
        on = torch.zeros(len(key), dtype=torch.bool, device=b.x.device)
        if len(self.key):
            pos = torch.searchsorted(self.key, key).clamp(max=len(self.key) - 1)
            same = self.key[pos] == key
            state[same], on[same] = self.state[pos[same]], self.on[pos[same]]
        self.key, self.i, self.j, self.state, self.on = key, i[at], j[at], state, on
        self.ref, self.tref = b.x.clone(), self.tri.clone()

    def forces(self, b, h):
        moved = self.ref is None
        if not moved:
            d2 = ((b.x - self.ref) ** 2).sum(1).max()
            t2 = ((self.tri - self.tref) ** 2).sum(2).max()
            moved = bool(torch.maximum(d2, t2) > (0.45 * self.skin) ** 2)
        if moved:
            self._search(b)
        n, i, j = self.np, self.i, self.j
        si, sj, wi, wt = i[:n], j[:n], i[n:], j[n:]
        # partner centres: the other sphere's, or the triangle's closest point
        q = b.x[si] - b.x[sj]
        cp = _closest(b.x[wi], self.tri[wt, 0], self.tri[wt, 1], self.tri[wt, 2])
        q = torch.cat([q, b.x[wi] - cp])
        length = (q * q).sum(1).sqrt()
        depth = torch.cat([self.r[si] + self.r[sj], self.r[wi]]) - length
        on = torch.where(self.on, depth >= 0, depth > 0)
        k = on.nonzero()[:, 0]
        sph = k < n
        I, Jp = i[k], j[k]
        nrm = q[k] / length[k, None]
        pj = torch.where(sph, Jp, torch.zeros_like(Jp))
        tj = torch.where(sph, torch.zeros_like(Jp), Jp)
        pnt = torch.where(sph[:, None], 0.5 * (b.x[I] + b.x[pj]), b.x[I] - q[k])
        vi = _cross(b.o[I], pnt - b.x[I]) + b.v[I]
        vj = _cross(b.o[pj], pnt - b.x[pj]) + b.v[pj]
        vw = torch.zeros_like(vi)
        if self.omega is not None:
            w = self.omega.expand_as(vi)
            vw = torch.where(self.moving[tj][:, None], _cross(w, pnt - self.point), vw)
        vij = torch.where(sph[:, None], vj, vw) - vi
        ma = torch.where(sph, 1.0 / (b.im[I] + b.im[pj]), b.m[I])
        en = self.damper * 2.0 * (self.kn * ma).sqrt()
        vn = (vij * nrm).sum(1)
        fn = self.kn * depth[k] + en * vn
        vt = vij - vn[:, None] * nrm
        st = self.state[k] * self.on[k][:, None] + h * vt
        ft = self.kn * self.kskn * st + (en * self.kskn)[:, None] * vt
        fl = (ft * ft).sum(1).sqrt()
        ft = torch.where((fl > self.mus * fn)[:, None], ft * (self.mud * fn / fl)[:, None], ft)
        f = fn[:, None] * nrm + ft
        self.state = torch.zeros_like(self.state)
        self.state[k] = st
        self.on = on
        F, T = torch.zeros_like(b.x), torch.zeros_like(b.x)
        F.index_add_(0, I, f)
        T.index_add_(0, I, _cross(pnt - b.x[I], f))
        F.index_add_(0, pj[sph], -f[sph])
        T.index_add_(0, pj[sph], _cross(pnt[sph] - b.x[pj[sph]], -f[sph]))
        return F, T

    def move(self, h):
        if self.omega is None:
            return
        R = _expmap(h * self.omega[None])[0]
        turned = (self.tri - self.point) @ R.T + self.point
        self.tri = torch.where(self.moving[:, None, None], turned, self.tri)


def _gravity(exc, t):
    a = sum(exc[8 + 3 * k] * math.sin(2.0 * math.pi * exc[9 + 3 * k] * t + exc[10 + 3 * k]) for k in range(int(exc[6])))
    return [exc[c] + exc[3 + c] * a for c in range(3)]


def _run_spheres(m, dt, steps, half, gravity, omega=None, pscene=None, tscene=None):
    """`steps` steps of a sphere model; gravity(k): (scenes, 3) at step k."""
    b, g = _Bodies(m), _Granular(m, pscene, tscene)
    g.omega = omega
    if half:
        b.half_step(dt)
        g.move(dt)
    for k in range(steps):
        F, T = g.forces(b, dt)
        F = F + b.m[:, None] * _t(gravity(k))[g.scene]
        b.advance(F, T, dt)
        g.move(dt)
    return b


class _Springs:
    """Nonlinear springs along the line of their ends, with lookup dashpots."""

    def __init__(self, m):
        n = m.sprnum
        self.a, self.b = _t(m.S.sprpart[0, :n], torch.long), _t(m.S.sprpart[1, :n], torch.long)
        self.pa, self.pb = _t(m.S.sprpnt[3:6, :n].T), _t(m.S.sprpnt[9:12, :n].T)
        self.s0 = _t(m.S.stroke0[:n])
        self.curve, self.dash = _t(np.array(m.spring_tab[:n])), _t(np.array(m.dashpot_tab[:n]))

    @staticmethod
    def _look(tab, x):
        k = (x[:, None] > tab[:, 1:-1, 0]).sum(1)
        lo, hi = (tab[torch.arange(len(x), device=x.device), k + c] for c in (0, 1))
        return lo[:, 1] + (hi[:, 1] - lo[:, 1]) / (hi[:, 0] - lo[:, 0]) * (x - lo[:, 0])

    def forces(self, b):
        arm_a, arm_b = _mv(b.L[self.a], self.pa - b.X[self.a]), _mv(b.L[self.b], self.pb - b.X[self.b])
        w = (b.x[self.b] + arm_b) - (b.x[self.a] + arm_a)
        length = (w * w).sum(1).sqrt()
        z = w / length[:, None]
        u = b.v[self.b] + _cross(b.o[self.b], arm_b) - b.v[self.a] - _cross(b.o[self.a], arm_a)
        self.stroke = length - self.s0
        spring = self._look(self.curve, self.stroke)
        total = spring + torch.where(spring == 0, torch.zeros_like(spring), self._look(self.dash, (z * u).sum(1)))
        self.total = total
        f = z * total[:, None]
        F, T = torch.zeros_like(b.x), torch.zeros_like(b.x)
        F.index_add_(0, self.a, f)
        T.index_add_(0, self.a, _cross(arm_a, f))
        F.index_add_(0, self.b, -f)
        T.index_add_(0, self.b, _cross(arm_b, -f))
        return F, T


def exact(case, seed):
    steps = case["steps"]
    if case.get("adaptive") or case.get("contact"):
        # the chosen steps need every particle's stiffness matrix and its
        # eigenvalues, the contacts between meshes the closest points of
        # millions of triangle pairs, one by one: far over 20 seconds
        return None
    down = (0.0, 0.0, -9.81)
    if case["kind"] == "hopper":
        m, dt = _hopper(case, seed)
        return _run_spheres(m, dt, steps, True, lambda k: [down]).outputs()
    if case["kind"] == "drum":
        m, dt, _ = scenes.drum(case["spheres"], seed=seed)
        return _run_spheres(m, dt, steps, True, lambda k: [down], omega=_t([2.0, 0.0, 0.0])).outputs()
    if case["kind"] == "batch":
        made = _boxes(case, seed)
        P, _ = batch.pool([m for m, _, _ in made])
        dt = made[0][1]
        return _run_spheres(P, dt, steps, True, lambda k: [_gravity(e, k * dt) for _, _, e in made],
                            pscene=P.pscene[:P.parnum], tscene=P.tscene[:P.trinum]).outputs()
    if case["kind"] == "serve":
        xs, vs, es = [], [], []
        for q in _requests(case, seed):
            b = _run_spheres(q.model, q.dt, q.steps, False, lambda k: [_gravity(q.excitation, k * q.dt)])
            g0 = _t(q.excitation[0:3])
            energy = (0.5 * b.m * (b.v * b.v).sum(1) + 0.5 * (b.O * _mv(b.J, b.O)).sum(1)
                      - b.m * (b.x * g0).sum(1)).sum()
            xs.append(b.x.T.cpu().numpy())
            vs.append(b.v.T.cpu().numpy())
            es.append(float(energy))
        return {"position": np.concatenate(xs, axis=1), "linear": np.concatenate(vs, axis=1), "energy": np.array(es)}
    m, dt = scenes.spring_lattice(case["side"], seed=seed)
    b, s = _Bodies(m), _Springs(m)
    base = m.parnum - 1
    weight = b.m[:, None] * _t([down])
    b.half_step(dt)
    for k in range(steps):
        F, T = s.forces(b)
        F = F + weight
        F[base] = b.m[base] * _t([0.5 * 9.81 * math.sin(2.0 * math.pi * 5.0 * (k * dt)), 0.0, 0.0])
        T[base] = 0.0 if m.prescribe[0]["ang"] is not None and m.prescribe[0]["angkind"] == 0 else T[base]
        b.advance(F, T, dt)
    out = b.outputs()
    out["spring_force"], out["stroke"] = s.total.cpu().numpy(), s.stroke.cpu().numpy()
    return out
