"""The work that users have this framework do, as measurable cases.

A pass is what an evolving simulation does between two outputs: `steps` steps of
the mesh (or of the batch of boxes) and the download of its state into pinned
host memory.  Meshes are uniform (one to many blocks, periodic or with physical
sides), statically refined, or batches of independent boxes; FP64 and mixed
precision; hydro and MHD; the Heun and the VL2 integrator; every face on HLLD
or the learned selector's choice.  Sizes are those of the benchmark and of the
tests' meshes, and ragged ones between them.

    listed()             the cases that stand for the range
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the engine with its initial state set
    run(state)           one pass: steps, then the state in host memory
    exact(case, seed)    the same pass in plain torch FP64 (uniform periodic
                         MHD, hydro with any sides, boxes), else None
"""
import functools
import math

import numpy as np
import torch

DEV = "cuda:0"
GAMMA_MHD, GAMMA_HYDRO, CFL = 5.0 / 3.0, 1.4, 0.3
FLOOR = 1e-9                       # density and temperature floors (the defaults)
W_FIX = (0.5, 0.4, 0.1, -0.05, 0.02)
BATCH_SEED = 5                     # the benchmark's batch: its boxes' sizes


def _mesh(name, mhd, nb, n, steps, precision, sides="per", riemann=0, integrator=0, flow="vortex"):
    return {"name": name, "kind": "mesh", "mhd": mhd, "nbx": nb[0], "nby": nb[1], "nbz": nb[2],
            "nx": n[0], "ny": n[1], "nz": n[2], "steps": steps, "precision": precision, "sides": sides,
            "riemann": riemann, "integrator": integrator, "flow": flow}


def _boxes(name, count, steps, precision, batched, riemann=0):
    return {"name": name, "kind": "boxes", "boxes": count, "steps": steps, "precision": precision,
            "batched": batched, "riemann": riemann}


def _refined(name, mhd, nb, n, levels, steps, precision):
    return {"name": name, "kind": "refined", "mhd": mhd, "nbx": nb[0], "nby": nb[1], "nbz": nb[2],
            "nx": n[0], "ny": n[1], "nz": n[2], "levels": levels, "steps": steps, "precision": precision}


def listed():
    return [
        # a few steps of a small test mesh: launches and latency
        _mesh("mhd_fp64_32", True, (2, 2, 2), (16, 16, 16), 5, 2),
        # the plain small hydro configuration: planar shock, 20 steps
        _mesh("hydro_fp64_64", False, (2, 2, 2), (32, 32, 32), 20, 2, flow="shock"),
        # hydro on ragged odd blocks between outflow, reflecting and free sides
        _mesh("hydro_mixed_sides", False, (3, 2, 2), (45, 28, 19), 10, 1, sides="out ref per per fre fre",
              flow="shock"),
        # supersonic turbulence on a mesh of eight blocks, mixed precision
        _mesh("mhd_mixed_64", True, (2, 2, 2), (32, 32, 32), 10, 1, flow="turbulence"),
        # the VL2 integrator on ragged odd blocks
        _mesh("mhd_vl2_ragged", True, (3, 2, 2), (40, 27, 18), 10, 1, integrator=1),
        # the benchmark's mesh in FP64, mixed precision, and with the learned selector
        _mesh("mhd_fp64_256", True, (4, 4, 4), (64, 64, 64), 20, 2),
        _mesh("mhd_mixed_256", True, (4, 4, 4), (64, 64, 64), 50, 1),
        _mesh("mhd_learned_256", True, (4, 4, 4), (64, 64, 64), 50, 1, riemann=2),
        # independent boxes of uneven sizes: a graph per size in FP64, and one
        # launch per kernel kind over all of them in mixed precision
        _boxes("boxes_fp64_64", 64, 10, 2, False),
        _boxes("boxes_batched_mixed_256", 256, 10, 1, True),
        # refined meshes of many small blocks: the hydro shock between slabs, and the
        # magnetized blast refined three times by its gradients
        _refined("refined_hydro_mixed", False, (8, 8, 8), (16, 16, 16), 2, 20, 1),
        _refined("refined_blast_mixed", True, (8, 8, 8), (16, 16, 16), 3, 10, 1),
    ]


def draw(rng):
    kind = rng.choice(["mhd", "mhd", "mhd", "hydro", "hydro", "learned", "boxes", "refined"])
    precision = rng.choice([1, 2])
    steps = rng.randint(1, 12)
    if kind == "boxes":
        return {k: v for k, v in _boxes("", int(round(math.exp(rng.uniform(math.log(4), math.log(256))))), steps,
                                        precision, rng.random() < 0.5).items() if k != "name"}
    if kind == "refined":
        mhd = rng.random() < 0.5
        r = 2 * rng.randint(2, 3)
        n = [2 * rng.randint(4, 10) for _ in range(3)]
        c = _refined("", mhd, (r, r, r), n, rng.randint(1, 2), steps, precision)
        return {k: v for k, v in c.items() if k != "name"}
    n = [int(round(math.exp(rng.uniform(math.log(8), math.log(80))))) for _ in range(3)]
    nb = [rng.randint(1, 4) for _ in range(3)]
    while n[0] * n[1] * n[2] * nb[0] * nb[1] * nb[2] > 12_000_000:
        a = max(range(3), key=lambda q: n[q] * nb[q])
        if nb[a] > 1:
            nb[a] -= 1
        else:
            n[a] //= 2
    if kind == "hydro":
        sides = []
        for _ in range(3):
            sides += ["per", "per"] if rng.random() < 0.5 else [rng.choice(["out", "ref", "fre", "fixd"])
                                                                for _ in range(2)]
        c = _mesh("", False, nb, n, steps, precision, sides=" ".join(sides), flow="shock",
                  integrator=int(rng.random() < 0.25))
    elif kind == "learned":
        c = _mesh("", True, nb, n, steps, 1, riemann=2, flow=rng.choice(["vortex", "turbulence"]))
    else:
        c = _mesh("", True, nb, n, steps, precision, integrator=int(rng.random() < 0.25),
                  riemann=int(rng.random() < 0.15), flow=rng.choice(["vortex", "turbulence"]))
    return {k: v for k, v in c.items() if k != "name"}


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _axes(shape):
    """Cell centres of a unit domain along x, y, z, shaped for [box, z, y, x]."""
    out = []
    for a in range(3):
        view = [1, 1, 1, 1]
        view[3 - a] = shape[a]
        out.append(((torch.arange(shape[a], device=DEV, dtype=torch.float64) + 0.5) / shape[a]).view(view))
    return out


def _conserved(rho, p, v, b, gamma):
    e = p / (gamma - 1) + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    if b is not None:
        bc = [(q + torch.roll(q, -1, 3 - a)) / 2 for a, q in enumerate(b)]
        e = e + 0.5 * (bc[0] ** 2 + bc[1] ** 2 + bc[2] ** 2)
    return torch.stack([rho, e, rho * v[0], rho * v[1], rho * v[2]])


def _flow_mhd(flow, shape, g):
    """Conserved words [5, 1, z, y, x] and lower-face B [3, 1, z, y, x] on a periodic unit domain."""
    x, y, z = _axes(shape)
    full = (1, shape[2], shape[1], shape[0])
    tau = 2 * math.pi
    ph = _rand(g, 4) * tau
    noise = [1e-3 * (2 * _rand(g, *full) - 1) for _ in range(3)]
    zero = torch.zeros(full, device=DEV, dtype=torch.float64)
    if flow == "vortex":
        # Orszag-Tang type with a guide field along z: B_a has no dependence on a, so face B is divergence free
        rho = zero + 25 / (36 * math.pi)
        p = zero + 5 / (12 * math.pi)
        v = [-torch.sin(tau * y + ph[0]) + noise[0], torch.sin(tau * x + ph[1]) + noise[1], noise[2]]
        b = [zero - torch.sin(tau * y + ph[2]) / math.sqrt(4 * math.pi),
             zero + torch.sin(2 * tau * x + ph[3]) / math.sqrt(4 * math.pi),
             zero + 0.25 / math.sqrt(4 * math.pi)]
    else:
        # random-phase solenoidal velocity, rms Mach 5, sound speed 1, uniform B_x at beta 0.1
        rho, p = zero + 1, zero + 1 / GAMMA_MHD
        k = torch.randint(1, 5, (12, 3), generator=g, device=DEV).double()
        a = torch.linalg.cross(2 * _rand(g, 12, 3) - 1, k)
        a = a / a.norm(dim=1, keepdim=True).clamp_min(1e-3) / (k * k).sum(1, keepdim=True)
        a = a * (5 * math.sqrt(2) / a.norm())
        v = [q.clone() for q in noise]
        for m in range(12):
            c = torch.cos(tau * (k[m, 0] * x + k[m, 1] * y + k[m, 2] * z) + tau * _rand(g, 1))
            for d in range(3):
                v[d] += a[m, d] * c
        b = [zero + math.sqrt(2 / GAMMA_MHD / 0.1), zero, zero]
    return _conserved(rho, p, v, b, GAMMA_MHD), torch.stack(b)


def _flow_hydro(shape, g):
    x = _axes(shape)[0]
    full = (1, shape[2], shape[1], shape[0])
    left = (x < 0.5).double()
    rho = (0.125 + 0.875 * left) * (1 + 1e-3 * (2 * _rand(g, *full) - 1))
    p = 0.1 + 0.9 * left + torch.zeros_like(rho)
    v = [0.05 * (2 * _rand(g, 1) - 1) + 1e-3 * (2 * _rand(g, *full) - 1) for _ in range(3)]
    return _conserved(rho, p, v, None, GAMMA_HYDRO), None


def _box_sizes(count):
    """Edge lengths of the benchmark's batch of boxes (SplitMix64 draws)."""
    mask = (1 << 64) - 1

    def mix(x):
        x = (x + 0x9E3779B97F4A7C15) & mask
        x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & mask
        return x ^ (x >> 31)
    out = []
    for k in range(count):
        h = mix(mix((BATCH_SEED * 0x100000001B3 + 32) & mask) ^ k)
        out.append((16, 24, 32, 48, 64)[min(4, int((h >> 11) * (2.0 / 9007199254740992.0) * 2.5))])
    return out


def _flow_boxes(n, count, g):
    """Boxes of n^3 cells: random density, pressure, velocity amplitude and field orientation each."""
    x, y, z = _axes((n, n, n))
    q = [_rand(g, count, 1, 1, 1) for _ in range(6)]
    rho, p, beta = 0.5 + 1.5 * q[0], 0.1 + 9.9 * q[1], 0.05 + 9.95 * q[2]
    amp = torch.sqrt(GAMMA_MHD * p / rho) * (0.1 + 1.9 * q[3])
    ct, ph = 2 * q[4] - 1, 2 * math.pi * q[5]
    st, bm = torch.sqrt(1 - ct * ct), torch.sqrt(2 * p / beta)
    one = torch.ones(count, n, n, n, device=DEV, dtype=torch.float64)
    v = [amp * (torch.sin(2 * math.pi * s) + 1e-3 * (2 * _rand(g, count, n, n, n) - 1)) for s in (y, z, x)]
    b = [one * bm * st * torch.cos(ph), one * bm * st * torch.sin(ph), one * bm * ct]
    return _conserved(rho * one, p * one, v, b, GAMMA_MHD), torch.stack(b)


def _to_blocks(q, nb, n, extra=0, axis=0):
    """[z, y, x] of the whole mesh as [block, z, y, x], x-fastest block order; extra: one more plane along
    `axis` (the upper faces of the last cells, periodic)."""
    if extra:
        out = []
        for b in range(nb[0] * nb[1] * nb[2]):
            r = (b % nb[0], (b // nb[0]) % nb[1], b // (nb[0] * nb[1]))
            sel = [(torch.arange(n[a] + (a == axis), device=q.device) + r[a] * n[a]) % (nb[a] * n[a])
                   for a in range(3)]
            out.append(q[sel[2]][:, sel[1]][:, :, sel[0]])
        return torch.stack(out)
    return (q.reshape(nb[2], n[2], nb[1], n[1], nb[0], n[0]).permute(0, 2, 4, 1, 3, 5)
            .reshape(nb[0] * nb[1] * nb[2], n[2], n[1], n[0]))


def _host_u(u, b):
    """Block arrays [5, blk, z, y, x] (and lists of face arrays) as the engine's [blk, z, y, x, words]."""
    if b is not None:
        bc = []
        for a in range(3):
            dim = 3 - a
            m = b[a].shape[dim] - 1
            bc.append((b[a].narrow(dim, 0, m) + b[a].narrow(dim, 1, m)) / 2)
        u = torch.cat([u, torch.stack(bc)])
    return u.permute(1, 2, 3, 4, 0).contiguous()


def _host_b(b, n):
    nblk = b[0].shape[0]
    out = torch.zeros((nblk, n[2] + 5, n[1] + 5, n[0] + 5, 3), device=DEV, dtype=torch.float64)
    for a in range(3):
        s = b[a].shape
        out[:, 2:2 + s[1], 2:2 + s[2], 2:2 + s[3], a] = b[a]
    return out


def _pinned(t):
    return torch.empty(t.shape, dtype=torch.float64, pin_memory=True).copy_(t).numpy()


def _owned(bf, n):
    """The faces a block owns (its storage also has ghost layers): per component [block, z, y, x]."""
    return [bf[:, 2:2 + n[2] + (a == 2), 2:2 + n[1] + (a == 1), 2:2 + n[0] + (a == 0), a] for a in range(3)]


def _dims(case):
    return (case["nbx"], case["nby"], case["nbz"]), (case["nx"], case["ny"], case["nz"])


def _initial(case, seed):
    nb, n = _dims(case)
    shape = [nb[a] * n[a] for a in range(3)]
    g = _gen(seed)
    return _flow_mhd(case["flow"], shape, g) if case["mhd"] else _flow_hydro(shape, g)


# ------------------------------------------------------------------ handles
@functools.lru_cache(maxsize=1)
def _selector():
    """The learned selector's weights: a program trains them once, on faces of its flow labelled by the gap
    between both solvers' fluxes, and keeps them."""
    from kratos_b200 import selector as S
    u, b = _flow_mhd("vortex", (48, 48, 48), _gen(3))
    u, b, _, _ = _evolve(u, b, 6, GAMMA_MHD, ("per",) * 6, False, False, False)
    w, bc, _ = _prims(u, b, GAMMA_MHD)
    feats, gaps = [], []
    for a in range(3):
        dim, t1, t2 = 3 - a, (a + 1) % 3, (a + 2) % 3
        lr = [_faces(w[k], a, ("per", "per"), (False, 0.0), True) for k in (0, 1, 2 + a, 2 + t1, 2 + t2)]
        lr += [_faces(bc[t], a, ("per", "per"), (False, 0.0), True) for t in (t1, t2)]
        bx = torch.cat([b[a], b[a].narrow(dim, 0, 1)], dim=dim)
        l, r = [x[0] for x in lr], [x[1] for x in lr]
        fd, fe = _hlld(l, r, bx, GAMMA_MHD, False), _hlld(l, r, bx, GAMMA_MHD, True)
        m = [(x + y) / 2 for x, y in lr]
        d = [x - y for x, y in lr]
        cs2, va2 = GAMMA_MHD * m[1] / m[0], (bx ** 2 + m[5] ** 2 + m[6] ** 2) / m[0]
        c = torch.sqrt(cs2 + va2)
        iva = 1 / (c * torch.sqrt(m[0]))
        f = [d[0] / m[0], d[1] / m[1], d[2] / c, d[3] / c, d[4] / c, m[2] / c, m[3] / c, m[4] / c,
             d[5] * iva, d[6] * iva, bx * iva, m[5] * iva, m[6] * iva, torch.sqrt(cs2) / c]
        f += [f[0].abs(), f[1].abs()]
        s = [m[0] * c, m[0] * c ** 3] + [m[0] * c * c] * 3 + [torch.sqrt(m[0]) * c * c] * 2
        feats.append(torch.stack([q.reshape(-1) for q in f], dim=1))
        gaps.append(torch.stack([((x - y).abs() / z).reshape(-1) for x, y, z in zip(fe, fd, s)]).amax(0))
    x, y = torch.cat(feats), (torch.cat(gaps) < S.DEFAULT_TOL)
    x, y = S.shuffle(x.float().cpu().numpy(), y.float().cpu().numpy(), 0)
    return S.train(x, y, epochs=10)[0]


@functools.lru_cache(maxsize=8)
def _regions(mhd, nb, n, levels):
    if mhd:
        from kratos_b200.amr import gradient_regions
        return gradient_regions(nb, n, levels)
    return [(lv, (0.5 - 0.2 / 2 ** lv, 0.0, 0.0), (0.5 + 0.2 / 2 ** lv, 1.0, 1.0)) for lv in range(1, levels + 1)]


def _refined_state(d, case, seed):
    """Blast (MHD) or planar shock (hydro) on the blocks of a refined mesh, with seeded density noise."""
    nb, n = _dims(case)
    g = _gen(seed)
    lvl = torch.tensor(d.level, device=DEV, dtype=torch.float64)
    reg = torch.tensor(d.reg, device=DEV, dtype=torch.float64)
    x = []
    for a in range(3):
        i = (torch.arange(n[a], device=DEV, dtype=torch.float64) + 0.5) / n[a]
        view = [d.nblk, 1, 1, 1]
        view[3 - a] = n[a]
        x.append(((reg[:, a, None] + i[None]) / (nb[a] * 2.0 ** lvl[:, None])).view(view))
    full = (d.nblk, n[2], n[1], n[0])
    noise = 1 + 1e-3 * (2 * _rand(g, *full) - 1)
    zero = torch.zeros(full, device=DEV, dtype=torch.float64)
    if case["mhd"]:
        # a moving medium: in a static one rounding alone decides which side is upwind
        r = torch.sqrt(sum((q - 0.5) ** 2 for q in x))
        p = 0.1 + 49.95 * (1 - torch.tanh((r - 0.1) / 0.015))
        rho, v, b = noise, (0.3, 0.2, 0.1), (math.sqrt(0.5), math.sqrt(0.5), 0.25)
        e = p / (GAMMA_MHD - 1) + 0.5 * rho * sum(q * q for q in v) + 0.5 * sum(q * q for q in b)
        bf = torch.zeros((d.nblk, n[2] + 5, n[1] + 5, n[0] + 5, 3), device=DEV, dtype=torch.float64)
        for a in range(3):
            bf[..., a] = b[a]
        u = torch.stack([rho, e] + [rho * q for q in v] + [zero + q for q in b], dim=-1)
        return u, bf
    left = (x[0] < 0.5).double()
    u = torch.stack([(0.125 + 0.875 * left) * noise, (0.1 + 0.9 * left + zero) / (GAMMA_HYDRO - 1),
                     zero, zero, zero], dim=-1)
    return u, None


def prepare(case, seed):
    from kratos_b200 import Dynamics
    if case["kind"] == "boxes":
        from kratos_b200.boxes import BoxBatch
        bb = BoxBatch(BATCH_SEED, case["boxes"], gamma=GAMMA_MHD, batched=case["batched"],
                      precision=case["precision"], riemann=case["riemann"])
        bufs = {}
        g = _gen(seed)
        for n, (d, ids) in bb.groups.items():
            u, b = _flow_boxes(n, len(ids), g)
            faces = [torch.cat([b[a], b[a].narrow(3 - a, 0, 1)], dim=3 - a) for a in range(3)]
            bufs[n] = (_pinned(_host_u(u, faces)), _pinned(_host_b(faces, (n, n, n))))
            d.set_state(*bufs[n])
        return {"case": case, "batch": bb, "bufs": bufs}
    nb, n = _dims(case)
    kw = {"precision": case["precision"], "gamma": GAMMA_MHD if case["mhd"] else GAMMA_HYDRO}
    if case["kind"] == "refined":
        d = Dynamics(case["mhd"], nb, n, regions=_regions(case["mhd"], nb, n, case["levels"]), **kw)
        u, bf = _refined_state(d, case, seed)
    else:
        if case["riemann"] == 2:
            kw["sel_period"] = 16
        d = Dynamics(case["mhd"], nb, n, riemann=case["riemann"], integrator=case["integrator"],
                     kinds=_kinds(case), w_fix=W_FIX, **kw)
        if case["riemann"] == 2:
            from kratos_b200 import selector as S
            d.set_selector(_selector(), S.DEFAULT_THRESHOLD)
        u, b = _initial(case, seed)
        u = torch.stack([_to_blocks(q[0], nb, n) for q in u])
        if case["mhd"]:
            faces = [_to_blocks(b[a][0], nb, n, 1, a) for a in range(3)]
            u, bf = _host_u(u, faces), _host_b(faces, n)
        else:
            u, bf = _host_u(u, None), None
    u = _pinned(u)
    bf = _pinned(bf) if bf is not None else None
    d.set_state(u, bf)
    return {"case": case, "dyn": d, "u": u, "bf": bf}


def _kinds(case):
    k = case["sides"].split()
    return tuple(k * 6 if len(k) == 1 else k)


def run(state):
    case = state["case"]
    if case["kind"] == "boxes":
        bb = state["batch"]
        bb.step(case["steps"])
        out = {}
        for n, (d, _) in bb.groups.items():
            u, bf = d.get_state(*state["bufs"][n])
            out["n%d" % n] = [u] + _owned(bf, d.n)
        t, dt = bb.times()
        return {"state": out, "t": t, "dt": dt}
    d = state["dyn"]
    d.step(case["steps"])
    u, bf = d.get_state(state["u"], state["bf"])
    tm = d.time()
    return {"state": [u] + (_owned(bf, d.n) if case["mhd"] else []), "t": tm["t"], "dt": tm["dt_last"]}


# --------------------------------------------------------------------- sizes
def _cells(case):
    if case["kind"] == "boxes":
        return sum(n ** 3 for n in _box_sizes(case["boxes"]))
    nb, n = _dims(case)
    cells = math.prod(nb) * math.prod(n)
    if case["kind"] == "refined":
        cells *= _refined_blocks(case["mhd"], nb, n, case["levels"]) / math.prod(nb)
    return cells


@functools.lru_cache(maxsize=8)
def _refined_blocks(mhd, nb, n, levels):
    """Leaves of the refined mesh: every refined block becomes eight, and its neighbours (periodic, edges and
    corners too) are at most one level coarser."""
    inside = [set() for _ in range(levels + 1)]           # refined blocks of each level

    def refine(lv, p):
        if p in inside[lv]:
            return
        if lv:
            for d in np.ndindex(3, 3, 3):
                q = [(p[a] + d[a] - 1) % (nb[a] << lv) >> 1 for a in range(3)]
                refine(lv - 1, tuple(q))
        inside[lv].add(p)
    for level, lo, hi in _regions(mhd, nb, n, levels):
        span = []
        for a in range(3):
            m = nb[a] << level
            i0, i1 = int(math.floor(lo[a] * m)), int(math.ceil(hi[a] * m))
            span.append(range(max(0, min(i0, m - 1)), min(m, max(i1, i0 + 1))))
        for p in ((i, j, k) for i in span[0] for j in span[1] for k in span[2]):
            refine(level - 1, tuple(q >> 1 for q in p))
    return math.prod(nb) + 7 * sum(len(q) for q in inside)


def work(case):
    """Per zone and step: the state read and written once (8 MHD or 5 hydro FP64 words), and the arithmetic of
    two stages of three face solves (reconstruction and Riemann solver), conversion and update; per pass, the
    download of the state."""
    words = 5 if case["kind"] != "boxes" and not case["mhd"] else 8
    cells, steps = _cells(case), case["steps"]
    flops = 2 * (3 * 420 + 150) if words == 8 else 2 * (3 * 190 + 50)
    return {"bytes": cells * (steps * words * 8 * 2 + words * 8), "flops": cells * steps * flops}


def tolerance(case):
    """About four times the difference between the engine's builds with and without fused multiply-adds."""
    mhd = case["kind"] == "boxes" or case["mhd"]
    if case["precision"] == 2:
        return {"rel": 1e-11, "max": 1e-8}
    if case.get("riemann") == 2:
        # a face whose logit lies at the threshold takes the other solver
        fine = case["kind"] == "mesh" and case["flow"] == "vortex" and _cells(case) > 4_000_000
        return {"rel": 5e-5, "max": 2e-3} if fine else {"rel": 1.2e-2, "max": 0.4}
    return {"rel": 6e-6, "max": 2.5e-3} if mhd else {"rel": 1e-6, "max": 1e-4}


# --------------------------------------------------------------------- exact
def _ghosted(q, a, bc, mom):
    """q [.., z, y, x] with two ghost cells along axis a; bc: the kinds of both sides; mom: (word is the normal
    velocity, fixed value)."""
    dim = q.dim() - 1 - a
    n = q.shape[dim]
    if bc[0] == "per":
        return torch.cat([q.narrow(dim, n - 2, 2), q, q.narrow(dim, 0, 2)], dim=dim)
    ends = []
    for s, kind in enumerate(bc):
        c0, c1 = (q.narrow(dim, n - 1, 1), q.narrow(dim, n - 2, 1)) if s else (q.narrow(dim, 0, 1), q.narrow(dim, 1, 1))
        if kind == "ref":
            g = [c0, c1] if not mom[0] else [-c0, -c1]
        elif kind == "fixd":
            g = [torch.full_like(c0, mom[1])] * 2
        else:
            if kind == "out" and mom[0]:
                c0 = torch.where(c0 * (-1 if s else 1) > 0, torch.zeros_like(c0), c0)
            g = [c0, c0]
        ends.append(g if s else g[::-1])
    return torch.cat(ends[0] + [q] + ends[1], dim=dim)


def _faces(q, a, bc, mom, plm):
    """Left and right states of the n + 1 faces along axis a (van Leer limited slopes, or piecewise constant)."""
    dim = q.dim() - 1 - a
    n = q.shape[dim]
    e = _ghosted(q, a, bc, mom)
    if not plm:
        return e.narrow(dim, 1, n + 1), e.narrow(dim, 2, n + 1)
    d = e.narrow(dim, 1, n + 3) - e.narrow(dim, 0, n + 3)
    dl, dr = d.narrow(dim, 0, n + 2), d.narrow(dim, 1, n + 2)
    p = dl * dr
    s = torch.where(p > 0, p / torch.where(p > 0, dl + dr, 1.0), torch.zeros_like(p))
    c = e.narrow(dim, 1, n + 2)
    return (c + s).narrow(dim, 0, n + 1), (c - s).narrow(dim, 1, n + 1)


def _hllc(l, r, gam):
    """Flux of (rho, p, vn, vt1, vt2) states: HLLC with Roe-averaged outer speeds."""
    cv = 1 / (gam - 1)
    e, c, h, sq = [], [], [], []
    for w in (l, r):
        e.append(w[1] * cv + 0.5 * w[0] * (w[2] ** 2 + w[3] ** 2 + w[4] ** 2))
        c.append(torch.sqrt(gam * torch.clamp_min(w[1] / w[0], 0)))
        sq.append(torch.sqrt(w[0]))
        h.append((e[-1] + w[1]) / sq[-1])
    isum = 1 / (sq[0] + sq[1])
    vr = [(sq[0] * l[k] + sq[1] * r[k]) * isum for k in (2, 3, 4)]
    q = (h[0] + h[1]) * isum - 0.5 * (vr[0] ** 2 + vr[1] ** 2 + vr[2] ** 2)
    a = torch.sqrt(torch.clamp_min((gam - 1) * q, 0))
    al, ar = torch.minimum(vr[0] - a, l[2] - c[0]), torch.maximum(vr[0] + a, r[2] + c[1])
    bp, bm = torch.clamp_min(ar, 0), torch.clamp_max(al, 0)
    tl, tr = l[1] + (l[2] - al) * l[0] * l[2], r[1] + (r[2] - ar) * r[0] * r[2]
    ml, mr = l[0] * (l[2] - al), -r[0] * (r[2] - ar)
    am = (tl - tr) / (ml + mr)
    cp = torch.clamp_min((ml * tr + mr * tl) / (ml + mr), 0)
    up = am >= 0
    tiny = 1e-300
    b = torch.where(up, bm, bp)
    den = am - b
    den = torch.where(den.abs() < tiny, torch.where(den > 0, tiny, -tiny), den)
    s, sm = am / den, -b / den
    out = []
    w = [torch.where(up, x, y) for x, y in zip(l, r)]
    ew = torch.where(up, e[0], e[1])
    v = w[2] - b
    for k in range(5):
        f = w[0] * v if k == 0 else w[1] * w[2] + ew * v if k == 1 else w[0] * w[k] * v
        if k == 2:
            f = f + w[1]
        out.append(s * f)
    out[2] = out[2] + sm * cp
    out[1] = out[1] + sm * cp * am
    return out


def _hlld(l, r, bx, gam, hlle):
    """Fluxes (rho, E, m_n, m_t1, m_t2, B_t1, B_t2) of states (rho, p, vn, vt1, vt2, bt1, bt2) with normal
    field bx."""
    b2 = bx * bx
    cv = 1 / (gam - 1)
    side = []
    for w in (l, r):
        bt2 = w[5] ** 2 + w[6] ** 2
        pm = 0.5 * (b2 + bt2)
        u = [w[0], w[1] * cv + 0.5 * w[0] * (w[2] ** 2 + w[3] ** 2 + w[4] ** 2) + pm,
             w[0] * w[2], w[0] * w[3], w[0] * w[4], w[5], w[6]]
        cs, va, vt = gam * w[1] / w[0], b2 / w[0], bt2 / w[0]
        cf = torch.sqrt(0.5 * (va + vt + cs + torch.sqrt((va + vt - cs) ** 2 + 4 * cs * vt)))
        pt = w[1] + pm
        f = [u[2], w[2] * (pt + u[1] - b2) - bx * (w[3] * w[5] + w[4] * w[6]), pt - b2 + u[2] * w[2],
             -bx * w[5] + u[3] * w[2], -bx * w[6] + u[4] * w[2], -bx * w[3] + w[5] * w[2], -bx * w[4] + w[6] * w[2]]
        side.append((w, u, cf, pt, f))
    sl = torch.minimum(l[2] - side[0][2], r[2] - side[1][2])
    sr = torch.maximum(l[2] + side[0][2], r[2] + side[1][2])
    if hlle:
        a, b = torch.clamp_max(sl, 0), torch.clamp_min(sr, 0)
        return [(b * f - a * g + a * b * (y - x)) / (b - a)
                for f, g, x, y in zip(side[0][4], side[1][4], side[0][1], side[1][1])]
    dl, dr = sl - l[2], sr - r[2]
    ul, ur, pl, pr = side[0][1], side[1][1], side[0][3], side[1][3]
    s0 = (dr * ur[2] - pr - dl * ul[2] + pl) / (dr * ur[0] - dl * ul[0])
    ps = pl + ul[0] * dl * (s0 - l[2])
    star = []
    for (w, u, _, pt, _), s, d in ((side[0], sl, dl), (side[1], sr, dr)):
        dm = s - s0
        rs = u[0] * d / dm
        den = u[0] * d * dm - b2
        flat = den.abs() < 1e-4 * ps
        den = torch.where(flat, torch.ones_like(den), den)
        tv = torch.where(flat, 0.0, bx * (d - dm) / den)
        tb = torch.where(flat, 1.0, (u[0] * d * d - b2) / den)
        v1, v2, c1, c2 = w[3] - w[5] * tv, w[4] - w[6] * tv, w[5] * tb, w[6] * tb
        ub = s0 * bx + v1 * c1 + v2 * c2
        wb = w[2] * bx + w[3] * w[5] + w[4] * w[6]
        es = (bx * (wb - ub) - pt * w[2] + d * u[1] + ps * s0) / dm
        star.append(([rs, es, rs * s0, rs * v1, rs * v2, c1, c2], ub, torch.sqrt(rs), v1, v2))
    (usl, ubl, ql, v1l, v2l), (usr, ubr, qr, v1r, v2r) = star
    m1, p1 = s0 - bx.abs() / ql, s0 + bx.abs() / qr
    sg = torch.where(bx > 0, 1.0, -1.0)
    live = b2 > 1e-4 * ps
    inv = 1 / (ql + qr)
    vt = [inv * (ql * x + qr * y + sg * (d - c)) for x, y, c, d in
          ((v1l, v1r, usl[5], usr[5]), (v2l, v2r, usl[6], usr[6]))]
    bt = [inv * (ql * d + qr * c + sg * ql * qr * (y - x)) for x, y, c, d in
          ((v1l, v1r, usl[5], usr[5]), (v2l, v2r, usl[6], usr[6]))]
    uv = s0 * bx + vt[0] * bt[0] + vt[1] * bt[1]
    left = s0 >= 0
    out = []
    for k in range(7):
        us, f, u = torch.where(left, usl[k], usr[k]), torch.where(left, side[0][4][k], side[1][4][k]), \
            torch.where(left, ul[k], ur[k])
        rs = torch.where(left, usl[0], usr[0])
        if k == 1:
            ss = us + torch.where(left, -ql * sg * (ubl - uv), qr * sg * (ubr - uv))
        elif k in (3, 4):
            ss = rs * vt[k - 3]
        elif k in (5, 6):
            ss = bt[k - 5]
        else:
            ss = us
        ss = torch.where(live, ss, us)
        so, si = torch.where(left, sl, sr), torch.where(left, m1, p1)
        inner = torch.where(left, m1 < 0, p1 > 0)         # the double-star region holds the face
        g = f + so * (us - u)
        g = torch.where(inner, f - so * u - (si - so) * us + si * ss, g)
        g = torch.where(sl >= 0, side[0][4][k], torch.where(sr <= 0, side[1][4][k], g))
        out.append(g)
    return out


def _prims(u, b, gam):
    """Primitives (and healed conserved words) of cells, MHD with face B [3]."""
    rho = torch.where(u[0] < FLOOR, FLOOR, u[0])
    em = 0
    bc = None
    if b is not None:
        bc = [(q + torch.roll(q, -1, 3 - a)) / 2 for a, q in enumerate(b)]
        em = 0.5 * (bc[0] ** 2 + bc[1] ** 2 + bc[2] ** 2)
    v = [u[2 + a] / rho for a in range(3)]
    ek = 0.5 * (u[2] ** 2 + u[3] ** 2 + u[4] ** 2) / rho
    p = (u[1] - em - ek) * (gam - 1)
    low = p < FLOOR * rho
    p = torch.where(low, FLOOR * rho, p)
    e = torch.where(low, ek + p / (gam - 1) + em, u[1])
    return torch.stack([rho, p] + v), bc, torch.stack([rho, e, u[2], u[3], u[4]])


def _time_step(w, b, bc, dx, gam, boxes):
    """CFL minimum: one dt, or one for each box."""
    best = None
    for a in range(3):
        cs = gam * w[1] / w[0]
        if b is None:
            c = torch.sqrt(cs)
        else:
            t = [bc[(a + 1) % 3], bc[(a + 2) % 3]]
            n2 = torch.maximum(b[a].abs(), torch.roll(b[a], -1, 3 - a).abs()) ** 2
            va, vt = n2 / w[0], (t[0] ** 2 + t[1] ** 2) / w[0]
            c = torch.sqrt(0.5 * (va + vt + cs + torch.sqrt((va + vt - cs) ** 2 + 4 * cs * vt)))
        s = (c + w[2 + a].abs()) / dx[a]
        best = s if best is None else torch.maximum(best, s)
    m = best.amax(dim=(1, 2, 3), keepdim=True) if boxes else best.max().view(1, 1, 1, 1)
    return CFL / m


def _rates(w, b, bc, dx, gam, kinds, plm, hlle):
    """Flux divergence [5] and, MHD, the edge fields [3] of one stage."""
    mhd = b is not None
    div, mass, emf = 0, [None] * 3, [[None] * 3 for _ in range(3)]
    for a in range(3):
        dim = 3 - a
        n = w.shape[1 + dim]
        t1, t2 = (a + 1) % 3, (a + 2) % 3
        words = [0, 1, 2 + a, 2 + t1, 2 + t2]
        lr = [_faces(w[k], a, kinds[2 * a:2 * a + 2], (k == 2 + a, W_FIX[k]), plm) for k in words]
        if mhd:
            lr += [_faces(bc[t], a, ("per", "per"), (False, 0.0), plm) for t in (t1, t2)]
            bx = torch.cat([b[a], b[a].narrow(dim, 0, 1)], dim=dim)
            f = _hlld([x[0] for x in lr], [x[1] for x in lr], bx, gam, hlle)
            mass[a] = f[0].narrow(dim, 0, n)
            emf[a][t1], emf[a][t2] = f[6].narrow(dim, 0, n), -f[5].narrow(dim, 0, n)
        else:
            f = _hllc([x[0] for x in lr], [x[1] for x in lr], gam)
        d = [None] * 5
        for k, q in zip(words, f):
            d[k] = (q.narrow(dim, 0, n) - q.narrow(dim, 1, n)) / dx[a]
        div = div + torch.stack(d)
        del f, lr, d
    if not mhd:
        return div, None
    edge = []
    for ax in range(3):
        a1, a2 = (ax + 1) % 3, (ax + 2) % 3
        back = lambda q, *axes: functools.reduce(lambda x, s: torch.roll(x, 1, 3 - s), axes, q)  # noqa: E731
        ce = bc[a1] * w[2 + a2] - bc[a2] * w[2 + a1]
        e = 0
        for para, perp in ((a1, a2), (a2, a1)):
            fp = emf[para][ax]
            fm = back(fp, perp)
            rp, rm = mass[perp], back(mass[perp], para)
            dp = torch.where(rp > 0, back(ce, perp) - fm, ce - fp)
            dm = torch.where(rm > 0, fm - back(ce, a1, a2), fp - back(ce, para))
            e = e + 0.25 * (fm + fp) + 0.25 * (dm - dp)
        edge.append(e)
    return div, edge


def _curl(edge, dx, c):
    a1, a2 = (c + 1) % 3, (c + 2) % 3
    e1, e2 = edge[a1], edge[a2]
    return -((e1 - torch.roll(e1, -1, 3 - a2)) / dx[a2] + (torch.roll(e2, -1, 3 - a1) - e2) / dx[a1])


def _evolve(u, b, steps, gam, kinds, vl2, hlle, boxes):
    dx = [1.0 / u.shape[4 - a] for a in range(3)]
    t = torch.zeros(u.shape[1] if boxes else 1, device=DEV, dtype=torch.float64).view(-1, 1, 1, 1)
    dt = None
    for _ in range(steps):
        w, bc, u = _prims(u, b, gam)
        bound = None if dt is None else 2 * dt
        dt = _time_step(w, b, bc, dx, gam, boxes)
        dt = dt if bound is None else torch.minimum(dt, bound)
        d, e = _rates(w, b, bc, dx, gam, kinds, not vl2, hlle)
        h = dt / 2 if vl2 else dt
        u1 = u + h * d
        b1 = None if b is None else torch.stack([b[c] + h * _curl(e, dx, c) for c in range(3)])
        del d, e, w, bc
        w, bc, u1 = _prims(u1, b1, gam)
        d, e = _rates(w, b1, bc, dx, gam, kinds, True, hlle)
        h = dt if vl2 else dt / 2
        u = (u if vl2 else (u + u1) / 2) + h * d
        if b is not None:
            b = torch.stack([(b[c] if vl2 else (b[c] + b1[c]) / 2) + h * _curl(e, dx, c) for c in range(3)])
        t = t + dt
    return u, b, t.reshape(-1), dt.reshape(-1)


def exact(case, seed):
    """None for refined meshes: their exchange across level jumps, block by block in plain torch, takes minutes.
    The learned selector's result is compared with the one of every face on HLLD, which it approximates."""
    if case["kind"] == "refined":
        return None
    if case["kind"] == "boxes":
        sizes = _box_sizes(case["boxes"])
        g = _gen(seed)
        out = {}
        t, dt = np.empty(len(sizes)), np.empty(len(sizes))
        for n in sorted(set(sizes)):
            ids = [k for k, s in enumerate(sizes) if s == n]
            u, b = _flow_boxes(n, len(ids), g)
            u, b, tn, dn = _evolve(u, b, case["steps"], GAMMA_MHD, ("per",) * 6, False, case["riemann"] == 1, True)
            faces = [torch.cat([b[a], b[a].narrow(3 - a, 0, 1)], dim=3 - a) for a in range(3)]
            out["n%d" % n] = [_host_u(u, faces)] + faces
            t[ids], dt[ids] = tn.cpu().numpy(), dn.cpu().numpy()
        return {"state": out, "t": t, "dt": dt}
    nb, n = _dims(case)
    u, b = _initial(case, seed)
    u, b, t, dt = _evolve(u, b, case["steps"], GAMMA_MHD if case["mhd"] else GAMMA_HYDRO, _kinds(case),
                          case["integrator"] == 1, case["riemann"] == 1, False)
    u = torch.stack([_to_blocks(q[0], nb, n) for q in u])
    faces = [_to_blocks(b[a][0], nb, n, 1, a) for a in range(3)] if case["mhd"] else []
    return {"state": [_host_u(u, faces if case["mhd"] else None)] + faces, "t": float(t), "dt": float(dt)}
