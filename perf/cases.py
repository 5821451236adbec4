"""The workloads this library's speed is measured on, with their inputs and 64-bit results.

    listed()             the cases
    draw(rng)            one more case of the ranges that the listed ones stand for
    prepare(case, seed)  what a program holds before the call: arrays and handles on the GPU
    run(state)           one pass through the public entry points; returns its outputs
    work(case)           bytes and flops that a pass cannot do without
    exact(case, seed)    run()'s outputs in plain 64-bit torch, or None

The kinds of work, all from this repository's own workloads and tests:

    eval      velocities (and gradients) of particles at themselves or at field points: the
              direct sum that a time step, a restart or a plot consists of
    rk2       a Ralston step of a free vortex system, replayed from its graph
    batch     many independent systems in one launch (ensembles, parameter sweeps)
    panpt     a solved body's panels acting on the particles (each stage of a coupled step)
    ptpan     the particles acting on the panels (the right-hand side of the body's system)
    bem       influence matrix of a body assembled and solved, by GMRES (one new body shape)
              or by LU with several right-hand sides (one shape, several flow states)
    coupled   a Ralston step of particles around a body that is solved for at each stage
    remesh    split of the stretched particles, then merge of the close ones
"""
import math
import random

import numpy as np
import torch

import omega3d_gb300 as G
from omega3d_gb300 import workloads as W
from omega3d_gb300.influence import device_matrix_view

DEV = "cuda"
DT = 0.01
FS = (1.0, 0.0, 0.0)
PAIR_FLOPS = {"rm": 63, "wl": 70, "exp": 68, "gauss": 69, "v2": 67}      # with gradients, with target radius
PAIR_FLOPS_V = {"rm": 31, "wl": 36, "exp": 40, "gauss": 40, "v2": 35}    # velocities only


def listed():
    return [
        # the smallest calls: one eddy or a start-up ring, where launches and latency count
        dict(name="eval_ring_1000", kind="eval", scene="ring", core="rm", prec="plain", ns=1000, nt=0, grads=True),
        # a plot or a tracer set: velocities only, at field points, with the reference's default core
        dict(name="eval_field_wl", kind="eval", scene="cloud", core="wl", prec="plain", ns=50021, nt=19683,
             grads=False),
        # the benchmark's precision cloud
        dict(name="eval_cloud_gauss", kind="eval", scene="cloud", core="gauss", prec="compensated", ns=262144, nt=0,
             grads=True),
        # the accuracy option: every target to 1e-6
        dict(name="eval_cloud_accurate", kind="eval", scene="cloud", core="gauss", prec="accurate", ns=30011, nt=0,
             grads=True),
        # the benchmark's vortex ring, one time step
        dict(name="rk2_ring", kind="rk2", core="rm", prec="plain", n=16384),
        # the benchmark's ensemble of uneven systems with field points
        dict(name="batch_64", kind="batch", core="gauss", prec="compensated", nsys=64, nmin=1024, nmax=65536,
             nfield=4096),
        # a sphere's panels on the wake, and the wake on a finer sphere's panels
        dict(name="panels_to_points", kind="panpt", level=4, nunk=2, prec="compensated", nt=262144, grads=True),
        dict(name="points_to_panels", kind="ptpan", level=5, prec="plain", ns=100000),
        # the benchmark's body: a new shape, solved once
        dict(name="bem_gmres", kind="bem", level=5, nunk=2, method="gmres", nrhs=1),
        # a body that several flow states are solved for
        dict(name="bem_lu", kind="bem", level=4, nunk=2, method="lu", nrhs=2),
        # body and wake together, one time step
        dict(name="coupled_step", kind="coupled", level=3, nunk=2, prec="compensated", n=65536),
        # the particle set's upkeep between steps
        dict(name="split_merge", kind="remesh", k=80),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "rk2", "batch", "panpt", "ptpan", "bem", "coupled", "remesh"])
    if kind == "eval":
        prec = rng.choice(["plain", "plain", "compensated", "compensated", "accurate"])
        core = rng.choice(["rm", "gauss"] if prec == "accurate" else ["rm", "wl", "exp", "gauss", "v2"])
        top = 200000 if prec != "accurate" and core != "exp" else 65536
        ns = _log_int(rng, 500, top)
        nt = rng.choice([0, 0, _log_int(rng, 500, top)])
        return dict(kind=kind, scene=rng.choice(["ring", "cloud"]), core=core, prec=prec, ns=ns, nt=nt,
                    grads=rng.random() < 0.7)
    if kind == "rk2":
        return dict(kind=kind, core=rng.choice(["rm", "wl", "gauss"]), prec=rng.choice(["plain", "compensated"]),
                    n=_log_int(rng, 1000, 65536))
    if kind == "batch":
        nsys = _log_int(rng, 4, 64)
        return dict(kind=kind, core=rng.choice(["rm", "wl", "gauss"]), prec=rng.choice(["plain", "compensated"]),
                    nsys=nsys, nmin=_log_int(rng, 500, 1024), nmax=_log_int(rng, 8000, 65536),
                    nfield=rng.choice([512, 1728, 4096]))
    if kind == "panpt":
        return dict(kind=kind, level=rng.randint(2, 4), nunk=rng.choice([2, 3]),
                    prec=rng.choice(["plain", "compensated"]), nt=_log_int(rng, 2000, 262144),
                    grads=rng.random() < 0.7)
    if kind == "ptpan":
        return dict(kind=kind, level=rng.randint(2, 5), prec=rng.choice(["plain", "compensated"]),
                    ns=_log_int(rng, 2000, 100000))
    if kind == "bem":
        method = rng.choice(["gmres", "lu"])
        nunk = rng.choice([2, 3])
        return dict(kind=kind, level=rng.randint(2, 5 if method == "gmres" and nunk == 2 else 4), nunk=nunk,
                    method=method, nrhs=rng.choice([1, 2]))
    if kind == "coupled":
        return dict(kind=kind, level=rng.randint(2, 3), nunk=rng.choice([2, 3]),
                    prec=rng.choice(["plain", "compensated"]), n=_log_int(rng, 2000, 65536))
    return dict(kind=kind, k=rng.randint(16, 80))


# ---------------------------------------------------------------------------------------
# inputs

def _dev(*arrays):
    out = tuple(torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in arrays)
    return out if len(out) > 1 else out[0]


def _scene(case, seed):
    if case["scene"] == "ring":
        return W.vortex_ring(case["ns"], seed=seed)
    return W.gaussian_cloud(case["ns"], seed=seed)


def _field_points(n, seed):
    # the first n points of a jittered grid over the particles' region
    rng = np.random.default_rng(seed + 7001)
    side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    g = np.linspace(-1.0, 1.0, side)
    f = np.stack(np.meshgrid(g, g, g, indexing="ij")).reshape(3, -1)[:, :n]
    return (f + rng.uniform(-0.3, 0.3, f.shape) * (2.0 / side)).astype(np.float32)


def _batch_sizes(case):
    # the sizes belong to the case, as a program's systems keep theirs; inputs follow the seed
    rng = random.Random(case["nsys"] * 1000003 + case["nmin"] * 101 + case["nmax"])
    return [_log_int(rng, case["nmin"], case["nmax"]) for _ in range(case["nsys"])]


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    side = int(round(case["nfield"] ** (1.0 / 3.0)))
    out = []
    for n in _batch_sizes(case):
        sb = rng.uniform(0.1, 0.5)
        x = rng.normal(0.0, sb, (3, n))
        s = rng.normal(0.0, 1e-3, (3, n))
        r = rng.uniform(0.01, 0.05, n)
        g = np.linspace(-2 * sb, 2 * sb, side)
        f = np.stack(np.meshgrid(g, g, g, indexing="ij")).reshape(3, -1)
        f = f + rng.uniform(-0.25, 0.25, f.shape) * (g[1] - g[0])
        out.append(tuple(a.astype(np.float32) for a in (x, s, r, f)))
    return out


def _sphere(level, nunk=2):
    nodes, idx = G.generate_ovoid(level, 2.0, 2.0, 2.0)
    return G.Surfaces(nodes, idx, nunk=nunk)


def _sheet(npan, nunk, seed):
    rng = np.random.default_rng(seed + 31)
    return rng.normal(0.0, 1.0, (nunk, npan)).astype(np.float32)


def _around_sphere(n, seed):
    # half near the body, half in the wake behind it; none within a cutoff layer of the surface
    h = n // 2
    a = W.shell_particles(h, seed=seed, rin=1.04, rout=1.6)
    b = W.wake_particles(n - h, seed=seed + 1, xmin=1.1, xmax=5.0)
    return tuple(np.concatenate([p, q], axis=-1) for p, q in zip(a, b))


def _free_streams(nrhs, seed):
    rng = np.random.default_rng(seed + 17)
    v = rng.normal(size=(nrhs, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _rhs(surf, streams):
    rows = [surf.x1, surf.x2] + ([surf.norm] if surf.nunk == 3 else [])
    b = np.empty((len(streams), surf.npanels * surf.nunk), np.float32)
    for m, v in enumerate(streams):
        for l, e in enumerate(rows):
            b[m, l::surf.nunk] = -(v[0] * e[0] + v[1] * e[1] + v[2] * e[2])
    return b


class _State:
    def __init__(self, case):
        self.case = case


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    if kind == "eval":
        x, s, r = _dev(*_scene(case, seed))
        st.src = G.Points(x, s, r, grads=case["grads"])
        st.targ = st.src if case["nt"] == 0 else G.Points(_dev(_field_points(case["nt"], seed)), inert=True,
                                                          grads=case["grads"])
        st.rest = G.ResultsType("velandgrad" if case["grads"] else "velonly")
        st.env = G.ExecEnv(case["core"], case["prec"])
    elif kind in ("rk2", "coupled"):
        if kind == "rk2":
            x, s, r = W.vortex_ring(case["n"], seed=seed)
        else:
            x, s, r = _around_sphere(case["n"], seed)
        st.x0, st.s0, r = _dev(x, s, r)
        st.e0 = torch.ones(case["n"], device=DEV)
        st.x, st.s, st.e = st.x0.clone(), st.s0.clone(), st.e0.clone()
        st.rk = G.Ralston(st.x, st.s, r, st.e, env=G.ExecEnv(case.get("core", "rm"), case["prec"]))
        if kind == "coupled":
            surf = _sphere(case["level"], case["nunk"])
            st.bem = G.BEM(surf.npanels * case["nunk"])
            st.rk.attach_body(surf, st.bem, ips=0.02)
        st.dt, st.fs = (DT, (0.0, 0.0, 0.0)) if kind == "rk2" else (0.005, FS)
        # the combined velocity of the step, in the handle's own memory
        u, _ = st.rk.velocities()
        st.u = device_matrix_view(u[0], (u[1] - u[0]) // 4, case["n"], 3)
    elif kind == "batch":
        data = _batch_inputs(case, seed)
        # all results in one block, so that one memset clears them
        sizes = [(x.shape[1], f.shape[1]) for x, _, _, f in data]
        st.out = torch.zeros(sum(12 * (a + b) for a, b in sizes), device=DEV)
        systems, at = [], 0

        def take(k, n):
            nonlocal at
            at += k * n
            return st.out[at - k * n:at].view(k, n)

        for x, s, r, f in data:
            x, s, r, f = _dev(x, s, r, f)
            n, m = x.shape[1], f.shape[1]
            systems.append(G.BatchSystem(x, s, r, take(3, n), take(9, n), f, take(3, m), take(9, m)))
        st.batch = G.Batch(systems, G.ExecEnv(case["core"], case["prec"]))
        # a fixed configuration: the sums then round alike from run to run
        st.batch.set_config(1 if case["prec"] == "compensated" else 2, 0, 4)
    elif kind in ("panpt", "ptpan"):
        st.surf = _sphere(case["level"], case.get("nunk", 2))
        st.env = G.ExecEnv("rm", case["prec"])
        if kind == "panpt":
            st.surf.set_sheet_strengths(*_sheet(st.surf.npanels, case["nunk"], seed))
            x, _, _ = _around_sphere(case["nt"], seed)
            st.targ = G.Points(_dev(x), inert=True, grads=case["grads"])
            st.rest = G.ResultsType("velandgrad" if case["grads"] else "velonly")
        else:
            st.src = G.Points(*_dev(*W.shell_particles(case["ns"], seed=seed)), grads=False)
            st.pu = torch.zeros(3, st.surf.npanels, device=DEV)
        st.arr = st.surf.device_arrays(DEV)
    elif kind == "bem":
        st.surf = _sphere(case["level"], case["nunk"])
        st.arr = st.surf.device_arrays(DEV)
        st.b = _dev(_rhs(st.surf, _free_streams(case["nrhs"], seed)))
        st.bem = G.BEM(st.surf.npanels * case["nunk"])
    else:
        x, s, r, _ = W.lattice_particles(k=case["k"], seed=seed)
        # the same elongations in another order for each seed: the number that split is the case's
        n = r.shape[0]
        e = 1.0 - 0.12 * np.log(1.0 - (np.arange(n) + 0.5) / n)
        st.parts = _dev(x, s, r, np.random.default_rng(seed + 5).permutation(e).astype(np.float32))
    return st


# ---------------------------------------------------------------------------------------
# one pass

def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "eval":
        st.targ.zero_vels()
        G.points_affect_points(st.src, st.targ, st.rest, st.env)
        return (st.targ.u, st.targ.ug) if case["grads"] else (st.targ.u,)
    if kind in ("rk2", "coupled"):
        # each pass is the step from the saved state
        st.x.copy_(st.x0)
        st.s.copy_(st.s0)
        st.e.copy_(st.e0)
        st.rk.step(st.dt, st.fs)
        return st.x, st.s, st.e, st.u.clone()     # the handle's memory ends with it
    if kind == "batch":
        st.out.zero_()
        st.batch.run()
        return st.out
    if kind == "panpt":
        st.targ.zero_vels()
        G.panels_affect_points(st.surf, st.targ, st.rest, st.env, arrays=st.arr)
        return (st.targ.u, st.targ.ug) if case["grads"] else (st.targ.u,)
    if kind == "ptpan":
        st.pu.zero_()
        G.points_affect_panels(st.src, st.surf, st.env, arrays=st.arr, pu=st.pu)
        return st.pu
    if kind == "bem":
        st.bem.assemble(st.arr, st.arr, case["nunk"], True)
        if case["nrhs"] == 1:
            return st.bem.solve(st.b[0], tol=1e-10, max_iter=300 if case["method"] == "gmres" else 30,
                                method=case["method"])
        return st.bem.solve_many(st.b, tol=1e-10, max_iter=300 if case["method"] == "gmres" else 30,
                                 method=case["method"])
    x, s, r, e, nsplit = G.split_elongated(*st.parts)
    n = r.shape[0]
    x, s, r, nmerged = G.merge_close_particles(x, s, r)
    # back into arrays of the program's own capacity
    out = torch.zeros(7, n, device=DEV)
    out[:3, :n - nmerged] = x
    out[3:6, :n - nmerged] = s
    out[6, :n - nmerged] = r
    return out, e, nsplit, nmerged


# ---------------------------------------------------------------------------------------
# what a pass cannot do without

def _npanels(level):
    return 20 * 4 ** level


def work(case):
    kind = case["kind"]
    if kind == "eval":
        nt = case["nt"] or case["ns"]
        f = (PAIR_FLOPS if case["grads"] else PAIR_FLOPS_V)[case["core"]]
        return {"bytes": 28 * case["ns"] + (12 * nt if case["nt"] else 0) + (48 if case["grads"] else 12) * nt,
                "flops": (f * case["ns"] + 12) * nt}
    if kind == "rk2":
        n = case["n"]
        return {"bytes": 32 * n + 40 * n, "flops": 2 * PAIR_FLOPS[case["core"]] * n * n}
    if kind == "batch":
        sizes, m = _batch_sizes(case), case["nfield"]
        return {"bytes": sum(28 * n + 12 * m + 48 * (n + m) for n in sizes),
                "flops": PAIR_FLOPS[case["core"]] * sum(n * (n + m) for n in sizes)}
    if kind == "panpt":
        np_, nt = _npanels(case["level"]), case["nt"]
        return {"bytes": 64 * np_ + 12 * nt + (48 if case["grads"] else 12) * nt,
                "flops": (70 if case["grads"] else 31) * np_ * nt}
    if kind == "ptpan":
        np_, ns = _npanels(case["level"]), case["ns"]
        return {"bytes": 64 * np_ + 24 * ns + 12 * np_, "flops": 31 * np_ * ns}
    if kind == "bem":
        n = _npanels(case["level"]) * case["nunk"]
        if case["method"] == "gmres":
            # the matrix written once and read for at least one product per right-hand side
            return {"bytes": 4.0 * n * n * 2, "flops": 2.0 * n * n * case["nrhs"]}
        return {"bytes": 4.0 * n * n * 4, "flops": 2.0 / 3.0 * n ** 3 + 4.0 * n * n * case["nrhs"]}
    if kind == "coupled":
        n, np_ = case["n"], _npanels(case["level"])
        return {"bytes": 72 * n + 64 * np_, "flops": 2 * (PAIR_FLOPS["rm"] * n + 101 * np_) * n}
    n = case["k"] ** 3
    return {"bytes": 2 * 32 * n, "flops": 300 * n}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch

FOUR_PI = 4.0 * math.pi


def _t64(a):
    return torch.as_tensor(np.asarray(a), device=DEV if torch.cuda.is_available() else "cpu").double()


def _core_factors(core, d2, s, t, grads):
    """r3 and bbb of all pairs from the squared distances d2[nt, ns] and radii s[1, ns], t[nt, 1]."""
    if core == "rm":
        r2 = d2 + (s * s + t * t)
        rs = r2.rsqrt()
        r3 = rs * rs * rs
        return r3, (-3.0 * r3 * rs * rs if grads else None)
    if core == "wl":
        c = s * s + t * t
        rs2 = 1.0 / (d2 + c)
        dn5 = rs2 * rs2 * rs2.sqrt()
        r3 = (d2 + 2.5 * c) * dn5
        return r3, (2.0 * dn5 - 5.0 * r3 * rs2 if grads else None)
    if core == "v2":
        rs = (d2 * d2 + (s ** 4 + t ** 4)).rsqrt()
        r3 = rs * rs.sqrt()
        return r3, (-3.0 * r3 * rs if grads else None)
    if core == "exp":
        cf = 1.0 / (s ** 3 + t ** 3)
        d = d2.sqrt()
        x = d2 * d * cf
        near, far = x < float(np.float32(0.001)), x > 16.0
        inv = 1.0 / torch.where(near, torch.ones_like(d), d2 * d)
        em1 = torch.expm1(-x)
        r3 = torch.where(near, cf.expand_as(x), torch.where(far, inv, -inv * em1))
        if not grads:
            return r3, None
        b = torch.where(far, -3.0 * r3, 3.0 * (cf * (em1 + 1.0) - r3)) / torch.where(near, torch.ones_like(d), d2)
        return r3, torch.where(near, -1.5 * d * r3 * r3, b)
    # Gaussian: the singular kernel, replaced where the core reaches
    c = s * s + t * t
    rs = d2.rsqrt()
    r3 = rs * rs * rs
    bbb = -3.0 * r3 * rs * rs if grads else None
    at = (d2 < 90.0 * c).reshape(-1).nonzero().squeeze(1)
    if at.numel():
        cc = c.expand_as(d2).reshape(-1)[at]
        q = d2.reshape(-1)[at] / cc
        a = math.sqrt(2.0 / math.pi)
        small = q < 0.5
        qs = torch.where(small, q, torch.zeros_like(q))
        g, gp = torch.zeros_like(q), torch.zeros_like(q)
        for n in range(14, 0, -1):
            cn = (-1.0) ** (n + 1) / ((2 * n + 1) * 2.0 ** (n - 1) * math.factorial(n - 1))
            g = g * qs + cn
            if n >= 2:
                gp = gp * qs + (n - 1) * cn
        ql = torch.where(small, torch.ones_like(q), q)
        rho = ql.sqrt()
        e = torch.exp(-0.5 * ql)
        gl = (torch.erf(rho / math.sqrt(2.0)) - a * rho * e) / (ql * rho)
        r3.reshape(-1)[at] = torch.where(small, a * g, gl) * cc ** -1.5
        if grads:
            dl = (a * e - 3.0 * gl) / ql
            bbb.reshape(-1)[at] = torch.where(small, 2.0 * a * gp, dl) * cc ** -2.5
    return r3, bbb


def _pair_sums(x, s, r, tx, tr, core, grads):
    """u[3, nt] (and ug[9, nt]): sums over sources of r3 s x d and its gradient, with the
    target's coordinates taken out of the sums so that they are matrix products."""
    ns, nt = x.shape[1], tx.shape[1]
    p = torch.linalg.cross(x, s, dim=0)
    cols3 = torch.cat([s, p]).t().contiguous()                                    # s, x x s
    cols5 = torch.cat([s, p, (x[:, None] * s[None]).reshape(9, ns),
                       (x[:, None] * p[None]).reshape(9, ns)]).t().contiguous()
    x2 = (x * x).sum(0)[None]
    u = torch.empty(3, nt, dtype=torch.float64, device=x.device)
    ug = torch.empty(9, nt, dtype=torch.float64, device=x.device) if grads else None
    step = max(1, (1 << 27) // ns)
    for a in range(0, nt, step):
        t = tx[:, a:a + step]
        # coincident points: the expanded square can round below zero
        d2 = ((t * t).sum(0)[:, None] + x2 - 2.0 * (t.t() @ x)).clamp_(min=1e-300)
        r3, bbb = _core_factors(core, d2, r[None], torch.zeros(t.shape[1], 1, dtype=torch.float64, device=x.device)
                                if tr is None else tr[a:a + step, None], grads)
        m3 = (r3 @ cols3).t()
        A, B = m3[:3], m3[3:]
        u[:, a:a + step] = torch.linalg.cross(A, t, dim=0) + B
        if grads:
            m5 = (bbb @ cols5).t()
            S, P, M, Q = m5[:3], m5[3:6], m5[6:15].reshape(3, 3, -1), m5[15:].reshape(3, 3, -1)
            g = t[:, None] * (torch.linalg.cross(S, t, dim=0) + P)[None]
            for i in range(3):
                g[i] -= torch.linalg.cross(M[i], t, dim=0) + Q[i]
            g[0, 1] += A[2]
            g[0, 2] -= A[1]
            g[1, 0] -= A[2]
            g[1, 2] += A[0]
            g[2, 0] += A[1]
            g[2, 1] -= A[0]
            ug[:, a:a + step] = g.reshape(9, -1)
    return u, ug


def _tri(surf):
    v = surf.x[:, surf.idx.reshape(-1, 3).astype(np.int64)]      # [3 components, panel, corner]
    return _t64(v).permute(1, 2, 0).contiguous()                # [panel, corner, component]


def _children(t):
    a, b, c = t[:, 0], t[:, 1], t[:, 2]
    ab, ac, bc = 0.5 * (a + b), 0.5 * (a + c), 0.5 * (b + c)
    return torch.stack([torch.stack(v, 1) for v in ((a, ab, ac), (ab, b, bc), (ab, bc, ac), (ac, bc, c))], 1)


def _leaf_rows(d, s, q, grads):
    """[m, 3 or 12]: velocity (and gradient) of singular vortex + source points, one per row."""
    d2 = (d * d).sum(1, keepdim=True)
    r3 = d2 ** -1.5
    c = torch.linalg.cross(s, d, dim=1)
    if q is not None:
        c = c + q * d
    if not grads:
        return r3 * c
    g = d[:, :, None] * (-3.0 * r3 / d2 * c)[:, None, :]
    a = r3 * s
    if q is not None:
        g = g + (q * r3)[:, :, None] * torch.eye(3, dtype=d.dtype, device=d.device)
    g[:, 0, 1] += a[:, 2]
    g[:, 0, 2] -= a[:, 1]
    g[:, 1, 0] -= a[:, 2]
    g[:, 1, 2] += a[:, 0]
    g[:, 2, 0] += a[:, 1]
    g[:, 2, 1] -= a[:, 0]
    return torch.cat([r3 * c, g.reshape(-1, 9)], 1)


def _panel_sums(tri, area, strength, src, pts, grads, on_panels, maxlev=3):
    """Panels acting on points: strength[panel, 3] (and src[panel, 1]), sums [point, 3 or 12].
    With on_panels the points carry the strength and the sums are the panels'."""
    np_, n, nc = tri.shape[0], pts.shape[0], 12 if grads else 3
    out = torch.zeros(np_ if on_panels else n, nc, dtype=torch.float64, device=tri.device)
    cen, reach = tri.mean(1), 4.0 * area.sqrt()
    step = max(1, (1 << 20) // np_) if not on_panels else max(1, (1 << 21) // np_)
    for a in range(0, n, step):
        p = pts[a:a + step]
        m = p.shape[0]
        d = p[:, None] - cen[None]
        dist = d.norm(dim=2)
        sv = strength[a:a + step, None].expand(m, np_, 3) if on_panels else strength[None].expand(m, np_, 3)
        q = None if src is None else src[None].expand(m, np_, 1).reshape(-1, 1)
        rows = _leaf_rows(d.reshape(-1, 3), sv.reshape(-1, 3), q, grads).reshape(m, np_, nc)
        near = (dist <= reach[None]).nonzero()
        rows[near[:, 0], near[:, 1]] = 0.0
        if on_panels:
            out += rows.sum(0)
        else:
            out[a:a + step] += rows.sum(1)
        ti, pj = near[:, 0] + a, near[:, 1]
        sub, lev = tri[pj], 0
        while ti.numel() and lev < maxlev:
            lev += 1
            sub = _children(sub).reshape(-1, 3, 3)
            ti, pj = ti.repeat_interleave(4), pj.repeat_interleave(4)
            d = pts[ti] - sub.mean(1)
            leaf = torch.ones_like(ti, dtype=torch.bool) if lev == maxlev else \
                d.norm(dim=1) > reach[pj] * 0.5 ** lev
            f = 0.25 ** lev
            to = (pj if on_panels else ti)[leaf]
            out.index_add_(0, to, _leaf_rows(d[leaf], f * strength[ti if on_panels else pj][leaf],
                                             None if src is None else f * src[pj][leaf], grads))
            ti, pj, sub = ti[~leaf], pj[~leaf], sub[~leaf]
    return out


def _coeff(surf):
    """The influence matrix [rows, columns] of the surface on itself."""
    nunk, np_ = surf.nunk, surf.npanels
    tri, area = _tri(surf), _t64(surf.area)
    b = torch.stack([_t64(v).t() for v in (surf.x1, surf.x2, surf.norm)[:nunk]], 1)     # [panel, unknown, 3]
    s = b * area[:, None, None]
    cen, reach = tri.mean(1), 4.0 * area.sqrt()
    A = torch.empty(np_, nunk, np_, nunk, dtype=torch.float64, device=tri.device)

    def project(d, js, is_, f):
        # unit strengths of the source panels js at separations d, on the bases of is_
        w = (f * (d * d).sum(1) ** -1.5)[:, None]
        u = [torch.linalg.cross(s[js, k], d, dim=1) * w for k in range(2)]
        if nunk == 3:
            u.append(area[js, None] * d * w)
        u = torch.stack(u, 1)                                       # [pair, source unknown, 3]
        return torch.einsum("mkc,mlc->mlk", u, b[is_])              # [pair, target unknown, source unknown]

    step = max(1, (1 << 21) // np_)
    every = torch.arange(np_, device=tri.device)
    for a in range(0, np_, step):
        i = every[a:a + step]
        m = i.numel()
        ti, pj = i.repeat_interleave(np_), every.repeat(m)
        d = cen[ti] - cen[pj]
        near = (d.norm(dim=1) <= reach[ti] + reach[pj]) & (ti != pj)
        d[ti == pj] = 1.0
        A[a:a + step] = project(d, pj, ti, 1.0).reshape(m, np_, nunk, nunk).permute(0, 2, 1, 3)
        ti, pj = ti[near], pj[near]
        for c0 in range(0, ti.numel(), 20000):
            bi, bj = ti[c0:c0 + 20000], pj[c0:c0 + 20000]
            own = torch.arange(bi.numel(), device=tri.device)
            v = torch.zeros(bi.numel(), nunk, nunk, dtype=torch.float64, device=tri.device)
            st, tt = tri[bj], tri[bi]
            for lev in (1, 2, 3):
                own = own.repeat_interleave(16)
                st = _children(st)[:, :, None].expand(-1, 4, 4, 3, 3).reshape(-1, 3, 3)
                tt = _children(tt)[:, None].expand(-1, 4, 4, 3, 3).reshape(-1, 3, 3)
                d = tt.mean(1) - st.mean(1)
                leaf = torch.ones_like(own, dtype=torch.bool) if lev == 3 else \
                    d.norm(dim=1) > (reach[bi[own]] + reach[bj[own]]) * 0.5 ** lev
                v.index_add_(0, own[leaf], project(d[leaf], bj[own[leaf]], bi[own[leaf]], 0.0625 ** lev))
                own, st, tt = own[~leaf], st[~leaf], tt[~leaf]
            A[bi, :, bj] = v
    A[every, :, every] = 0.0
    A[every, 1, every, 0] = 2.0 * math.pi
    A[every, 0, every, 1] = -2.0 * math.pi
    if nunk == 3:
        A[every, 2, every, 2] = 2.0 * math.pi
    return A.reshape(np_ * nunk, np_ * nunk).mul_(1.0 / FOUR_PI)


def _solve(A, b):
    """A x = b in 64 bits: direct when small, else restarted GMRES to 1e-13."""
    if A.shape[0] <= 8192:
        return torch.linalg.solve(A, b)
    x = torch.zeros_like(b)
    for _ in range(20):
        r = b - A @ x
        beta = r.norm()
        if beta <= 1e-13 * b.norm():
            break
        V, H = [r / beta], torch.zeros(41, 40, dtype=torch.float64)
        for k in range(40):
            w = A @ V[k]
            for _ in range(2):
                for j, v in enumerate(V):
                    h = torch.dot(v, w)
                    w = w - h * v
                    H[j, k] += h.cpu()
            H[k + 1, k] = w.norm().cpu()
            V.append(w / w.norm())
        e = torch.zeros(41, 1, dtype=torch.float64)
        e[0] = beta.cpu()
        y = torch.linalg.lstsq(H, e).solution.squeeze(1)
        x = x + torch.stack(V[:40], 1) @ y.to(b.device)
    return x


def _ralston(derivs, x, s, dt):
    def s_dot_g(v, g):
        return torch.einsum("in,ikn->kn", v, g.reshape(3, 3, -1))

    e = torch.ones(x.shape[1], dtype=torch.float64, device=x.device)
    u1, g1 = derivs(x, s)
    h = 2.0 / 3.0 * dt
    u2, g2 = derivs(x + h * u1, s + h * s_dot_g(s, g1))
    u = 0.25 * u1 + 0.75 * u2
    w = 0.25 * s_dot_g(s, g1) + 0.75 * s_dot_g(s, g2)
    return x + dt * u, s + dt * w, e * (1.0 + dt * (s * w).sum(0) / (s * s).sum(0)), u


def exact(case, seed):
    kind = case["kind"]
    if kind == "eval":
        x, s, r = (_t64(a) for a in _scene(case, seed))
        tx, tr = (_t64(_field_points(case["nt"], seed)), None) if case["nt"] else (x, r)
        out = _pair_sums(x, s, r, tx, tr, case["core"], case["grads"])
        return out if case["grads"] else out[:1]
    if kind == "rk2":
        x, s, r = (_t64(a) for a in W.vortex_ring(case["n"], seed=seed))

        def derivs(x, s):
            u, g = _pair_sums(x, s, r, x, r, case["core"], True)
            return u / FOUR_PI, g / FOUR_PI
        return _ralston(derivs, x, s, DT)
    if kind == "batch":
        out = []
        for x, s, r, f in _batch_inputs(case, seed):
            x, s, r, f = (_t64(a) for a in (x, s, r, f))
            for t, tr in ((x, r), (f, None)):
                out += [v.reshape(-1) for v in _pair_sums(x, s, r, t, tr, case["core"], True)]
        return torch.cat(out)
    if kind == "panpt":
        surf = _sphere(case["level"], case["nunk"])
        ps = _t64(_sheet(surf.npanels, case["nunk"], seed))
        area = _t64(surf.area)
        ts = ((ps[0] * _t64(surf.x1) + ps[1] * _t64(surf.x2)) * area).t()
        src = (ps[2] * area)[:, None] if case["nunk"] == 3 else None
        x, _, _ = _around_sphere(case["nt"], seed)
        o = _panel_sums(_tri(surf), area, ts, src, _t64(x).t().contiguous(), case["grads"], False).t()
        return (o[:3], o[3:]) if case["grads"] else (o,)
    if kind == "ptpan":
        surf = _sphere(case["level"])
        x, s, _ = W.shell_particles(case["ns"], seed=seed)
        return -_panel_sums(_tri(surf), _t64(surf.area), _t64(s).t().contiguous(), None, _t64(x).t().contiguous(),
                            False, True).t()
    if kind == "bem":
        surf = _sphere(case["level"], case["nunk"])
        A = _coeff(surf)
        x = [_solve(A, _t64(b)) for b in _rhs(surf, _free_streams(case["nrhs"], seed))]
        return x[0] if case["nrhs"] == 1 else torch.stack(x)
    if kind == "coupled":
        surf = _sphere(case["level"], case["nunk"])
        nunk = case["nunk"]
        lu = torch.linalg.lu_factor(_coeff(surf))
        tri, area = _tri(surf), _t64(surf.area)
        b = [_t64(v) for v in (surf.x1, surf.x2, surf.norm)[:nunk]]
        x, s, r = (_t64(a) for a in _around_sphere(case["n"], seed))
        fs = _t64(FS)[:, None]

        def derivs(x, s):
            pts = x.t().contiguous()
            pu = fs - _panel_sums(tri, area, s.t().contiguous(), None, pts, False, True).t() / FOUR_PI
            rhs = torch.stack([-(pu * v).sum(0) for v in b], 1).reshape(-1, 1)
            y = torch.linalg.lu_solve(*lu, rhs).reshape(-1, nunk)
            ts = ((y[:, 0] * b[0] + y[:, 1] * b[1]) * area).t()
            o = _panel_sums(tri, area, ts, (y[:, 2] * area)[:, None] if nunk == 3 else None, pts, True, False).t()
            u, g = _pair_sums(x, s, r, x, r, "rm", True)
            return fs + (u + o[:3]) / FOUR_PI, (g + o[3:]) / FOUR_PI
        return _ralston(derivs, x, s, 0.005)
    return None         # split and merge decide particle by particle: there is no 64-bit value
