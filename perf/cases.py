"""What a user of this framework has it do, as cases that can be timed: one call (or one step, or
one rollout with its gradient) each, through the public entry points, over the sizes in use.

The kinds:
  box        BoxContactEngine: a pile of random boxes, one macro step of 2 substeps
  boxgrid    BoxContactEngine: a lattice of equal cubes settling under its own weight
  boxbatch   BatchedBoxEngine: many independent piles of uneven size in one engine
  jacobi     RelaxedJacobiContactEngine on bead boxes
  cached     ColorCacheContactEngine on bead boxes
  island     IslandSolveContactEngine on bead boxes
  ncp        NCPSolverB200: the exact-cone sweeps on a resident scene, float32 or float64
  admm       BatchProxADMM: a batch of legged stances, step and both gradients
  bncp       BatchNCP: the same problems in Delassus form, solve and vector-Jacobian product
  rollout    BoxRollout: a differentiable rollout of pushed pyramids, forward and backward

An engine's run() is what a control loop does each tick: put the body state in, step, read the
state back, all on the device.
"""
import math
from importlib import import_module

import numpy as np
import torch

import __graft_entry__ as _entry

_me = _entry.load_package()
_scenes = import_module("motion_engine_b200.scenes")
_badmm = import_module("motion_engine_b200.badmm")
_bncp = import_module("motion_engine_b200.bncp")
_ncp = import_module("motion_engine_b200.ncp")
_world = import_module("motion_engine_b200.world")
_rollout = import_module("motion_engine_b200.rollout")

DT = 1.0 / 240.0
DEV = "cuda"


def listed():
    return [
        # one robot's table top: a few dozen loose boxes, where the step's launches are the time
        {"name": "box_pile_48", "kind": "box", "n": 48, "vit": 16, "pit": 10},
        # the repository's default workload: ten thousand random boxes in one pile
        {"name": "box_pile_10000", "kind": "box", "n": 10000, "vit": 16, "pit": 10},
        # the stress scene: a field of one hundred thousand cubes
        {"name": "box_grid_100000", "kind": "boxgrid", "n": 100000, "vit": 16, "pit": 16},
        # a learner's batch: 160 scenes of 8 to 2000 boxes, 10 % of the boxes 100 times denser
        {"name": "box_batch_160", "kind": "boxbatch", "scenes": 160, "nmin": 8, "nmax": 2000, "vit": 16, "pit": 10},
        # the reference's lattice under relaxed Jacobi, at the size it publishes
        {"name": "jacobi_lattice_10000", "kind": "jacobi", "n": 10000, "vit": 40, "pit": 20},
        # the same lattice under the colour-cached solve
        {"name": "cached_lattice_10000", "kind": "cached", "n": 10000, "vit": 40, "pit": 20},
        # a thousand boxes of the lattice under the island solve
        {"name": "island_lattice_1000", "kind": "island", "n": 1000, "vit": 40, "pit": 10},
        # the reference's exact-cone timing fixture: 40 000 contacts, 40 sweeps, float64
        {"name": "ncp_f64_10000", "kind": "ncp", "n": 10000, "iters": 40, "f64": True},
        # an exact-cone solve of a small scene in float32, 60 sweeps
        {"name": "ncp_f32_600", "kind": "ncp", "n": 600, "iters": 60, "f64": False},
        # the batched ADMM and its adjoint at the reference's benchmark configuration
        {"name": "admm_4096", "kind": "admm", "B": 4096, "nc": 4, "per_leg": 3, "n_iter": 200},
        # the batched exact-cone solve to a residual of 1e-6 and one gradient
        {"name": "bncp_4096", "kind": "bncp", "B": 4096, "nc": 4, "per_leg": 3},
        # learning through contact: 24 pushed pyramids, 4 steps of 2 substeps, forward and backward
        {"name": "rollout_24", "kind": "rollout", "scenes": 24, "steps": 4, "iters": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "boxgrid", "boxbatch", "jacobi", "cached", "island", "ncp", "ncp", "admm", "bncp",
                       "rollout"])
    if kind == "box":
        return {"kind": kind, "n": _log(rng, 24, 10000), "vit": rng.choice([8, 12, 16]), "pit": rng.choice([5, 10])}
    if kind == "boxgrid":
        return {"kind": kind, "n": _log(rng, 1000, 100000), "vit": rng.choice([8, 16]), "pit": rng.choice([8, 16])}
    if kind == "boxbatch":
        return {"kind": kind, "scenes": _log(rng, 8, 160), "nmin": 8, "nmax": _log(rng, 64, 2000),
                "vit": rng.choice([8, 16]), "pit": rng.choice([5, 10])}
    if kind in ("jacobi", "cached"):
        return {"kind": kind, "n": _log(rng, 100, 10000), "vit": rng.choice([20, 40]), "pit": rng.choice([10, 20])}
    if kind == "island":
        return {"kind": kind, "n": _log(rng, 50, 4000), "vit": rng.choice([20, 40]), "pit": rng.choice([10, 20])}
    if kind == "ncp":
        return {"kind": kind, "n": _log(rng, 60, 10000), "iters": rng.randint(20, 40), "f64": rng.random() < 0.5}
    if kind == "admm":
        return {"kind": kind, "B": _log(rng, 50, 4096), "nc": rng.choice([1, 2, 3, 4, 5]),
                "per_leg": rng.choice([3, 4]), "n_iter": rng.randint(80, 200)}
    if kind == "bncp":
        return {"kind": kind, "B": _log(rng, 50, 4096), "nc": rng.choice([1, 2, 3, 4, 6]),
                "per_leg": rng.choice([3, 4])}
    return {"kind": kind, "scenes": _log(rng, 2, 24), "steps": rng.randint(1, 4), "iters": rng.choice([8, 16])}


# ---- inputs -------------------------------------------------------------------------------------

def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _ready_engine(e, before, substeps, seed):
    """Steps the scene until its contacts are those of the working state, and keeps that state,
    each body given a small seeded push, as the input of every pass."""
    for _ in range(before):
        e.step(DT, substeps)
    start = e.state.clone()
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    start[2, :, :3] += 1e-3 * torch.randn(start[2, :, :3].shape, generator=g, device=DEV)
    return {"engine": e, "start": start, "out": torch.empty_like(start), "substeps": substeps}


def _box_scene(case, rng):
    if case["kind"] == "boxgrid":
        n = case["n"]
        side = 50.0 * math.sqrt(n / 1e5)
        return _scenes.box_lattice(n=n, extent=(max(side, 2.0), max(side, 2.0), 10.0), seed=int(rng.integers(1 << 30)))
    return _scenes.jittered_boxes(case["n"], height=10.0 if case["n"] >= 1000 else 2.5, rng=rng)


def _stance(case, seed):
    return _scenes.stance_batch(B=case["B"], nv=6 + case["nc"] * case["per_leg"], nc=case["nc"], mu=0.5, seed=int(seed))


def _ncp_scene(case, seed):
    """The lattice with every body pushed sideways at its own speed, so the cone is in play."""
    d = _scenes.ncp_lattice(n=case["n"])
    rng = np.random.default_rng(seed)
    d["v_free"] = d["v_free"] + rng.normal(0.0, 0.05, d["v_free"].shape)
    d["mu"] = rng.uniform(0.3, 0.8, d["mu"].shape)
    return d


def prepare(case, seed):
    k = case["kind"]
    rng = np.random.default_rng(int(seed))
    if k in ("box", "boxgrid"):
        sc = _box_scene(case, rng)
        e = _me.BoxContactEngine(mu=0.55, vit=case["vit"], pit=case["pit"])
        for c, d, m, de in zip(sc["centers"], sc["dims"], sc["mu"], sc["density"]):
            e.add_box(c, dims=d, density=de, mu=m)
        before = 200 if k == "boxgrid" else 300 if case["n"] >= 1000 else 150
        return _ready_engine(e, before, 2, seed)
    if k == "boxbatch":
        a, b = (int(x) for x in rng.integers(1 << 30, size=2))
        scs = _scenes.batched_scenes(n_scenes=case["scenes"], nmin=case["nmin"], nmax=case["nmax"], seed_mass=a,
                                     seed_boxes=b)
        e = _me.BatchedBoxEngine(scs, mu=0.55, vit=case["vit"], pit=case["pit"])
        return _ready_engine(e, 150, 2, seed)
    if k in ("jacobi", "cached", "island"):
        cls = {"jacobi": _me.RelaxedJacobiContactEngine, "cached": _me.ColorCacheContactEngine,
               "island": _me.IslandSolveContactEngine}[k]
        e = cls(dims=(0.3, 0.3, 0.2), mu=0.5, vit=case["vit"], pit=case["pit"])
        for c in _scenes.lattice(case["n"]):
            j = rng.uniform(-1e-3, 1e-3, 3)
            e.add_body([c[0] + j[0], c[1] + j[1], c[2] + abs(j[2])])
        return _ready_engine(e, 20, 1, seed)
    if k == "ncp":
        d = _ncp_scene(case, seed)
        bs = _ncp.BlockScene(**d)
        s = _ncp.NCPSolverB200(bs.n_b, bs.n_c, dtype="float64" if case["f64"] else "float32")
        s.upload(bs)
        return {"solver": s, "iters": case["iters"]}
    if k == "admm":
        J, Minv, v, mu = _stance(case, seed)
        s = _badmm.BatchProxADMM(case["B"], v.shape[1], case["nc"]).upload(J, Minv, v, mu, DT).set_rho("regime")
        return {"admm": s, "n_iter": case["n_iter"], "n_calls": case["nc"] + 2}
    if k == "bncp":
        J, Minv, v, mu = _stance(case, seed)
        G, b = _bncp.delassus(_dev(J), _dev(Minv), _dev(v))
        seed_dir = _dev(rng.standard_normal(tuple(b.shape)))
        return {"bncp": _bncp.BatchNCP(G, b, _dev(mu)), "seed": seed_dir}
    p = _scenes.pushed_pyramids(n_scenes=case["scenes"], seed_jitter=int(seed), seed_target=int(seed) + 1,
                                seed_v0=int(seed) + 2)
    w = _world.BoxWorldB200(dt=DT, iters=case["iters"], substeps=2, warm_start=True)
    for i in range(len(p["mass"])):
        w.add(p["half"][i], p["mass"][i], p["x"][i], kin=bool(p["kin"][i]), v_kin=p["v_kin"][i], mu=p["mu"][i],
              scene=int(p["scene"][i]))
    return {"rollout": _rollout.BoxRollout(w), "steps": case["steps"], "target": _dev(p["target"]),
            "dyn": _dev(1.0 - p["kin"].astype(np.float64))[:, None], "v0": _dev(p["v0"]), "mu": _dev(p["mu"])}


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    if "engine" in state:
        e = state["engine"]
        e.set_state_packed(state["start"])
        e.step(DT, state["substeps"])
        return {"state": e.get_state_packed(out=state["out"])}
    if "solver" in state:
        s = state["solver"]
        s.solve_resident(state["iters"])
        return {"lam": s.lam[:s.C], "v": s.v}
    if "admm" in state:
        s = state["admm"]
        s.step_and_grad(state["n_iter"], 8, 4, 1e-8, n_calls=state["n_calls"], grad_cg=60)
        return {"lam": s.lam, "u": s.u, "v_plus": s.v_plus, "rho": s.rho, "dlam_tau": s.dlam_tau, "dv_tau": s.dv_tau,
                "dlam_mu": s.dlam_mu, "labels": s.labels, "mask": s.mask}
    if "bncp" in state:
        s = state["bncp"]
        lam = s.solve(5000, 1e-6)
        gb, gmu = s.vjp(state["seed"])
        return {"lam": lam, "gb": gb, "gmu": gmu, "labels": s.labels, "iters": s.iters}
    v0 = state["v0"].clone().requires_grad_(True)
    mu = state["mu"].clone().requires_grad_(True)
    x = _rollout.rollout(state["rollout"], v0, mu, state["steps"])
    loss = (((x - state["target"]) * state["dyn"]) ** 2).sum()
    loss.backward()
    return {"x": x.detach(), "loss": loss.detach(), "v0": v0.grad, "mu": mu.grad}


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    """Bytes: the inputs once and the outputs once.  Operations: those of the method's own
    arithmetic on the contacts that such a scene has."""
    k = case["kind"]
    if k in ("box", "boxgrid", "boxbatch", "jacobi", "cached", "island"):
        if k == "boxbatch":
            lo, hi = case["nmin"], case["nmax"]
            n = int(case["scenes"] * (hi - lo) / math.log(hi / lo)) if hi > lo else case["scenes"] * lo
        else:
            n = case["n"]
        bead = k in ("jacobi", "cached", "island")
        contacts = 8 * n if k == "jacobi" else 4 * n  # 4 a box in the piles and lattices; Jacobi keeps every bead's
        sub = 1 if bead else 2
        # state in and out (64 B each way), mass, inertia, size and friction (68 B), warm impulses (24 B a contact)
        return {"bytes": float(n * (128 + 68) + 2 * 24 * 4 * n),
                "flops": float(sub * contacts * (150 * case["vit"] + 60 * case["pit"]))}
    if k == "ncp":
        n, s = case["n"], 8 if case["f64"] else 4
        c = 4 * n
        return {"bytes": float(c * ((36 + 4 + 3) * s + 12) + n * (36 + 6 + 6) * s + 3 * c * s),
                "flops": float(c * case["iters"] * 260)}
    if k == "admm":
        B, C, nv = case["B"], case["nc"], 6 + case["nc"] * case["per_leg"]
        m = 3 * C
        products = case["n_iter"] * 9 + case["n_iter"] // 4 + 2 * (C + 2) * 61
        return {"bytes": float(8 * B * (m * nv + nv * nv + nv + C + 4 * m + 2 * nv + 1) + 4 * B * (C + 1)),
                "flops": float(B * (products * (2 * m * m + 14 * m) + 2 * m * nv * nv + 2 * m * m * nv))}
    if k == "bncp":
        B, m = case["B"], 3 * case["nc"]
        return {"bytes": float(8 * B * (m * m + 4 * m + 2 * (m // 3)) + 4 * B * (m // 3 + 1)),
                "flops": float(B * (100 * (2 * m * m + 12 * m) + 2 * m * m * m))}
    n = 65 * case["scenes"]
    subs = case["steps"] * 2
    c = 11 * n  # contacts a substep: a box's faces lie within the margin of its neighbours'
    return {"bytes": float(n * 8 * (3 + 1 + 3 + 3 + 1) + 2 * subs * n * 13 * 8),
            "flops": float(subs * c * case["iters"] * (260 + 260 + 700))}


# ---- the same in 64 bits, by plain torch ---------------------------------------------------------

def _proj(z, mu):
    """The friction cone's projection: z (..., 3), mu (...)."""
    zn, zt = z[..., 0], torch.sqrt(z[..., 1] ** 2 + z[..., 2] ** 2)
    s = (zn + mu * zt) / (1 + mu * mu)
    f = mu * s / torch.where(zt > 0, zt, torch.ones_like(zt))
    side = torch.stack([s, f * z[..., 1], f * z[..., 2]], -1)
    inside, below = zt <= mu * zn, mu * zt <= -zn
    return torch.where(inside[..., None], z, torch.where(below[..., None], torch.zeros_like(z), side))


def _blocks(G, nc):
    return torch.stack([G[:, 3 * c:3 * c + 3, 3 * c:3 * c + 3] for c in range(nc)], 1)


def _desaxce(u, mu):
    w = u.clone()
    w[..., 0] += mu * torch.sqrt(u[..., 1] ** 2 + u[..., 2] ** 2)
    return w


def _branches(lam, mu):
    """open 0, stick 1, slip 2 of lam (B, nc, 3)."""
    scale = lam.abs().amax((1, 2), keepdim=True)[..., 0].clamp(min=1e-30)
    ln, lt = lam[..., 0], torch.sqrt(lam[..., 1] ** 2 + lam[..., 2] ** 2)
    lab = torch.where(lt >= mu * ln * (1 - 1e-6) - 1e-10, 2, 1)
    return torch.where(ln <= 1e-10 + 1e-6 * scale, 0, lab)


def _exact_bncp(case, seed):
    J, Minv, v, mu = (_dev(a) for a in _stance(case, seed))
    G = J @ Minv @ J.transpose(1, 2)
    b = (J @ v.unsqueeze(-1)).squeeze(-1)
    B, nc = mu.shape
    rng = np.random.default_rng(int(seed))
    g = _dev(rng.standard_normal((B, 3 * nc)))
    rho = 1 / torch.linalg.eigvalsh(_blocks(G, nc))[..., -1]
    lam, live = torch.zeros(B, nc, 3, dtype=torch.float64, device=DEV), torch.arange(B, device=DEV)
    for it in range(5000):  # projected Gauss-Seidel, the residual read every ten sweeps
        Gl, bl, ml, rl, x = G[live], b[live], mu[live], rho[live], lam[live]
        for j in range(10):
            for c in range(nc):
                u = (Gl[:, 3 * c:3 * c + 3] @ x.reshape(len(live), -1, 1))[..., 0] + bl[:, 3 * c:3 * c + 3]
                x[:, c] = _proj(x[:, c] - rl[:, c, None] * _desaxce(u, ml[:, c]), ml[:, c])
        u = ((Gl @ x.reshape(len(live), -1, 1))[..., 0] + bl).reshape(-1, nc, 3)
        res = (x - _proj(x - rl[..., None] * _desaxce(u, ml), ml)).abs().amax((1, 2))
        lam[live] = x
        live = live[res >= 1e-6]
        if not len(live) or it >= 499:
            break
    # the derivative on the fixed branch: F(lam, b, mu) = 0, one row a component
    u = ((G @ lam.reshape(B, -1, 1))[..., 0] + b).reshape(B, nc, 3)
    lab = _branches(lam, mu)
    n = 3 * nc
    A = torch.zeros(B, n, n, dtype=torch.float64, device=DEV)
    Bb = torch.zeros_like(A)
    Bm = torch.zeros(B, n, nc, dtype=torch.float64, device=DEV)
    for c in range(nc):
        i = 3 * c
        ut = u[:, c, 1:]
        ns = torch.sqrt((ut ** 2).sum(-1)).clamp(min=1e-14)
        h = ut / ns[:, None]
        P = (torch.eye(2, dtype=torch.float64, device=DEV) - h[:, :, None] * h[:, None, :]) / ns[:, None, None]
        ml = mu[:, c] * lam[:, c, 0]
        slip = torch.zeros(B, 3, n, dtype=torch.float64, device=DEV)
        slip[:, 0] = G[:, i]
        slip[:, 1:] = ml[:, None, None] * (P @ G[:, i + 1:i + 3])
        slip[:, 1:, i] += mu[:, c, None] * h
        slip[:, 1, i + 1] += 1
        slip[:, 2, i + 2] += 1
        free = torch.zeros_like(slip)
        free[:, 0, i] = free[:, 1, i + 1] = free[:, 2, i + 2] = 1
        l3 = lab[:, c, None, None]
        A[:, i:i + 3] = torch.where(l3 == 0, free, torch.where(l3 == 1, G[:, i:i + 3], slip))
        db = torch.zeros(B, 3, 3, dtype=torch.float64, device=DEV)
        db[:, 0, 0] = 1
        db[:, 1:, 1:] = ml[:, None, None] * P
        eye = torch.eye(3, dtype=torch.float64, device=DEV).expand(B, 3, 3)
        Bb[:, i:i + 3, i:i + 3] = torch.where(l3 == 0, torch.zeros_like(db), torch.where(l3 == 1, eye, db))
        Bm[:, i + 1:i + 3, c] = torch.where(lab[:, c, None] == 2, lam[:, c, 0, None] * h, torch.zeros_like(h))
    y = torch.linalg.solve(A.transpose(1, 2), g.unsqueeze(-1))
    gb = -(Bb.transpose(1, 2) @ y)[..., 0]
    gmu = -(Bm.transpose(1, 2) @ y)[..., 0]
    return {"lam": lam.reshape(B, n), "gb": gb, "gmu": gmu, "labels": None, "iters": None}


def _exact_admm(case, seed):
    J, Minv, v, mu = (_dev(a) for a in _stance(case, seed))
    B, nc = mu.shape
    n = 3 * nc
    G = J @ Minv @ J.transpose(1, 2)
    b = (J @ v.unsqueeze(-1))[..., 0]
    ev = torch.linalg.eigvalsh(G)
    mx = ev[:, -1]
    mn = torch.where(ev > 1e-12 * mx[:, None], ev, mx[:, None]).amin(1)
    w = -torch.linalg.solve(G, b.unsqueeze(-1))[..., 0].reshape(B, nc, 3)
    bind = ((w[..., 0] <= 0) | (torch.sqrt(w[..., 1] ** 2 + w[..., 2] ** 2) > mu * w[..., 0])).any(1)
    rho = torch.where(bind, mx, mn)
    D = _blocks(G, nc)
    eye3 = torch.eye(3, dtype=torch.float64, device=DEV)
    P = torch.linalg.inv(D + rho[:, None, None, None] * eye3)
    rc = 1 / torch.linalg.eigvalsh(D)[..., -1]
    H = G + rho[:, None, None] * torch.eye(n, dtype=torch.float64, device=DEV)
    mv = lambda A, x: (A @ x.unsqueeze(-1))[..., 0]
    pre = lambda r: (P @ r.reshape(B, nc, 3, 1)).reshape(B, n)
    dot = lambda a, c: (a * c).sum(1, keepdim=True)
    over = lambda a, c: torch.where(c != 0, a / torch.where(c != 0, c, torch.ones_like(c)), torch.zeros_like(a))
    x, z, gam, u = (torch.zeros(B, n, dtype=torch.float64, device=DEV) for _ in range(4))
    s, live, r1 = torch.zeros(B, nc, dtype=torch.float64, device=DEV), torch.ones(B, 1, dtype=torch.bool, device=DEV), rho[:, None]
    for it in range(case["n_iter"]):
        q = b.clone()
        q[:, 0::3] += mu * s
        rhs = -((q + gam) - r1 * z)
        xn = x.clone()
        r = rhs - mv(H, xn)
        zz = pre(r)
        p, s0 = zz.clone(), dot(r, zz)
        for _ in range(8):
            Ap = mv(H, p)
            a = over(s0, dot(p, Ap))
            xn, r = xn + a * p, r - a * Ap
            zz = pre(r)
            s3 = dot(r, zz)
            p, s0 = zz + over(s3, s0) * p, s3
        zn = _proj((xn + gam / r1).reshape(B, nc, 3), mu).reshape(B, n)
        gn = gam + r1 * (xn - zn)
        x, z, gam = (torch.where(live, a, c) for a, c in ((xn, x), (zn, z), (gn, gam)))
        if (it + 1) % 4 == 0:
            u = mv(G, z) + b
            u3, z3 = u.reshape(B, nc, 3), z.reshape(B, nc, 3)
            s = torch.sqrt(u3[..., 1] ** 2 + u3[..., 2] ** 2)
            res = (z3 - _proj(z3 - rc[..., None] * _desaxce(u3, mu), mu)).abs().amax((1, 2))
            live = live & (res >= 1e-8)[:, None]
    lam, u3 = z.reshape(B, nc, 3), u.reshape(B, nc, 3)
    v_plus = v + mv(Minv @ J.transpose(1, 2), z)
    # the fixed-branch derivative: lam' = Z y + p, Z^T (G lam' + b') + D y + mu (w . (G lam' + b')_t) e_n = 0
    lab = _branches(lam, mu)
    Z = torch.zeros(B, n, n, dtype=torch.float64, device=DEV)
    L = torch.zeros(B, n, n, dtype=torch.float64, device=DEV)  # Z^T plus the slip speed's row
    Dv = torch.zeros(B, n, dtype=torch.float64, device=DEV)
    hat = torch.zeros(B, nc, 2, dtype=torch.float64, device=DEV)
    for c in range(nc):
        i, l3 = 3 * c, lab[:, c, None, None]
        ut = u3[:, c, 1:]
        nw = torch.sqrt((ut ** 2).sum(-1)).clamp(min=1e-300)
        h = ut / nw[:, None]
        zs = torch.zeros(B, 3, 3, dtype=torch.float64, device=DEV)
        zs[:, 0, 0] = 1
        zs[:, 1:, 0] = -mu[:, c, None] * h
        zs[:, 1, 1], zs[:, 2, 1] = -h[:, 1], h[:, 0]
        zc = torch.where(l3 == 2, zs, torch.where(l3 == 1, eye3.expand(B, 3, 3), torch.zeros_like(zs)))
        Z[:, i:i + 3, i:i + 3] = zc
        L[:, i:i + 3, i:i + 3] = zc.transpose(1, 2)
        slip = lab[:, c] == 2
        L[:, i, i + 1:i + 3] += torch.where(slip[:, None], mu[:, c, None] * h, torch.zeros_like(h))
        ds = torch.stack([torch.zeros_like(nw), nw / (mu[:, c] * lam[:, c, 0]).clamp(min=1e-300), torch.ones_like(nw)], 1)
        Dv[:, i:i + 3] = torch.where(lab[:, c, None] == 0, torch.ones_like(ds), torch.where(slip[:, None], ds, torch.zeros_like(ds)))
        hat[:, c] = torch.where(slip[:, None], h, torch.zeros_like(h))
    A = L @ G @ Z + torch.diag_embed(Dv)
    first = torch.where((lab == 2).any(1), (lab == 2).int().argmax(1), torch.full((B,), -1, device=DEV))

    def response(p, db):
        y = torch.linalg.solve(A, -(L @ (G @ p.unsqueeze(-1) + db.unsqueeze(-1))))[..., 0]
        return mv(Z, y) + p

    d_tau = response(torch.zeros_like(b), DT * mv(J, Minv[:, :, 0]))
    dv_tau = DT * Minv[:, :, 0] + mv(Minv @ J.transpose(1, 2), d_tau)
    p = torch.zeros(B, nc, 3, dtype=torch.float64, device=DEV)
    at = torch.arange(B, device=DEV)[first >= 0], first[first >= 0]
    p[at[0], at[1], 1:] = -lam[at[0], at[1], 0, None] * hat[at[0], at[1]]
    d_mu = response(p.reshape(B, n), torch.zeros_like(b))
    return {"lam": lam, "u": u3, "v_plus": v_plus, "rho": rho, "dlam_tau": d_tau.reshape(B, nc, 3), "dv_tau": dv_tau,
            "dlam_mu": d_mu.reshape(B, nc, 3), "labels": None, "mask": None}


def exact(case, seed):
    """The batched solvers in 64 bits.  The engines, the sweeps and the rollout have no such value
    apart from their own order of contacts and colours: a few sweeps over an indeterminate pile
    end where that order takes them."""
    if case["kind"] == "admm":
        return _exact_admm(case, seed)
    if case["kind"] == "bncp":
        return _exact_bncp(case, seed)
    return None
