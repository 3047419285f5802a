"""Performance cases: what a program of this framework has it do, through the
public entry points, with inputs made from a seed.

A case is a dict of plain values; `listed()` gives the named ones, `draw()`
more of the same ranges.  `prepare()` makes what the program holds before the
call, `run()` is one pass, `work()` the operations and bytes one pass cannot do
without, and `exact()` what the pass computes, restated in plain FP64 torch.

Most passes are a block of steps of a device-resident system that goes on from
pass to pass, ended by the observables (the monitor line) and the state copied
into page-locked arrays the program keeps.  Such runs use the corrected forces
where the field has them (`set_physics`): the reference's AIREBO and MM forces
are not gradients and leave the crystal within a hundred steps, so no long run
is made with them.  The reference's own AIREBO forces are measured the way they
are used, as whole short jobs from host arrays.  What a pass with FP32 or BF16
pair arithmetic returns is kept in single precision, as such a run's trajectory
is.
"""
import math

import numpy as np
import torch

from fuller_md_en_b200 import Batch, Context, RunConfig, System, _lib, api, crystal
from fuller_md_en_b200 import Rebo2Knots
from fuller_md_en_b200 import surrogate as sgm

KB, CONV, EV2GPA, MC = 8.617333262e-5, 9.64853321e-3, 160.21766208, 12.011
JITTER = 0.01
_CTX = None


def ctx():
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


def listed():
    f64, f32 = "f64", "f32"
    return [
        # rigid-body core: 108 C60, the smallest headline run; one monitor interval
        dict(name="rigid nc=3", kind="rigid", nc=3, st="FCC", prec=f64, T=300.0, P=0.0, steps=50),
        # rigid-body full: 4,000 C60 / 240,000 sites, FP32 pairs, 1 GPa
        dict(name="rigid nc=10 f32", kind="rigid", nc=10, st="FCC", prec=f32, T=300.0, P=1.0, steps=50),
        # the headline workload as a job: host arrays in, lists, 50 steps, state out
        dict(name="airebo job nc=5", kind="job", nc=5, st="FCC", prec=f64, T=300.0, P=0.0, steps=50),
        # a short job on one unit cell (240 atoms): latency of everything
        dict(name="airebo job nc=1", kind="job", nc=1, st="FCC", prec=f64, T=300.0, P=0.0, steps=20),
        # AIREBO production runs: small, the headline size, and the largest (FP32 pairs)
        dict(name="airebo nc=2", kind="airebo", nc=2, st="FCC", prec=f64, T=300.0, P=0.0, steps=100, ramp=False),
        dict(name="airebo nc=5", kind="airebo", nc=5, st="FCC", prec=f64, T=300.0, P=0.0, steps=100, ramp=False),
        dict(name="airebo nc=8 f32", kind="airebo", nc=8, st="FCC", prec=f32, T=300.0, P=0.0, steps=40, ramp=False),
        # molecular mechanics: one crystal, and a batch of uneven replicas
        dict(name="mm nc=4", kind="mm", nc=4, st="FCC", prec=f64, T=500.0, P=1.0, steps=100, ramp=False),
        dict(name="mm batch 32", kind="batch", reps=32, lo=2, hi=5, prec=f64, steps=20),
        # the learned bond order: inference at its configuration's size, judged once; training
        dict(name="learned nc=8", kind="learned", nc=8, steps=40, judge=40),
        dict(name="train nc=5", kind="train", nc=5, snaps=16, batch=8, steps=10),
        # the REBO-II extension with switched LJ
        dict(name="rebo2 job nc=5", kind="rebo2", nc=5, steps=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rigid", "rigid", "airebo", "airebo", "airebo", "mm", "mm", "job", "batch", "learned", "train",
                       "rebo2"])
    steps = _log(rng, 20, 100)
    st = rng.choice(["FCC", "FCC", "FCC", "BCC", "HCP"])
    prec = rng.choice(["f64", "f64", "f32"])
    if kind == "rigid":
        return dict(kind=kind, nc=_log(rng, 2, 9), st=st, prec=prec, T=round(rng.uniform(50, 500), 1),
                    P=round(rng.uniform(0, 2), 2), steps=min(steps, 50))
    if kind == "airebo":
        return dict(kind=kind, nc=_log(rng, 1, 7), st=st, prec=prec, T=round(rng.uniform(50, 320), 1),
                    P=round(rng.uniform(0, 1), 2), steps=steps, ramp=rng.random() < 0.2)
    if kind == "mm":
        return dict(kind=kind, nc=_log(rng, 1, 6), st=st, prec=prec, T=round(rng.uniform(50, 700), 1),
                    P=round(rng.uniform(0, 2), 2), steps=steps, ramp=rng.random() < 0.2)
    if kind == "job":
        return dict(kind=kind, nc=_log(rng, 1, 6), st=st, prec=prec, T=round(rng.uniform(50, 400), 1),
                    P=round(rng.uniform(0, 2), 2), steps=min(steps, 50))
    if kind == "batch":
        lo = rng.randint(1, 3)
        return dict(kind=kind, reps=rng.randint(3, 24), lo=lo, hi=lo + rng.randint(1, 2), prec="f64", steps=steps)
    if kind == "learned":
        return dict(kind=kind, nc=_log(rng, 1, 7), steps=min(steps, 40), judge=rng.choice([10, 15, 40]))
    if kind == "train":
        return dict(kind=kind, nc=_log(rng, 1, 4), snaps=rng.randint(2, 12), batch=rng.randint(1, 8),
                    steps=rng.randint(2, 20))
    return dict(kind="rebo2", nc=_log(rng, 1, 5), steps=min(steps, 40))


# --------------------------------------------------------------------- inputs

def _crystal(case, seed):
    """Initial state of an atomistic or rigid case: host arrays, as the drivers build them."""
    st = case.get("st", "FCC")
    if case["kind"] == "rigid":
        return crystal.rigid(case["nc"], T=case["T"], seed=seed, st=st)
    mm = case["kind"] == "mm"
    return crystal.atomistic(case["nc"], T=case.get("T", 300.0), jitter=JITTER, seed=seed, st=st,
                             mol_base=0 if mm else 1)


def _config(case, nmol):
    return RunConfig(dt={"rigid": 1.0, "mm": 0.1}.get(case["kind"], 0.5), T=case.get("T", 300.0),
                     Pe=case.get("P", 0.0), T_cold=4.0, warmup=10 ** 6 if case.get("ramp") else 0, nsteps=10 ** 6,
                     nlup=25 if case["kind"] == "rigid" else 20, gavg_from=1, gavg_to=10 ** 6, nc=case["nc"],
                     nmol=nmol, precision=_lib.FMD_PREC_FP32_PAIR if case.get("prec") == "f32" else _lib.FMD_PREC_FP64)


def _rmcut(s):
    return 3.0 * 3.431 + 2.0 * s["Rmol"] + 1.0


def _system(case, s):
    """A new system of the case from its host arrays, not yet initialised."""
    T, P = case.get("T", 300.0), case.get("P", 0.0)
    if case["kind"] == "rigid":
        return System.rigid(ctx(), _config(case, s["n"]), 60, s["body"], s["I0"], s["Mmol"], _rmcut(s), s["pos"],
                            s["vel"], s["qv"], s["omg"], s["h"], crystal.npt_rigid(T, P, s["n"]))
    na = s["pos"].size // 3
    npt = crystal.npt_atom(T, P, na)
    if case["kind"] == "mm":
        y = System.mm_replicated(ctx(), _config(case, s["nmol"]), s["nmol"], na // s["nmol"], s["pos"], s["vel"],
                                 _molecule()[1], s["h"], npt)
        y.set_physics(_lib.FMD_PHYS_MM_BONDED)
        return y
    y = System.airebo(ctx(), _config(case, s["nmol"]), s["pos"], s["vel"], s["mass"], s["mol_id"], s["h"], npt)
    if case["kind"] == "airebo":
        y.set_physics(_lib.FMD_PHYS_REBO)
    return y


_MOL = []


def _molecule():
    """One C60's MM topology, as a dict and as the handle the systems take."""
    if not _MOL:
        c = crystal.c60_ih()
        t = crystal.mm_topology(c, crystal.bonds_from_geometry(c), 1)
        _MOL.extend([t, api.Topology(t["bonds"], t["kb"], t["r0"], t["angles"], t["kth"], t["th0"], t["dihedrals"],
                                     t["vn"], t["mult"], t["gamma"], t["impropers"], t["ki"], t["igamma"])])
    return _MOL


def _net(seed):
    """A network about the fullerene's own bond order (0.955), as early in training."""
    P = sgm.init_params(seed)
    P["b0"], P["bs"] = 0.955, 0.005
    return P


def _knots():
    """Spline knots of the published tables' scale (the tables are the caller's)."""
    rng = np.random.default_rng(0)

    def tri(shift, amp):
        t = rng.uniform(-0.3 * amp, 0.3 * amp, (5, 5, 10, 8))
        t[..., 0] = rng.uniform(-amp, amp, (5, 5, 10)) + shift
        return t

    pcc = np.column_stack([rng.uniform(-0.05, 0.05, 5), rng.uniform(-0.03, 0.03, 5)])
    return Rebo2Knots(pcc, tri(-0.05, 0.03), tri(0.0, 0.01))


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _buffers(n, rigid):
    b = {"pos": _pinned(3 * n), "vel": _pinned(3 * n), "h": _pinned(9)}
    if rigid:
        b |= {"qv": _pinned(4 * n), "omg": _pinned(3 * n)}
    return b


def _replicas(case, seed):
    rng = np.random.default_rng(seed)
    span = case["hi"] - case["lo"] + 1
    return [dict(kind="mm", nc=case["lo"] + r % span, T=float(rng.uniform(100.0, 700.0)),
                 P=float(rng.uniform(0.0, 2.0)), prec=case["prec"], steps=case["steps"], seed=int(rng.integers(1 << 30)))
            for r in range(case["reps"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        reps = _replicas(case, seed)
        ys = [_system(c, _crystal(c, c["seed"])) for c in reps]
        n = sum(y.n for y in ys)
        pos, vel, h, at, outs = _pinned(3 * n), _pinned(3 * n), _pinned(9 * len(ys)), 0, []
        for k, y in enumerate(ys):
            outs.append({"pos": pos[at:at + 3 * y.n], "vel": vel[at:at + 3 * y.n], "h": h[9 * k:9 * k + 9]})
            at += 3 * y.n
        return {"case": case, "ys": ys, "b": Batch(ctx(), ys), "g": 0, "outs": outs, "pos": pos, "vel": vel, "h": h}
    if kind == "train":
        s = _crystal(dict(case, kind="job"), seed)
        y = _system(dict(case, kind="job"), s)
        y.init()
        data = sgm.Dataset(ctx())
        for g in range(1, case["snaps"] + 1):
            y.enqueue(g, g)
            data.add_system(y)
        ctx().synchronize()
        y.close()
        return {"case": case, "data": data, "model": sgm.Surrogate(ctx(), _net(seed))}
    s = _crystal(case, seed)
    n = s["n"] if kind == "rigid" else s["pos"].size // 3
    state = {"case": case, "s": s, "out": _buffers(n, kind == "rigid"), "g": 0}
    if kind in ("rigid", "airebo", "mm"):
        state["y"] = _system(case, s)
        state["y"].init()
    elif kind == "learned":
        state["model"] = sgm.Surrogate(ctx(), _net(seed))
    elif kind == "rebo2":
        state["knots"] = _knots()
    return state


def _obs(o):
    return np.array([o.T, o.P, o.a, o.KE, *o.E])


def _kept(case, r):
    """What the program keeps of a pass: FP64, or single precision of a mixed-precision run."""
    if case.get("prec") == "f32" or case["kind"] in ("learned", "train"):
        return {k: np.asarray(v).astype(np.float32) for k, v in r.items()}
    return r


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    K = case["steps"]
    if kind == "batch":
        o = state["b"].run(state["g"] + 1, state["g"] + K)
        state["g"] += K
        npt = [y.download(out=out)["npt"] for y, out in zip(state["ys"], state["outs"])]
        return {"obs": np.array([_obs(x) for x in o]), "npt": np.array(npt), "pos": state["pos"],
                "vel": state["vel"], "h": state["h"]}
    if kind == "train":
        hist = state["model"].train(state["data"], steps=K, batch=case["batch"], lr=3e-3, lr_final=3e-5, wE=0.1,
                                    wF=1.0, wW=0.1, seed=1)
        return _kept(case, {"hist": hist, **state["model"].params()})
    if kind in ("rigid", "airebo", "mm"):
        o = state["y"].run(state["g"] + 1, state["g"] + K)
        state["g"] += K
        d = state["y"].download(out=state["out"])
    else:
        y = _system(dict(case, kind="job"), state["s"])
        if kind == "rebo2":
            y.set_rebo2(state["knots"], _lib.FMD_REBO2_BOND_ORDER | _lib.FMD_REBO2_LJ_SWITCH)
        y.init()
        if kind == "learned":
            y.use_surrogate(state["model"], judge_every=case["judge"], rmse_max=1e9)
        o = y.run(1, K)
        d = y.download(out=state["out"])
        y.close()
    return _kept(case, {"obs": _obs(o), **{k: v for k, v in d.items() if v is not None}})


# ----------------------------------------------------------------------- work

def _atoms(case):
    return case["nc"] ** 3 * (4 if case.get("st", "FCC") == "FCC" else 2) * 60


def work(case):
    """Operations of the pair, bond and network terms over a pass's steps (in-cutoff
    pairs of the crystal as made: 155 atom pairs an atom, 10,200 site pairs a rigid
    molecule, once each), and the state read and written once a pass."""
    kind, K = case["kind"], case["steps"]
    if kind == "batch":
        w = [work(dict(kind="mm", nc=case["lo"] + r % (case["hi"] - case["lo"] + 1), steps=K))
             for r in range(case["reps"])]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    n = _atoms(case)
    mlp = 3 * n * 3 * 2 * (32 * 128 + 2 * 128 * 128 + 128)      # rows x (forward + gradient network)
    if kind == "train":
        nsnap = K * case["batch"]
        return {"bytes": nsnap * n * (48 + 12 * 4), "flops": nsnap * 3 * mlp}
    if kind == "rigid":
        m = n // 60
        return {"bytes": 2 * 13 * 8 * m, "flops": K * m * 10200 * 72}
    lj = 155 * n * 48
    bonded = n * (1.5 * 30 + 3 * 80 + 6 * 150 + 150) if kind == "mm" else n * 1.5 * 400
    return {"bytes": 96 * n, "flops": K * (lj + bonded + (mlp if kind == "learned" else 0))}


# ---------------------------------------------------------- the same in FP64

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_dev())


def _image(d, h):
    return _wrap_with(d, h, torch.round)


def _wrap_with(d, h, f):
    s = d @ torch.linalg.inv(h).T
    return (s - f(s)) @ h.T


def _add(F, i, f):
    return F.index_add_(0, i.reshape(-1), f.reshape(-1, 3))


def _lj_consts(sig, eps, sr):
    s6 = (sr * sr) ** 3
    return sig * sig, eps, 4 * eps * (s6 * s6 - s6)


AIREBO_LJ, MM_LJ = _lj_consts(3.40, 2.84e-3, 3.40 / (3.0 * 3.40)), _lj_consts(3.431, 2.635e-3, 1.0 / 3.0)


def _lj_pair(r2, c):
    """(fm, e) of in-cutoff pairs: f = -fm d on the first atom."""
    r2 = r2.clamp(min=0.25)
    s6 = (c[0] / r2) ** 3
    return 24 * c[1] * (2 * s6 * s6 - s6) / r2, 4 * c[1] * (s6 * s6 - s6) - c[2]


def _half_list(pos, h, rc):
    """(i, j) of the half list, j > i in other molecules of 60, ascending, 400 an atom."""
    n = len(pos)
    M = n // 60
    x = pos.reshape(M, 60, 3)
    # whole-molecule screen: the span about the first atom bounds every atom pair
    span = _image(x - x[:, :1], h).norm(dim=-1).max()
    wide = float(torch.linalg.svdvals(h).min()) > 2 * (rc + 2 * float(span))
    ii, jj = [], []
    for A in range(M):
        B = torch.arange(A + 1, M, device=pos.device)
        if wide and len(B):
            B = B[_image(x[B, 0] - x[A, 0], h).norm(dim=-1) < rc + 2 * span]
        if not len(B):
            continue
        d = _image(x[B].reshape(1, -1, 3) - x[A].reshape(60, 1, 3), h)
        ok = (d * d).sum(-1) < rc * rc
        ok &= ok.cumsum(1) <= 400
        a, b = ok.nonzero(as_tuple=True)
        ii.append(60 * A + a)
        jj.append(60 * B[b // 60] + b % 60)
    z = torch.zeros(0, dtype=torch.long, device=pos.device)
    return torch.cat(ii + [z]), torch.cat(jj + [z])


def _lj(pos, h, pairs, c, rc, F, full):
    E, W = 0.0, torch.zeros(3, 3, dtype=pos.dtype, device=pos.device)
    for i, j in zip(pairs[0].split(1 << 24), pairs[1].split(1 << 24)):
        d = _image(pos[j] - pos[i], h)
        r2 = (d * d).sum(-1)
        k = r2 <= rc * rc
        i, j, d, r2 = i[k], j[k], d[k], r2[k]
        fm, e = _lj_pair(r2, c)
        g = fm[:, None] * d
        _add(F, i, -g)
        _add(F, j, g)
        E, W = E + e.sum(), W + d.T @ g
    return E, W if full else torch.diag(torch.diag(W))


def _bond_list(pos, h, rc=2.3):
    """Neighbour table (n, m) within the molecules of 60 and its mask, m the longest row."""
    x = pos.reshape(-1, 60, 3)
    d = _image(x[:, None] - x[:, :, None], h)
    ok = ((d * d).sum(-1) < rc * rc) & ~torch.eye(60, dtype=torch.bool, device=pos.device)
    m = int(ok.sum(-1).max())
    order = torch.argsort((~ok).to(torch.uint8), dim=-1, stable=True)[..., :m]
    base = 60 * torch.arange(len(x), device=pos.device)[:, None, None]
    return (order + base).reshape(-1, m), torch.gather(ok, 2, order).reshape(-1, m)


def _cheb(x, n):
    T = [torch.ones_like(x), x]
    while len(T) < n:
        T.append(2 * x * T[-1] - T[-2])
    return torch.stack(T[:n], -1)


def _net_order(P, ct, rk, fk, use):
    """Bond order of every directed bond (n, m) from the network, over k (n, m, m),
    and its derivatives with respect to r_k and cos."""
    with torch.enable_grad():
        ct, rk = ct.detach().requires_grad_(), rk.detach().requires_grad_()
        s = (rk - 1.7) / 0.3
        fk = torch.where(rk <= 1.7, 1.0, torch.where(rk >= 2.0, 0.0, 0.5 * (1 + torch.cos(math.pi * s))))
        phi = fk[..., None] * _cheb((rk - 1.55) / 0.45, 4)
        feat = phi[..., :, None] * _cheb(ct, 8)[..., None, :]
        x = (feat.flatten(-2) * use[..., None]).sum(2)
        x = (x - _t(P["m"])) / _t(P["s"])
        one = torch.ones_like(x[..., :1])
        a = torch.cat([x[..., :31], one], -1)
        for l in ("W1", "W2", "W3"):
            a = torch.cat([torch.nn.functional.silu(a @ _t(P[l]))[..., :127], one], -1)
        b = P["b0"] + P["bs"] * (a @ _t(P["w4"]))
        gr, gc = torch.autograd.grad(b.sum(), (rk, ct))
    return b.detach(), gr, gc


def _formula_order(ct, rk, fk, use):
    """The reference's bond order (1 + sum f_c G)^-1/2 and its derivatives."""
    s = (rk - 1.7) / 0.3
    dfk = torch.where((rk <= 1.7) | (rk >= 2.0), 0.0, -0.5 * math.pi / 0.3 * torch.sin(math.pi * s))
    c2, d2 = 330.0 ** 2, 3.5 ** 2
    q = d2 + (1 + ct) ** 2
    G, dG = 0.00020813 * (1 + c2 / d2 - c2 / q), 0.00020813 * 2 * c2 * (1 + ct) / (q * q)
    g = (fk * G * use).sum(2)
    b = (1 + g) ** -0.5
    dbp = torch.where(g.abs() > 1e-20, -0.5 * b / (1 + g), 0.0)[:, :, None]
    return b, dbp * dfk * G, dbp * fk * dG


def _rebo(pos, h, nb, F, order, corrected):
    """REBO energy and pair virial; adds the reference's forces, or the gradient's."""
    j, ok = nb
    n, m = j.shape
    i = torch.arange(n, device=pos.device)[:, None].expand(n, m)
    d = _image(pos[j] - pos[:, None], h)
    r = torch.where(ok, d.norm(dim=-1), 3.0)
    s = (r - 1.7) / 0.3
    inside = (r > 1.7) & (r < 2.0)
    fc = torch.where(r <= 1.7, 1.0, torch.where(inside, 0.5 * (1 + torch.cos(math.pi * s)), 0.0))
    dfc = torch.where(inside, -0.5 * math.pi / 0.3 * torch.sin(math.pi * s), 0.0)
    bond = ok & (r <= 2.0) & ~((fc < 1e-15) & (dfc == 0))
    ex = 10953.544162170 * torch.exp(-4.7465390606595 * r)
    q = 0.3134602960833
    vr, dvr = (1 + q / r) * ex, -q / (r * r) * ex - (1 + q / r) * 4.7465390606595 * ex
    terms = [(12388.79197798, 4.7204523127), (17.56740646509, 1.4332132499), (30.71493208065, 1.3826912506)]
    va = sum(B * torch.exp(-b * r) for B, b in terms)
    dva = sum(-b * B * torch.exp(-b * r) for B, b in terms)
    u = d / r[..., None]
    # three-body slots (i, bond, k): the centre's other neighbours
    ct = (u @ u.transpose(1, 2)).clamp(-1.0, 1.0)
    use = (ok & (r <= 2.0) & (fc >= 1e-15))[:, None, :] & ~torch.eye(m, dtype=torch.bool, device=pos.device)
    rk, fk = r[:, None, :].expand(n, m, m), fc[:, None, :].expand(n, m, m)
    b, gr, gc = order(ct, rk, fk, use)
    coef = torch.where(bond, -0.5 * fc * va, 0.0)[..., None, None]
    uk, ub = u[:, None], u[:, :, None]
    sg = -1.0 if corrected else 1.0
    w = torch.where(use, 1.0, 0.0)[..., None]
    fk3 = sg * w * coef * (gr[..., None] * uk + gc[..., None] * (ub - ct[..., None] * uk) / rk[..., None])
    _add(F, j[:, None, :].expand(n, m, m)[use], fk3[use])
    F -= fk3.sum((1, 2))
    if corrected:
        fb = (sg * w * coef * gc[..., None] * (uk - ct[..., None] * ub) / r[:, :, None, None]).sum(2)
        _add(F, j[bond], fb[bond])
        F -= fb.sum(1)
    # partner slot: where i stands in j's row (rows are symmetric)
    back = (j[j] == i[..., None]) & ok[j]
    bji = torch.gather(b[j], 2, back.to(torch.uint8).argmax(-1, keepdim=True))[..., 0]
    bbar = 0.5 * (b + bji)
    half = bond & (j > i)
    e = torch.where(half, fc * (vr - bbar * va), 0.0)
    fp = torch.where(half, (dfc * (vr - bbar * va) + fc * (dvr - bbar * dva)) / r, 0.0)
    f = fp[..., None] * d
    F += f.sum(1)
    _add(F, j[half], -f[half])
    return e.sum(), -torch.einsum("nma,nmb->ab", d, f)


def _bonded(pos, h, t, F):
    """MM bonded energies and the bonds' diagonal virial; adds -grad E."""
    n = len(pos)
    off = 60 * torch.arange(n // 60, device=pos.device)[:, None, None]

    def ids(k):
        return (torch.as_tensor(np.asarray(t[k]), device=pos.device).long()[None] + off).flatten(0, 1).unbind(1)

    def par(k):
        return _t(t[k]).repeat(n // 60)

    with torch.enable_grad():
        x = pos.detach().requires_grad_()

        def v(a, b):
            return _image(x[b] - x[a], h)

        def torsion(a, b, c, e, mult, vn, gamma):
            b1, b2, b3 = v(a, b), v(b, c), v(c, e)
            m, q = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
            phi = torch.atan2((m * b3).sum(-1) * b2.norm(dim=-1), (m * q).sum(-1))
            return (0.5 * vn * (1 + torch.cos(mult * phi - gamma))).sum()

        a, b = ids("bonds")
        d = v(a, b)
        r = d.norm(dim=-1)
        eb = (0.5 * par("kb") * (r - par("r0")) ** 2).sum()
        i, j, k = ids("angles")
        p, q = v(j, i), v(j, k)
        c = (p * q).sum(-1) / (p.norm(dim=-1) * q.norm(dim=-1))
        ea = (0.5 * par("kth") * (torch.acos(c.clamp(-0.999999, 0.999999)) - par("th0")) ** 2).sum()
        ed = torsion(*ids("dihedrals"), par("mult"), par("vn"), par("gamma"))
        c0, c1, c2, c3 = ids("impropers")
        ei = torsion(c1, c0, c2, c3, 2, par("ki"), par("igamma"))
        F -= torch.autograd.grad(eb + ea + ed + ei, x)[0]
    fm = par("kb") * (r - par("r0")) / r
    W = torch.diag((d * fm[:, None] * d).sum(0)).detach()
    return [e.detach() for e in (eb, ea, ed, ei)], W


def _rot(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                        1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                        1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


def _rigid_forces(pos, qv, body, h, pairs, rmcut):
    """Forces, torques, energy and virial of the site-site LJ over molecule pairs i < j."""
    n = len(pos)
    lab = torch.einsum("nab,sb->nsa", _rot(qv), body)
    F, T = torch.zeros_like(pos), torch.zeros_like(pos)
    E, W = 0.0, torch.zeros(3, 3, dtype=pos.dtype, device=pos.device)
    rc = 3.0 * 3.431
    for i, j in zip(pairs[0].split(4096), pairs[1].split(4096)):
        m = _image(pos[j] - pos[i], h)
        k = (m * m).sum(-1) <= rmcut * rmcut
        i, j, m = i[k], j[k], m[k]
        if not len(i):
            continue
        d = (m[:, None] + lab[j])[:, None] - lab[i][:, :, None]
        r2 = (d * d).sum(-1)
        fm, e = _lj_pair(r2, MM_LJ)
        on = r2 < rc * rc
        g = torch.where(on, fm, 0.0)[..., None] * d
        fi, fj = -g.sum(2), g.sum(1)
        _add(F, i, fi.sum(1))
        _add(F, j, fj.sum(1))
        _add(T, i, torch.linalg.cross(lab[i], fi).sum(1))
        _add(T, j, torch.linalg.cross(lab[j], fj).sum(1))
        E, W = E + torch.where(on, e, 0.0).sum(), W + torch.einsum("psta,pstb->ab", d, g)
    return F, T, E, W


def _clamp(x, a):
    return max(-a, min(a, float(x)))


def _trajectory(case, s, P=None):
    """The state and observables after the first pass, in FP64."""
    kind, K = case["kind"], case["steps"]
    rigid, mm = kind == "rigid", kind == "mm"
    dt, T, nlup = {"rigid": 1.0, "mm": 0.1}.get(kind, 0.5), case.get("T", 300.0), 25 if rigid else 20
    pos, vel, h = _t(s["pos"]).reshape(-1, 3), _t(s["vel"]).reshape(-1, 3), _t(s["h"]).reshape(3, 3)
    n = len(pos)
    npt = (crystal.npt_rigid if rigid else crystal.npt_atom)(T, case.get("P", 0.0), n).copy()
    xi, Q, Vg, Wb, Pe, Tt, Nf = 0.0, npt[1], np.zeros(3), npt[11], npt[12], npt[13], npt[14]
    mass = s["Mmol"] if rigid else MC
    if rigid:
        qv, omg, body = _t(s["qv"]).reshape(-1, 4), _t(s["omg"]).reshape(-1, 3), _t(s["body"]).reshape(-1, 3)
    lists = None

    def rebuild():
        if rigid:
            a, b = torch.triu_indices(n, n, 1, device=pos.device)
            ok = torch.cat([(_image(pos[y] - pos[x], h) ** 2).sum(-1) < (_rmcut(s) + 3.0) ** 2
                            for x, y in zip(a.split(1 << 22), b.split(1 << 22))])
            return a[ok], b[ok]
        pairs = _half_list(pos, h, (3.0 * 3.431 if mm else 3.0 * 3.40) + 2.0)
        return pairs, None if mm else _bond_list(pos, h)

    def forces():
        if rigid:
            F, Tq, E, W = _rigid_forces(pos, qv, body, h, lists, _rmcut(s))
            return F, Tq, [E], W
        F = torch.zeros_like(pos)
        if mm:
            e, W = _bonded(pos, h, _molecule()[0], F)
            el, Wl = _lj(pos, h, lists[0], MM_LJ, 3.0 * 3.431, F, False)
            return F, None, e + [el, 0.0, sum(e) + el], W + Wl
        order = (lambda *a: _net_order(P, *a)) if P is not None else _formula_order
        er, Wr = _rebo(pos, h, lists[1], F, order, kind == "airebo")
        el, Wl = _lj(pos, h, lists[0], AIREBO_LJ, 3.0 * 3.40, F, True)
        return F, None, [er + el, er, el], Wr + Wl

    def kinetic():
        kt = 0.5 * mass * float((vel * vel).sum()) / CONV
        return (kt, 0.5 * s["I0"] * float((omg * omg).sum()) / CONV) if rigid else (kt, 0.0)

    def half(xi, Vg, W):
        xi = _clamp(xi + 0.5 * dt * (2 * (kt + kr) - Nf * KB * Tt) / Q, 0.1 if rigid else 0.05)
        V = abs(float(torch.linalg.det(h)))
        dP = (2 * kt + float(torch.trace(W))) / (3 * V) * EV2GPA - Pe
        return xi, np.clip(Vg + 0.5 * dt * V * dP / (Wb * EV2GPA), *((-0.01, 0.01) if rigid else (-0.005, 0.005)))

    lists = rebuild()
    pos = _wrap_with(pos, h, torch.floor)
    F, Tq, E, W = forces()
    kt, kr = kinetic()
    Tn = Pn = 0.0
    for g in range(1, K + 1):
        if g % nlup == 0:
            lists = rebuild()
        if case.get("ramp"):
            Tt = 4.0 + (T - 4.0) * g / 10 ** 6
        xi, Vg = half(xi, Vg, W)
        hi = torch.linalg.inv(h)
        nh = math.exp(-0.5 * dt * xi)
        tr = lambda m: float((torch.diag(m) * _t(Vg)).sum())
        sc = nh * math.exp(-0.5 * dt * tr(hi) / 3)
        vel = vel * sc + 0.5 * dt * F * (CONV / mass)
        fr = pos @ hi.T + dt * (vel @ hi.T)
        h = h + dt * torch.diag(_t(Vg))
        pos = (fr - torch.floor(fr)) @ h.T
        sc2 = nh * math.exp(-0.5 * dt * tr(torch.linalg.inv(h)) / 3)
        if rigid:
            omg = omg * nh + 0.5 * dt * Tq * (CONV / s["I0"])
            wm = omg.norm(dim=-1, keepdim=True)
            dq = torch.cat([torch.cos(wm * dt / 2), torch.sin(wm * dt / 2) / wm * omg], -1)
            a, b, c, d = qv.unbind(-1)
            R = torch.stack([a, -b, -c, -d, b, a, -d, c, c, d, a, -b, d, -c, b, a], -1).reshape(-1, 4, 4)
            qv = (R @ dq[..., None])[..., 0]
            qv = qv / qv.norm(dim=-1, keepdim=True)
        F, Tq, E, W = forces()
        vel = (vel + 0.5 * dt * F * (CONV / mass)) * sc2
        if rigid:
            omg = (omg + 0.5 * dt * Tq * (CONV / s["I0"])) * nh
        kt, kr = kinetic()
        xi, Vg = half(xi, Vg, W)
        Tn = 2 * (kt + kr) / (Nf * KB)
        Pn = (2 * kt + float(torch.trace(W))) / (3 * abs(float(torch.linalg.det(h)))) * EV2GPA
        if case.get("ramp") and Tn > 0.1:
            vel = vel * math.sqrt(max(Tt, 0.1) / Tn)
            kt, kr = kinetic()
            Tn, xi = 2 * kt / (Nf * KB), 0.0
    E = [float(x) for x in E]
    r = {"obs": np.array([Tn, Pn, float(h[0, 0]) / case["nc"], kt + kr] + E + [0.0] * (8 - len(E))),
         "pos": pos.reshape(-1).cpu().numpy(), "vel": vel.reshape(-1).cpu().numpy(), "h": h.reshape(-1).cpu().numpy()}
    if rigid:
        r |= {"qv": qv.reshape(-1).cpu().numpy(), "omg": omg.reshape(-1).cpu().numpy()}
    vg = np.zeros(9)
    vg[[0, 4, 8]] = Vg
    r["npt"] = np.array([xi, Q, *vg, Wb, Pe, Tt, Nf])
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "rebo2"):
        return None               # the draw of the batches / the splines are the library's own
    with torch.no_grad():
        if kind == "batch":
            # a replica's first pass is its own run's
            cs = _replicas(case, seed)
            if case["steps"] * sum(_atoms(c) for c in cs) > 12e6:
                return None
            rs = [_trajectory(c, _crystal(c, c["seed"])) for c in cs]
            return {"obs": np.array([r["obs"] for r in rs]), "npt": np.array([r["npt"] for r in rs]),
                    **{k: np.concatenate([r[k] for r in rs]) for k in ("pos", "vel", "h")}}
        s = _crystal(case, seed)
        return _trajectory(case, s, _net(seed) if kind == "learned" else None)
