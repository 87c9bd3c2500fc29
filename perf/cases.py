"""Performance cases of the framework's main paths, through its public entry points.

Each case is a dict of plain values; ``prepare`` builds what a program has in
hand before the call, ``run`` makes one pass, ``exact`` gives the same outputs
in 64 bits from plain torch, written from the equations without this package.

Kinds of case:
  step   an RK4 step of one box, the state on the device (``evolve_rk_rk4``)
  rhs    the evolution callbacks of a host code that runs its own integrator:
         right-hand side and radiative boundary (``evolve_rhs``)
  host   an RK4 step of a state that lives in pinned host memory (``evolve_host``)
  fmr    a coarse step of a nested hierarchy (``Hierarchy.advance``)
  mg     coefficients and multigrid solve of a binary's puncture equation
  warm   the learned initial guess of that solve (network and smoothing)
  train  sixteen training steps of the network and its weights
  adm    ADM variables, constraints and their norms of one level
"""
import math

import numpy as np
import torch

from baum_b200 import abi, adm, bssn, fmr, punctures, warmstart, z4

F64 = torch.float64


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # the smallest evolution call: a 32^3 box, where launches and latency count
        dict(name="bssn_step_34", kind="step", system="bssn", m=34, n=34, o=34, dx=0.25, order=4, lop6=3, data="wave",
             tune=False),
        # the single-puncture BSSN box that the benchmark quotes, its launch shape tuned once as there
        dict(name="bssn_step_66", kind="step", system="bssn", m=66, n=66, o=66, dx=0.25, order=4, lop6=3,
             data="puncture", tune=True),
        # a host code's callbacks on a box of uneven sides, 6th order with lopsided advection
        dict(name="bssn_rhs_ragged_o6", kind="rhs", system="bssn", m=107, n=93, o=82, dx=0.3, order=6, lop6=2,
             data="wave", tune=False),
        # the benchmark's box stepped from and to host memory
        dict(name="bssn_host_66", kind="host", system="bssn", m=66, n=66, o=66, dx=0.25, order=4, lop6=3,
             data="puncture", tune=True),
        # the large 6th-order Z4c box of the benchmark: the throughput case
        dict(name="z4_step_162_o6", kind="step", system="z4", m=162, n=162, o=162, dx=0.15, order=6, lop6=3,
             data="puncture", tune=True),
        # a Z4c box of uneven, odd sides at the usual order
        dict(name="z4_step_ragged_o4", kind="step", system="z4", m=109, n=97, o=91, dx=0.25, order=4, lop6=3,
             data="wave", tune=False),
        # the three-level grid that is also timed against the reference: small levels, many launches
        dict(name="fmr_3_levels", kind="fmr", sizes="50-56-56", dx=0.5, order=4),
        # the batched seven-level grid of the benchmark, the largest call
        dict(name="fmr_7_levels", kind="fmr", sizes="162-136-168-104-136-72-104", dx=0.5, order=4),
        # a binary's initial data to the survey's tolerance on the benchmark's grid
        dict(name="mg_130", kind="mg", m=130, dx=0.25),
        # the guess that shortens that solve
        dict(name="warm_guess_130", kind="warm", m=130, dx=0.25),
        # training of the network behind the guess, at its batch size
        dict(name="mlp_train_16384", kind="train", rows=16384, m=130, dx=0.25),
        # the constraint monitoring of an output step
        dict(name="adm_constraints_104", kind="adm", m=104, n=104, o=104, dx=0.25, order=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    m = _log(rng, lo, hi)
    return {k: m if rng.random() < 0.3 else max(lo, min(hi, int(m * rng.uniform(0.8, 1.2)))) for k in "mno"}


def draw(rng):
    kind = rng.choice(["step", "step", "step", "rhs", "host", "fmr", "fmr", "mg", "warm", "train", "adm"])
    if kind in ("step", "rhs", "host"):
        system = "bssn" if kind == "host" else rng.choice(["bssn", "z4"])
        return dict(kind=kind, system=system, **_sides(rng, 20, 110 if kind == "host" else 168),
                    dx=round(rng.uniform(0.15, 0.5), 3), order=rng.choice([4, 4, 6]), lop6=rng.choice([2, 3]),
                    data=rng.choice(["wave", "puncture"]), tune=rng.random() < 0.5)
    if kind == "fmr":
        sizes = [4 * rng.randint(10, 24) + 2]
        while len(sizes) < rng.randint(2, 5):
            most = min(96, 2 * sizes[-1] - 12) // 4
            sizes.append(4 * rng.randint(min(8, most), most))
        return dict(kind=kind, sizes="-".join(map(str, sizes)), dx=rng.choice([0.25, 0.5, 1.0]), order=rng.choice([4, 6]))
    if kind == "mg":
        m = rng.choice([34, 66, 130])
        return dict(kind=kind, m=m, dx=round(32.0 / (m - 2) * rng.uniform(0.9, 1.1), 4))
    if kind == "warm":
        m = 4 * rng.randint(8, 32) + 2
        return dict(kind=kind, m=m, dx=round(32.0 / m, 4))
    if kind == "train":
        return dict(kind=kind, rows=64 * _log(rng, 14, 256), m=130, dx=0.25)
    return dict(kind="adm", **_sides(rng, 20, 136), dx=round(rng.uniform(0.1, 0.5), 3), order=rng.choice([2, 4, 6]))


# ---- inputs ---------------------------------------------------------------------
def _axes(m, n, o, dx):
    """x, y, z coordinates of a box centred on the origin, as (1, 1, m), (1, n, 1), (o, 1, 1)."""
    c = [(torch.arange(s, dtype=F64, device="cuda") - 0.5 * (s - 1)) * dx for s in (m, n, o)]
    return c[0].view(1, 1, -1), c[1].view(1, -1, 1), c[2].view(-1, 1, 1)


def _state(nv, xyz, data, seed, length=16.0):
    """An evolution state (nv, points): flat space or two punctures with precollapsed lapse, every field
    perturbed by eight sine modes of amplitude 1e-3 (gauge and gravitational waves)."""
    g = torch.Generator().manual_seed(int(seed))
    x, y, z = xyz
    unit = (0, 3, 5, 6, nv - 7)
    k = 2.0 * math.pi / length * (torch.randint(0, 5, (8, 3), generator=g) - 2).to(F64)
    c = (2.0 * torch.rand(nv, 8, generator=g, dtype=F64) - 1.0) * 1e-3
    ph = 2.0 * math.pi * torch.rand(nv, 8, generator=g, dtype=F64)
    shape = torch.broadcast_shapes(x.shape, y.shape, z.shape)
    u = torch.zeros((nv,) + shape, dtype=F64, device="cuda")
    for a in range(8):
        arg = float(k[a, 0]) * x + float(k[a, 1]) * y + float(k[a, 2]) * z
        s, co = torch.sin(arg), torch.cos(arg)
        for v in range(nv):
            u[v] += float(c[v, a] * torch.cos(ph[v, a])) * s + float(c[v, a] * torch.sin(ph[v, a])) * co
    for v in unit:
        u[v] += 1.0
    if data == "puncture":
        psi = torch.ones(shape, dtype=F64, device="cuda")
        for sign in (1.0, -1.0):
            off = sign * (1.0 + 0.2 * float(torch.rand(1, generator=g)))
            psi += 0.25 / torch.sqrt((x - off) ** 2 + y * y + z * z)
        u[6] *= psi ** -4
        u[nv - 7] *= psi ** -2
    return u.reshape(nv, -1)


def _level(case):
    m, n, o = case["m"], case["n"], case["o"]
    b = np.zeros((o, n, m), dtype=np.int32)
    b[0], b[-1], b[:, 0], b[:, -1], b[:, :, 0], b[:, :, -1] = (abi.PHYBOUND,) * 6
    h = case["dx"]
    return abi.Level([(m, n, o, -0.5 * (m - 1) * h, -0.5 * (n - 1) * h, -0.5 * (o - 1) * h)], h, b.ravel())


def _params(case, dissfactor=0.1 / 64):
    kw = dict(order_centered=case["order"], order_advection=case["order"], advection_lopsided6=case.get("lop6", 3),
              dissfactor=dissfactor)
    return abi.bssn_params(**kw) if case.get("system") == "bssn" else abi.z4_params_from_par(**kw)


def _sizes(case):
    return [int(s) for s in case["sizes"].split("-")]


def _diss(level):
    """The dissipation factor of a refinement level (0.1, and a fifth of it on the finer ones)."""
    return (0.1 if level == 0 else 0.02) / 64


def _binary(seed):
    """Two nearly equal punctures near x = +-4 with Bowen-York momenta and spins."""
    r = np.random.default_rng(int(seed))
    j = lambda s: 1.0 + s * r.uniform(-1, 1)  # noqa: E731
    spin = np.zeros((2, 3))
    spin[:, 2] = 0.1 * j(0.1), -0.1 * j(0.1)
    return punctures.Binary([0.5 * j(0.05), 0.5 * j(0.05)], [[4.0 * j(0.02), 0, 0], [-4.0 * j(0.02), 0, 0]],
                            [[0, 0.1 * j(0.1), 0], [0, -0.1 * j(0.1), 0]], spin)


TRAIN_STEPS, TRAIN_RATE = 16, 1e-4


def _train_inputs(case, seed):
    """Weights, conditions, and per step the rows' binaries, grid points and targets."""
    r = np.random.default_rng(int(seed))
    conds = np.stack([warmstart.cond_vector(punctures.Binary.sample(r)) for _ in range(64)])
    w = warmstart.init_params(r)
    n = TRAIN_STEPS * case["rows"]
    sets = r.integers(0, 64, n).astype(np.int32)
    pts = r.integers(0, case["m"] ** 3, n).astype(np.int32)
    f = _features(conds, sets, pts, case["m"], case["dx"])
    y = (0.3 * f[:, 7] + 0.3 * f[:, 19] + 0.1 * torch.sin(3.0 * f[:, 0])).float()
    return w, conds, torch.from_numpy(sets).cuda(), torch.from_numpy(pts).cuda(), y


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "rhs", "host"):
        nv = abi.NVARS if case["system"] == "bssn" else abi.Z4_NVARS
        lev = _level(case)
        s = dict(case=case, dl=bssn.DeviceLevel(lev), p=_params(case),
                 u=_state(nv, _axes(case["m"], case["n"], case["o"], case["dx"]), case["data"], seed))
        if case["tune"]:
            s["dl"].autotune(abi.SYSTEM_BSSN if case["system"] == "bssn" else abi.SYSTEM_Z4C, s["p"])
        if kind == "rhs":
            s["r"] = torch.zeros_like(s["u"])
        if kind == "host":
            s["u"] = s["u"].cpu().pin_memory()
        return s
    if kind == "fmr":
        sizes = _sizes(case)
        levels = fmr.nested_levels(sizes, case["dx"])
        dt = [0.25 * case["dx"] / 2 ** l for l in range(len(sizes))]
        return dict(case=case, h=fmr.Hierarchy(levels, dt, [_params(case, _diss(l)) for l in range(len(sizes))]),
                    u=_fmr_state(case, seed))
    if kind == "mg":
        return dict(case=case, mg=punctures.Multigrid(case["m"], case["dx"], abi.mg_params()), binary=_binary(seed))
    if kind == "warm":
        return dict(case=case, net=warmstart.Network.load(), binary=_binary(seed),
                    mg=punctures.Multigrid(case["m"], case["dx"], abi.mg_params(fullV=0)))
    if kind == "train":
        w, conds, sets, pts, y = _train_inputs(case, seed)
        net = warmstart.Network(case["rows"], w)
        net.set_conditions(conds)
        return dict(case=case, net=net, sets=sets, pts=pts, y=y)
    return dict(case=case, dl=bssn.DeviceLevel(_level(case)),
                u=_state(abi.Z4_NVARS, _axes(case["m"], case["n"], case["o"], case["dx"]), "wave", seed))


def _fmr_state(case, seed):
    sizes = _sizes(case)
    return [_state(abi.Z4_NVARS, _axes(m, m, m, case["dx"] / 2 ** l), "wave", seed) for l, m in enumerate(sizes)]


# ---- one pass -------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("step", "rhs", "host"):
        mod = bssn if c["system"] == "bssn" else z4
        if kind == "step":
            mod.evolve_rk_rk4(s["dl"], s["u"], 0.25 * c["dx"], s["p"])
            return s["u"]
        if kind == "rhs":
            mod.evolve_rhs(s["dl"], s["r"], s["u"], 0.0, s["u"], s["p"])
            return s["r"]
        return bssn.evolve_host(s["dl"], s["u"], 1, 0.25 * c["dx"], s["p"])
    if kind == "fmr":
        return s["h"].advance(s["u"], 1)
    if kind == "mg":
        a, b = s["mg"].coefficients(s["binary"])
        u = torch.zeros(c["m"] ** 3, dtype=F64, device="cuda")
        s["mg"].solve(a, b, u)
        return u
    if kind == "warm":
        return warmstart.warm_guess(s["net"], s["mg"], s["binary"], c["m"], c["dx"])
    if kind == "train":
        n = c["rows"]
        for t in range(TRAIN_STEPS):
            q = slice(t * n, (t + 1) * n)
            s["net"].features(s["sets"][q], s["pts"][q], c["m"], c["dx"])
            loss = s["net"].train_step(s["y"][q], TRAIN_RATE, want_loss=t == TRAIN_STEPS - 1)
        return {"weights": s["net"].params(), "loss": loss}
    a, con, norms = adm.computeadmconstraints(s["dl"], s["u"], c["order"])
    return {"adm": a, "con": con, "norms": np.array([norms[k] for k in sorted(norms)])}


# ---- what a pass cannot do without, and how exact it is ---------------------------
# operations of the right-hand side per point, counted in the reference's code
RHS_FLOPS = {("bssn", 4): 4973, ("bssn", 6): 6400, ("z4", 4): 6770, ("z4", 6): 8726}
NET_FLOPS = 2 * (32 * 128 + 3 * 128 * 128 + 128)


def work(case):
    kind = case["kind"]
    if kind in ("step", "rhs", "host"):
        nv = 24 if case["system"] == "bssn" else 25
        pts = case["m"] * case["n"] * case["o"]
        inner = (case["m"] - 2) * (case["n"] - 2) * (case["o"] - 2)
        return {"bytes": 2 * nv * 8 * pts, "flops": (1 if kind == "rhs" else 4) * RHS_FLOPS[case["system"], case["order"]] * inner}
    if kind == "fmr":
        sizes = _sizes(case)
        return {"bytes": sum(2 * 25 * 8 * m ** 3 * 2 ** l for l, m in enumerate(sizes)),
                "flops": sum(4 * RHS_FLOPS["z4", case["order"]] * (m - 2) ** 3 * 2 ** l for l, m in enumerate(sizes))}
    if kind == "mg":
        # about 300 V cycles of six sweeps and the transfers, each reading u, a, b, f and writing u
        return {"bytes": 300 * 7 * 8 / 7 * 40 * case["m"] ** 3, "flops": 300 * 7 * 8 / 7 * 45 * case["m"] ** 3}
    if kind == "warm":
        n = case["m"] ** 3
        return {"bytes": warmstart.NSMOOTH * 32 * n, "flops": (NET_FLOPS + warmstart.NSMOOTH * 45) * n}
    if kind == "train":
        return {"bytes": TRAIN_STEPS * case["rows"] * 12, "flops": TRAIN_STEPS * 3 * NET_FLOPS * case["rows"]}
    pts = case["m"] * case["n"] * case["o"]
    return {"bytes": (14 + 12 + 4) * 8 * pts, "flops": 3000 * pts}


def tolerance(case):
    kind = case["kind"]
    if kind in ("step", "host"):
        return {"rel": 1e-13, "max": 1e-9}   # sums of stencil terms in another order
    if kind == "fmr":
        return {"rel": 1e-13, "max": 1e-8}   # second differences of a unit background over dx^2 on the finest level
    if kind == "rhs":
        return {"rel": 2e-11, "max": 1e-7}   # the same relative to the derivatives alone
    if kind == "mg":
        return {"rel": 1e-5, "max": 1e-4}    # solved to a residual of 1e-10, the slow modes to less
    if kind == "warm":
        return {"rel": 2e-6, "max": 1e-4}    # 32-bit network
    if kind == "train":
        return {"rel": 1e-3, "max": 0.1}     # 16-bit products, sixteen steps of Adam
    return {"rel": 1e-9, "max": 1e-5}        # constraints: differences of nearly equal terms


# ---- the same in 64 bits, from the equations --------------------------------------
def _sh(f, a, n):
    """f at n points further along axis a (x: the last dimension); wraps at the ends, which no kept value uses."""
    return f if n == 0 else torch.roll(f, -n, -1 - a)


W1 = {2: [1 / 2], 4: [8 / 12, -1 / 12], 6: [45 / 60, -9 / 60, 1 / 60]}
W2 = {2: (-2.0, [1.0]), 4: (-30 / 12, [16 / 12, -1 / 12]), 6: (-490 / 180, [270 / 180, -27 / 180, 2 / 180])}
ADV = {2: ([[3, -4, 1], [1, 0, -1], [-1, 4, -3]], 2),
       4: ([[25, -48, 36, -16, 3], [3, 10, -18, 6, -1], [-1, 8, 0, -8, 1], [1, -6, 18, -10, -3], [-3, 16, -36, 48, -25]], 12),
       6: ([[147, -360, 450, -400, 225, -72, 10], [10, 77, -150, 100, -50, 15, -2], [-2, 24, 35, -80, 30, -8, 1],
            [1, -9, 45, 0, -45, 9, -1], [-1, 8, -30, 80, -35, -24, 2], [2, -15, 50, -100, 150, -77, -10],
            [-10, 72, -225, 400, -450, 360, -147]], 60)}


def _d1(f, a, q, h):
    return sum(w * (_sh(f, a, n) - _sh(f, a, -n)) for n, w in enumerate(W1[q], 1)) / h


def _d2(f, a, b, q, h):
    if a != b:
        return _d1(_d1(f, a, q, h), b, q, h)
    c, ws = W2[q]
    return (c * f + sum(w * (_sh(f, a, n) + _sh(f, a, -n)) for n, w in enumerate(ws, 1))) / (h * h)


def _full(t):
    """A symmetric tensor's six components as 3 x 3."""
    return t[[0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape((3, 3) + t.shape[1:])


def _six(t):
    return torch.stack([t[a, b] for a in range(3) for b in range(a, 3)])


def _ein(spec, *ops):
    """A sum over index letters, point by point: every combination added up term by term."""
    ins, out = spec.split("->")
    ins = ins.split(",")
    letters = sorted(set("".join(ins)))
    res = torch.zeros((3,) * len(out) + ops[0].shape[len(ins[0]):], dtype=F64, device=ops[0].device)
    for code in range(3 ** len(letters)):
        at, q = {}, code
        for s in letters:
            at[s], q = q % 3, q // 3
        t = None
        for i, x in zip(ins, ops):
            v = x[tuple(at[s] for s in i)]
            t = v if t is None else t * v
        res[tuple(at[s] for s in out)] += t
    return res


def _inverse(g):
    c = [torch.linalg.cross(g[(a + 1) % 3], g[(a + 2) % 3], dim=0) for a in range(3)]
    det = (g[0] * c[0]).sum(0)
    return torch.stack(c) / det, det


def _advect(f, w, q, lop):
    """sum over axes of the upwind derivative with lopsided rows, shifted further near the box's faces."""
    rows, den = ADV[q]
    lop = 0 if q == 2 else lop
    out = torch.zeros_like(f)
    for a in range(3):
        size = f.shape[-1 - a]
        i = torch.arange(size, device=f.device).view([-1 if d == 2 - a else 1 for d in range(3)])
        for s in (1, -1):
            room = size - 1 - i if s > 0 else i
            row = lop + (q - lop - room).clamp(min=0)
            for r in range(lop, q + 1):
                mask = (w[a] * s > 0) & (row == r)
                if bool(mask.any()):
                    t = sum(rows[r][n] * _sh(f, a, s * (n - r)) for n in range(q + 1) if rows[r][n])
                    out += torch.where(mask, -s / den * w[a], 0.0) * t
    return out


def _rhs(u, z4c, q, lop, h, e, dist):
    """The right-hand side at stencil order q over the whole box: 1+log lapse, Gamma-driver shift."""
    it = 18 if z4c else 17
    g, A, chi, Kh, G = _full(u[0:6]), _full(u[7:13]), u[6], u[13], u[14:17]
    al, be, B = u[it], u[it + 1:it + 4], u[it + 4:it + 7]
    Th = u[17] if z4c else torch.zeros_like(al)
    K = Kh + 2.0 * Th
    gi, _ = _inverse(g)
    d = lambda f: torch.stack([_d1(f, a, q, h) for a in range(3)])  # noqa: E731
    dd = lambda f: torch.stack([torch.stack([_d2(f, min(a, b), max(a, b), q, h) for b in range(3)]) for a in range(3)])  # noqa: E731
    dg = torch.stack([_full(_d1(u[0:6], a, q, h)) for a in range(3)])
    gdo = 0.5 * (torch.stack([torch.stack([torch.stack([dg[a, b, c] + dg[b, a, c] - dg[c, a, b] for b in range(3)])
                                           for a in range(3)]) for c in range(3)]))
    gam = _ein("cd,dab->cab", gi, gdo)
    Gg = _ein("bc,abc->a", gi, gam)
    R = torch.zeros_like(g)
    for a in range(3):
        for b in range(3):
            R -= 0.5 * gi[a, b] * _full(_d2(u[0:6], min(a, b), max(a, b), q, h))
    R += _ein("cd,eca,bed->ab", gi, gam, gdo) + _ein("cd,ecb,aed->ab", gi, gam, gdo) + _ein("cd,ead,ecb->ab", gi, gam, gdo)
    dG = d(G)
    t = _ein("ca,bc->ab", g, dG) + _ein("c,abc->ab", Gg, gdo)
    R += 0.5 * (t + t.transpose(0, 1))
    # conformal factor chi = psi^-4
    dchi = d(chi)
    df = -0.25 * dchi / chi
    cddf = -0.25 * dd(chi) / chi + 4.0 * df[:, None] * df[None] - _ein("cab,c->ab", gam, df)
    R += 4.0 * df[:, None] * df[None] - 2.0 * cddf - 2.0 * g * (_ein("ab,ab->", gi, cddf) + 2.0 * _ein("ab,a,b->", gi, df, df))
    psim4 = chi
    da = d(al)
    cdda = dd(al) - _ein("cab,c->ab", gam, da) - 2.0 * (df[:, None] * da[None] + da[:, None] * df[None] -
                                                        g * _ein("ab,a,b->", gi, df, da))
    tra = psim4 * _ein("ab,ab->", gi, cdda)
    AA = _ein("cd,ac,db->ab", gi, A, A)
    Ai = _ein("ac,bd,cd->ab", gi, gi, A)
    AAs = _ein("ab,ab->", gi, AA)
    Rs = psim4 * _ein("ab,ab->", gi, R) if z4c else AAs - 2.0 * K * K / 3.0
    db = d(be)
    div = db[0, 0] + db[1, 1] + db[2, 2]
    lie = lambda t: _ein("ac,bc->ab", db, t) + _ein("bc,ac->ab", db, t) - 2.0 / 3.0 * div * t  # noqa: E731
    rg = -2.0 * al * A + lie(g)
    rA = psim4 * (al * R - cdda) - g / 3.0 * (al * Rs - tra) + al * (K * A - 2.0 * AA) + lie(A)
    rK = -tra + al * (AAs + K * K / 3.0)
    rchi = 2.0 / 3.0 * chi * (al * K - div)
    dv = _ein("abc,bc->a", gam, Ai) - 1.5 * _ein("ab,b->a", Ai, dchi / chi)
    if z4c:
        k1 = 0.02
        rK = rK + k1 * al * Th
        rT = al * (0.5 * (Rs + 2.0 * K * K / 3.0 - AAs) - 2.0 * k1 * Th)
        dv = dv - _ein("ab,b->a", gi, 2.0 * d(Kh) + d(Th)) / 3.0
        rG = 2.0 * al * dv - 2.0 * al * k1 * (G - Gg)
    else:
        rG = 2.0 * al * (dv - 2.0 / 3.0 * _ein("ab,b->a", gi, d(K)))
    rG = rG - 2.0 * _ein("ab,b->a", Ai, da) + 2.0 / 3.0 * Gg * div - _ein("b,ba->a", Gg, db)
    ddb = torch.stack([torch.stack([_d2(be, min(a, b), max(a, b), q, h) for b in range(3)]) for a in range(3)])
    ddiv = torch.stack([sum(ddb[a, b, b] for b in range(3)) for a in range(3)])
    rG = rG + _ein("bc,bca->a", gi, ddb) + _ein("ab,b->a", gi, ddiv) / 3.0
    adv = _advect(u, be / h, q, lop)
    r = torch.zeros_like(u)
    r[0:6], r[7:13], r[6], r[13], r[14:17], r[it] = _six(rg), _six(rA), rchi, rK, rG, -2.0 * al * Kh
    if z4c:
        # the shift string of the refinement workload switches B off: its token test reads withBadv first
        r[17] = rT
        r[it + 1:it + 4] = G - 2.0 * be
        adv[it + 4:it + 7] = 0.0
    else:
        r[it + 1:it + 4] = 0.75 * B
        r[it + 4:it + 7] = rG - 2.0 * B
    r += adv
    ko = sum(_sh(u, a, 3) + _sh(u, a, -3) - 6.0 * (_sh(u, a, 2) + _sh(u, a, -2)) + 15.0 * (_sh(u, a, 1) + _sh(u, a, -1)) -
             20.0 * u for a in range(3)) / h
    if not z4c:
        ko[17:] = 0.0
    return r + torch.where(dist >= 3, e, 0.0) * ko


def _radiative(u, z4c, h, xyz, faces):
    """Outgoing waves on the outer layer: -v (u - u0)/r - v x/r . d u, one-sided second-order differences."""
    nv = u.shape[0]
    v = torch.ones(nv, 1, dtype=F64, device="cuda")
    v[[6, 13, nv - 7]] = math.sqrt(2.0)
    u0 = torch.zeros_like(v)
    u0[[0, 3, 5, 6, nv - 7]] = 1.0
    k, j, i = faces
    x = [xyz[0].reshape(-1)[i], xyz[1].reshape(-1)[j], xyz[2].reshape(-1)[k]]
    r = torch.sqrt(x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
    c = u[:, k, j, i]
    rhs = -v * (c - u0) / r
    for a, at in enumerate((i, j, k)):
        size = u.shape[-1 - a]

        def tap(n):
            p = (at + n).clamp(0, size - 1)
            return u[:, k, j, p] if a == 0 else u[:, k, p, i] if a == 1 else u[:, p, j, i]
        lo, mid, hi = 3.0 * c + tap(-2) - 4.0 * tap(-1), tap(1) - tap(-1), 4.0 * tap(1) - tap(2) - 3.0 * c
        up = torch.where(at > 1, lo, torch.where(at > 0, mid, hi))
        down = torch.where(at < size - 2, hi, torch.where(at > 0, mid, lo))
        flat = torch.where((at > 0) & (at < size - 1), mid, torch.where(at == 0, hi, lo))
        W = v * x[a] / r
        rhs -= W * torch.where(W > 0, up, torch.where(W < 0, down, flat)) / (2.0 * h)
    return rhs


class _Box:
    """One box of the 64-bit evolution: the state u as (variables, o, n, m)."""

    def __init__(self, u, z4c, m, n, o, h, order, lop6, e, physical=True):
        self.u, self.z4c, self.h, self.order, self.lop6, self.e = u.reshape(-1, o, n, m), z4c, h, order, lop6, e
        self.xyz, self.physical = _axes(m, n, o, h), physical
        i = [torch.arange(s, device="cuda") for s in (m, n, o)]
        d = [torch.minimum(a, a.flip(0)) for a in i]
        self.dist = torch.minimum(torch.minimum(d[0].view(1, 1, -1), d[1].view(1, -1, 1)), d[2].view(-1, 1, 1))
        self.faces = torch.nonzero(self.dist == 0, as_tuple=True)

    def rhs(self, u):
        r = torch.zeros_like(u)
        for q in range(2, self.order + 1, 2):
            mask = self.dist >= q // 2 if q == self.order else self.dist == q // 2
            if bool(mask.any()):
                r = torch.where(mask, _rhs(u, self.z4c, q, self.lop6 if q == 6 else 1, self.h, self.e, self.dist), r)
        k, j, i = self.faces
        if self.physical:
            r[:, k, j, i] = _radiative(u, self.z4c, self.h, self.xyz, self.faces)
        return r

    def rk4(self, dt):
        acc = self.u.clone()
        v = self.u
        for c, w in ((0.5, 6), (0.5, 3), (1.0, 3), (0.0, 6)):
            r = self.rhs(v)
            acc += dt / w * r
            v = self.u + c * dt * r
        self.u = acc

    def constrain(self):
        """Unit determinant of the conformal metric, then a trace-free A."""
        g = self.u[0:6]
        g *= _inverse(_full(g))[1] ** (-1.0 / 3.0)
        gi, _ = _inverse(_full(g))
        self.u[7:13] -= _ein("ab,ab->", gi, _full(self.u[7:13])) / 3.0 * g


def _lagrange(n, x):
    return torch.tensor([math.prod((x - j) / (i - j) for j in range(n) if j != i) for i in range(n)], dtype=F64, device="cuda")


def _along(mat, f, a):
    return torch.movedim(torch.tensordot(f, mat, ([f.dim() - 1 - a], [1])), -1, f.dim() - 1 - a)


class _Nest:
    """Berger-Oliger steps of centred nested cubes: fourth-order Lagrange transfer, third-order in time."""

    def __init__(self, case, u):
        self.m = _sizes(case)
        self.box = [_Box(u[l], True, m, m, m, case["dx"] / 2 ** l, case["order"], 3, _diss(l), l == 0)
                    for l, m in enumerate(self.m)]
        self.dt = [0.25 * case["dx"] / 2 ** l for l in range(len(self.m))]
        self.it, self.prev, self.mid = [0] * len(self.m), [None] * len(self.m), [None] * len(self.m)

    def step(self, l):
        b = self.box[l]
        u = b.u.clone()
        b.rk4(self.dt[l])
        self.mid[l] = 0.5 * u + 0.5 * b.u if self.it[l] == 0 else 0.75 * u - 0.125 * self.prev[l] + 0.375 * b.u
        self.prev[l] = u
        b.constrain()
        self.it[l] += 1

    def transfer(self, l, uc):
        """The fine level's interior into uc, then the fine level's outer points from uc."""
        m, mc = self.m[l], self.m[l - 1]
        p0 = (2 * mc - m + 1) // 4             # the parent point of the fine points 0 and 1
        half = m // 2
        R = torch.zeros(half - 4, m, dtype=F64, device="cuda")
        for t in range(half - 4):
            R[t, 2 * t + 3:2 * t + 7] = _lagrange(4, 1.5)
        f = self.box[l].u
        lo, hi = p0 + 2, p0 + half - 2
        uc[:, lo:hi, lo:hi, lo:hi] = _along(R, _along(R, _along(R, f, 2), 1), 0)
        P = torch.zeros(m, mc, dtype=F64, device="cuda")
        first = (2 * mc - m - 1) // 4 - 1
        for t in range(m):
            s = first + t // 2 + t % 2
            P[t, s:s + 4] = _lagrange(4, 1.25 if t % 2 else 1.75)
        q = torch.arange(m, device="cuda")
        inner = (q >= 3) & (q <= m - 4)
        pair = 2 * (q // 2)
        keep = ((pair >= 3) & (pair <= m - 4)).view(1, 1, -1) & inner.view(1, -1, 1) & inner.view(-1, 1, 1)
        self.box[l].u = torch.where(keep, f, _along(P, _along(P, _along(P, uc, 2), 1), 0))

    def advance(self, l=0):
        self.step(l)
        if l + 1 < len(self.m):
            self.advance(l + 1)
            self.advance(l + 1)
        if l > 0:
            aligned = abs(self.it[l] * self.dt[l] - self.it[l - 1] * self.dt[l - 1]) < 1e-10
            self.transfer(l, self.box[l - 1].u if aligned else self.mid[l - 1])


def _puncture(m, dx, b):
    """a = 1/(psi - 1) and b = a^7 K_ij K^ij / 8 of Brill-Lindquist and Bowen-York."""
    xyz = _axes(m, m, m, dx)
    p = 0.0
    K = [[0.0] * 3 for _ in range(3)]
    for mass, pos, P, S in zip(b.mass, b.pos, b.mom, b.spin):
        x = [xyz[a] - float(pos[a]) for a in range(3)]
        r = torch.sqrt(x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
        p = p + 0.5 * float(mass) / r
        n = [v / r for v in x]
        nP = sum(n[a] * float(P[a]) for a in range(3))
        e = [n[(a + 1) % 3] * float(S[(a + 2) % 3]) - n[(a + 2) % 3] * float(S[(a + 1) % 3]) for a in range(3)]
        for s in range(3):
            for t in range(3):
                K[s][t] = K[s][t] + 1.5 / r ** 2 * (n[s] * float(P[t]) + n[t] * float(P[s]) - (float(s == t) - n[s] * n[t]) * nP) - \
                    3.0 / r ** 3 * (e[s] * n[t] + e[t] * n[s])
    a = 1.0 / p
    return a, 0.125 * a ** 7 * sum(K[s][t] ** 2 for s in range(3) for t in range(3))


class _Elliptic:
    """Laplace u + b (1 + a (1 + u))^-7 on the inner points of a cube; the outer layer follows its most inward
    inner neighbour by the Robin condition of a 1/r falloff."""

    def __init__(self, m, dx, binary):
        self.m, self.dx = m, dx
        self.a, self.b = _puncture(m, dx, binary)
        q = torch.arange(m, device="cuda")
        edge = (q == 0) | (q == m - 1)
        self.out = edge.view(1, 1, -1) | edge.view(1, -1, 1) | edge.view(-1, 1, 1)
        at = torch.stack(torch.nonzero(self.out, as_tuple=True)).flip(0)      # x, y, z indices
        offs = [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1) if i or j or k]
        unit = [torch.tensor(o, dtype=F64, device="cuda") / math.sqrt(sum(c * c for c in o)) for o in offs]
        inside = [((at + torch.tensor(o, device="cuda").view(3, 1) >= 1) & (at + torch.tensor(o, device="cuda").view(3, 1) <= m - 2)).all(0)
                  for o in offs]
        mean = sum(torch.where(s, u.view(3, 1), 0.0) for s, u in zip(inside, unit))
        best, to = torch.zeros(at.shape[1], dtype=F64, device="cuda"), at.clone()
        for o, u, s in zip(offs, unit, inside):
            dot = (mean * u.view(3, 1)).sum(0)
            better = s & (dot > best + 1e-12)
            best, to = torch.where(better, dot, best), torch.where(better, at + torch.tensor(o, device="cuda").view(3, 1), to)
        x1, x0 = (at - 0.5 * (m - 1)) * dx, (to - 0.5 * (m - 1)) * dx
        mid = 0.5 * (x1 + x0)
        c = 0.5 * ((x1 - x0) * mid).sum(0) / (mid * mid).sum(0)
        flat = lambda p: p[0] + m * (p[1] + m * p[2])  # noqa: E731
        self.dst, self.src, self.fac = flat(at), flat(to), (1.0 - c) / (1.0 + c)

    def robin(self, u):
        v = u.reshape(-1)
        v[self.dst] = self.fac * v[self.src]
        return u

    def laplace(self, u):
        return (sum(_sh(u, a, 1) + _sh(u, a, -1) for a in range(3)) - 6.0 * u) / self.dx ** 2

    def residual(self, u):
        return torch.where(self.out, 0.0, self.laplace(u) + self.b * (1.0 + self.a * (1.0 + u)) ** -7)

    def slope(self, u):
        return -7.0 * self.a * self.b * (1.0 + self.a * (1.0 + u)) ** -8

    def smooth(self, u, n, omega):
        for _ in range(n):
            u = self.robin(u + torch.where(self.out, 0.0, omega * -self.residual(u) / (-6.0 / self.dx ** 2 + self.slope(u))))
        return u

    def solve(self):
        """Newton steps, each by BiCGStab."""
        u = torch.zeros((self.m,) * 3, dtype=F64, device="cuda")
        for _ in range(6):
            f, s = -self.residual(u), self.slope(u)
            if float(f.norm()) < 1e-11 * self.m ** 1.5:
                break
            A = lambda v: torch.where(self.out, 0.0, self.laplace(self.robin(v.clone())) + s * v)  # noqa: E731
            x, r = torch.zeros_like(f), f.clone()
            r0, p, rho, stop = r.clone(), r.clone(), (r * r).sum(), 1e-10 * float(f.norm())
            for it in range(4000):
                v = A(p)
                alpha = rho / (r0 * v).sum()
                t = r - alpha * v
                w = A(t)
                om = (w * t).sum() / (w * w).sum()
                x, r = x + alpha * p + om * t, t - om * w
                if it % 10 == 0 and float(r.norm()) < stop:
                    break
                new = (r0 * r).sum()
                p, rho = r + new / rho * alpha / om * (p - om * v), new
            u = self.robin(u + x)
        return u.reshape(-1)


def _features(conds, sets, pts, m, dx):
    """Network inputs of grid points: position, and per puncture offset, distance, mass terms, momentum, spin."""
    c = torch.as_tensor(conds, dtype=F64, device="cuda")[torch.as_tensor(sets, device="cuda").long()]
    p = torch.as_tensor(pts, device="cuda").long()
    x = (torch.stack([p % m, p // m % m, p // (m * m)], 1) - 0.5 * (m - 1)) * dx
    f = [x / 8.0]
    for q in range(2):
        d = x - c[:, 2 + 3 * q:5 + 3 * q]
        r = d.norm(dim=1, keepdim=True)
        mass = c[:, q:q + 1]
        f += [d / 8.0, r / 8.0, mass / (r + mass), 2.0 * mass, 5.0 * c[:, 8 + 3 * q:11 + 3 * q], 5.0 * c[:, 14 + 3 * q:17 + 3 * q]]
    f = torch.cat(f, 1)
    return torch.nn.functional.pad(f, (0, 32 - f.shape[1]))


def _unpack(w):
    out, at = [], 0
    for k, n in ((32, 128), (128, 128), (128, 128), (128, 128), (128, 1)):
        out.append((w[at:at + k * n].view(k, n), w[at + k * n:at + k * n + n]))
        at += k * n + n
    return out


def _network(w, x):
    layers = _unpack(w)
    for W, b in layers[:-1]:
        x = torch.nn.functional.silu(x @ W + b)
    return (x @ layers[-1][0] + layers[-1][1])[:, 0]


def _warm(case, seed):
    m, dx, b = case["m"], case["dx"], _binary(seed)
    z = np.load(warmstart.WEIGHTS)
    w = torch.from_numpy(np.asarray(z["params"], dtype=np.float64)).cuda()
    cond = np.concatenate([b.mass, b.pos.ravel(), b.mom.ravel(), b.spin.ravel()])[None]
    u = torch.cat([_network(w, _features(cond, torch.zeros_like(p), p, m, dx))
                   for p in torch.arange(m ** 3, device="cuda").split(1 << 18)]) * float(z["uscale"])
    e = _Elliptic(m, dx, b)
    return e.smooth(u.view(m, m, m), warmstart.NSMOOTH, warmstart.OMEGA).reshape(-1)


def _train(case, seed):
    w, conds, sets, pts, y = _train_inputs(case, seed)
    w = torch.from_numpy(w).cuda().double()
    mo, vo, n = torch.zeros_like(w), torch.zeros_like(w), case["rows"]
    for t in range(TRAIN_STEPS):
        q = slice(t * n, (t + 1) * n)
        w.requires_grad_(True)
        loss = ((_network(w, _features(conds, sets[q], pts[q], case["m"], case["dx"])) - y[q].double()) ** 2).mean()
        g, = torch.autograd.grad(loss, w)
        w = w.detach()
        mo, vo = 0.9 * mo + 0.1 * g, 0.999 * vo + 0.001 * g * g
        w = w - TRAIN_RATE * (mo / (1 - 0.9 ** (t + 1))) / (torch.sqrt(vo / (1 - 0.999 ** (t + 1))) + 1e-8)
    return {"weights": w, "loss": float(loss)}


def _constraints(g6, K6, q, h):
    """Hamiltonian and momentum constraints of the metric and extrinsic curvature at stencil order q."""
    g, K = _full(g6), _full(K6)
    gi, _ = _inverse(g)
    dg = torch.stack([_full(_d1(g6, a, q, h)) for a in range(3)])
    dK = torch.stack([_full(_d1(K6, a, q, h)) for a in range(3)])
    ddg = torch.stack([torch.stack([_full(_d2(g6, min(a, b), max(a, b), q, h)) for b in range(3)]) for a in range(3)])
    gd = 0.5 * torch.stack([torch.stack([torch.stack([dg[a, b, c] + dg[b, a, c] - dg[c, a, b] for b in range(3)])
                                         for a in range(3)]) for c in range(3)])
    gu = _ein("cd,dab->cab", gi, gd)
    R = torch.zeros_like(g)
    for a in range(3):
        for b in range(3):
            for c in range(3):
                for d in range(3):
                    R[a, b] += 0.5 * gi[c, d] * (ddg[b, c, a, d] + ddg[a, c, b, d] - ddg[c, d, a, b] - ddg[a, b, c, d])
    Gt = _ein("cd,ecd->e", gi, gd)
    R += _ein("cd,eac,ebd->ab", gi, gu, gd) - _ein("eab,e->ab", gu, Gt)
    ham = _ein("ab,ab->", gi, R) + _ein("ab,ab->", gi, K) ** 2 - _ein("ac,bd,ab,cd->", gi, gi, K, K)
    cK = dK - _ein("dab,dc->abc", gu, K) - _ein("dac,bd->abc", gu, K)
    mom = _ein("bc,cab->a", gi, cK) - _ein("bc,abc->a", gi, cK)
    return torch.cat([ham[None], mom])


def _adm(case, seed):
    m, n, o, h = case["m"], case["n"], case["o"], case["dx"]
    u = _state(25, _axes(m, n, o, h), "wave", seed).reshape(25, o, n, m)
    g = u[0:6] / u[6]
    K = u[7:13] / u[6] + u[13] * g / 3.0
    box = _Box(u, True, m, n, o, h, case["order"], 3, 0.0)
    con = torch.zeros(4, o, n, m, dtype=F64, device="cuda")
    for q in range(2, case["order"] + 1, 2):
        mask = box.dist >= q // 2 if q == case["order"] else box.dist == q // 2
        if bool(mask.any()):
            con = torch.where(mask, _constraints(g, K, q, h), con)
    v = con[:, box.dist > 0]
    n2, ni = v.square().mean(1).sqrt(), v.abs().amax(1)
    return {"adm": torch.cat([g, K]).reshape(12, -1), "con": con.reshape(4, -1),
            "norms": torch.stack([n2, ni], 1).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "rhs", "host"):
        z4c = case["system"] == "z4"
        m, n, o, h = case["m"], case["n"], case["o"], case["dx"]
        u = _state(25 if z4c else 24, _axes(m, n, o, h), case["data"], seed)
        nv = u.shape[0]
        b = _Box(u, z4c, m, n, o, h, case["order"], case["lop6"], 0.1 / 64)
        if kind == "rhs":
            return b.rhs(b.u).reshape(nv, -1)
        b.rk4(0.25 * h)
        b.constrain()
        return b.u.reshape(nv, -1)
    if kind == "fmr":
        if sum(m ** 3 * 2 ** l for l, m in enumerate(_sizes(case))) > 2e7:
            return None
        nest = _Nest(case, _fmr_state(case, seed))
        nest.advance()
        return [b.u.reshape(b.u.shape[0], -1) for b in nest.box]
    if kind == "mg":
        return _Elliptic(case["m"], case["dx"], _binary(seed)).solve()
    if kind == "warm":
        return _warm(case, seed)
    if kind == "train":
        return _train(case, seed)
    return _adm(case, seed)
