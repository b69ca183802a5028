"""The work that users of the framework have it do, as measurable cases.

Five kinds of call, each through a public entry point:

  steps    a run in progress: the state goes up from page-locked host arrays,
           `steps` time steps are made on the tree it has, the state comes
           back.  The tree and state are those of an FP64 run advanced
           `develop` steps from the initial condition (the remesh is then
           switched off, as a caller does who remeshes at intervals).
  frozen   the same for the uniform Kelvin-Helmholtz mesh (maxlevs 1).
  adjoint  forward steps of the uniform mesh with checkpoints, then their
           discrete adjoint: the gradient of a linear loss.
  program  a whole small program: handle, initial condition, time steps with
           the remesh after each, the state read back.
  cfl      the allocation-free CFL reduction on the caller's device arrays.
  riemann  Riemann fluxes of host arrays of face states.

Seeds choose the state (the strength of the flow and its pressure, the
perturbation amplitudes, the face states); nothing else is random, and a
case's trees are the same for every seed.
"""
import ctypes
import math
import random

import numpy as np
import torch

import amr2d_mhd_gb300 as amr

# leaf blocks of one instance after the develop steps below, for work()
LEAVES = {("rotor", 3): 28, ("rotor", 4): 100, ("rotor", 5): 196, ("blast", 0): 140, ("OT", 2): 64,
          ("OT", 3): 256, ("BWx", 3): 40, ("BWx", 4): 88, ("BWy", 3): 40, ("SST", 3): 40}
BLAST_BATCH = 20261205   # the batch whose instances the blast cases take
# floating-point operations per cell and RK stage (both face directions):
# reconstruction + solver, counted from the formulas
RECON_FLOPS = {"MUSCL": 7 * 2 * 22, "WENO3": 7 * 2 * 50, "WENO5": 7 * 2 * 120}
FLUX_FLOPS = {"RUSA": 2 * 250, "HLLE": 2 * 350, "HLLC": 2 * 420, "HLLD": 2 * 480}


def recon_of(limiter):
    return limiter if limiter in ("WENO3", "WENO5") else "MUSCL"


def listed():
    return [
        # the time-step limit of a handful of blocks inside a caller's own loop: launch latency
        dict(name="cfl_64_blocks", kind="cfl", blocks=64, nghosts=2),
        # the same over a large mesh the caller owns (20011 blocks, 0.5 GB)
        dict(name="cfl_20011_blocks", kind="cfl", blocks=20011, nghosts=2),
        # riemannS as a service for another solver's face states (host arrays)
        dict(name="riemann_hlld_100003", kind="riemann", flux="HLLD", dir_y=0, n=100003),
        # the reference's example program: Brio-Wu, 3 levels, from the initial condition, remesh every step
        dict(name="brio_wu_program", kind="program", ic="BWx", limiter="MC", flux="RUSA", levels=3, nghosts=2, steps=30),
        # the headline benchmark: the 5-level rotor, MC + HLLD, plain FP64 path, autotuned
        dict(name="rotor_fp64", kind="steps", ic="rotor", limiter="MC", flux="HLLD", levels=5, precision="fp64",
             instances=1, develop=200, steps=4, tune=True),
        # the same in the FP32 bulk path
        dict(name="rotor_fp32", kind="steps", ic="rotor", limiter="MC", flux="HLLD", levels=5, precision="fp32",
             instances=1, develop=200, steps=10, tune=True),
        # a batch of rotors in one handle (parameter study), FP32
        dict(name="rotor_batch_fp32", kind="steps", ic="rotor", limiter="MC", flux="HLLD", levels=5,
             precision="fp32", instances=32, develop=200, steps=12, tune=True),
        # the seeded blast batch: uneven trees of 3 to 6 levels, HLLE, FP32
        dict(name="blast_batch_fp32", kind="steps", ic="blast", limiter="MC", flux="HLLE", levels=0,
             precision="fp32", instances=24, develop=16, steps=10, tune=True),
        # Orszag-Tang, WENO5 with four ghost layers, FP64, default schedule
        dict(name="ot_weno5_fp64", kind="steps", ic="OT", limiter="WENO5", flux="HLLD", levels=3, precision="fp64",
             instances=1, develop=12, steps=2, tune=False),
        # uniform 256^2 Kelvin-Helmholtz layer, Rusanov, FP64, default schedule
        dict(name="kh_256_fp64", kind="frozen", roots=16, precision="fp64", limiter="MC", steps=4, tune=False),
        # uniform 512^2 in the FP32 bulk path, autotuned
        dict(name="kh_512_fp32", kind="frozen", roots=32, precision="fp32", limiter="MC", steps=8, tune=True),
        # gradient through 3 steps of a smooth flow on the 256^2 mesh: recorded forward steps and their adjoint
        dict(name="kh_256_adjoint", kind="adjoint", roots=16, limiter="MC", steps=3),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# initial condition, limiter, solver, levels, ghost layers: combinations that run for many steps at CFL 0.4
PROGRAMS = [("BWx", "MC", "RUSA", 4, 2), ("BWx", "MC", "HLLE", 4, 2), ("BWx", "MC", "HLLC", 4, 2),
            ("BWy", "minmod", "HLLD", 3, 2), ("SST", "Superbee", "HLLE", 3, 2), ("BWx", "WENO3", "RUSA", 3, 2),
            ("BWx", "WENO5", "HLLD", 3, 4), ("rotor", "MC", "HLLD", 5, 2), ("rotor", "WENO5", "RUSA", 3, 4),
            ("rotor", "MC", "RUSA", 5, 2)]


def draw(rng):
    kind = rng.choice(["cfl", "riemann", "program", "steps", "steps", "steps", "frozen", "adjoint"])
    if kind == "cfl":
        return dict(kind=kind, blocks=log_int(rng, 32, 16000), nghosts=rng.choice([2, 2, 4]))
    if kind == "riemann":
        return dict(kind=kind, flux=rng.choice(["RUSA", "HLLE", "HLLC", "HLLD"]), dir_y=rng.randrange(2),
                    n=log_int(rng, 500, 200000))
    if kind == "program":
        ic, lim, fl, lev, ng = rng.choice(PROGRAMS)
        return dict(kind=kind, ic=ic, limiter=lim, flux=fl, levels=lev, nghosts=ng, steps=rng.randrange(12, 41))
    precision = rng.choice(["fp64", "fp32"])
    if kind == "steps":
        ic = rng.choice(["rotor", "blast", "OT"])
        n, dev, lev, lim, fl = 1, 12, 3, "MC", "HLLD"
        if ic == "rotor":
            lev, lim, fl = rng.randrange(3, 6), rng.choice(["MC", "minmod", "VanLeer"]), rng.choice(["HLLD", "HLLE", "RUSA"])
            dev = rng.randrange(30, 200)
            n = log_int(rng, 1, 24 if precision == "fp32" else 3)
        elif ic == "blast":
            lev, lim, fl, dev = 0, "MC", "HLLE", rng.randrange(10, 20)
            n = log_int(rng, 2, 20 if precision == "fp32" else 6)
        else:
            lev, lim = rng.randrange(2, 4), rng.choice(["MC", "WENO3", "WENO5"])
        return dict(kind=kind, ic=ic, limiter=lim, flux=fl, levels=lev, precision=precision, instances=n, develop=dev,
                    steps=rng.randrange(1, 9), tune=rng.random() < 0.5)
    if kind == "frozen":
        return dict(kind=kind, roots=rng.randrange(4, 33), precision=precision, limiter=rng.choice(["MC", "minmod"]),
                    steps=rng.randrange(1, 9), tune=rng.random() < 0.5)
    return dict(kind=kind, roots=rng.randrange(4, 21), limiter=rng.choice(["MC", "minmod"]), steps=rng.randrange(1, 4))


# ------------------------------------------------------------- configurations
def step_configs(case, precision):
    out = []
    for q in range(case["instances"]):
        if case["ic"] == "blast":
            c = amr.blast_config(BLAST_BATCH, q, precision)
        elif case["ic"] == "OT":
            c = amr.ot_config(maxlevs=case["levels"], precision=precision, cfl=0.35, limiter=case["limiter"])
        else:
            c = amr.make_config(ic=case["ic"], limiter=case["limiter"], flux=case["flux"], cfl=0.35,
                                maxlevs=case["levels"], geometry=1, gamma=5.0 / 3.0, precision=precision)
        c.t_end = 1e9
        out.append(c)
    return out


def kh_config(case, seed, precision):
    c = amr.kh_config(seed, precision)
    c.nroots_x = c.nroots_y = case["roots"]
    c.limiter = case["limiter"].encode()
    c.dt_fixed = 2e-4 * 16 / case["roots"]
    c.t_end = 1e9
    return c


def pinned(n):
    return torch.empty(int(n), dtype=torch.float64, pin_memory=True)


class Run:
    """A handle with its page-locked upload and download arrays."""

    def __init__(self, sim, states, precision, steps):
        self.sim, self.steps, self.precision = sim, steps, precision
        self.up, self.down, self.flat = [], [], {}
        for f in ("U", "Bi"):
            sizes = [s[f].size for s in states]
            src, dst = pinned(sum(sizes)), pinned(sum(sizes))
            self.flat[f] = dst
            at = 0
            for q, s in enumerate(states):
                a, b = (t[at:at + sizes[q]].view(s[f].shape).numpy() for t in (src, dst))
                a[...] = s[f]
                self.up.append((f, q, a))
                self.down.append((f, q, b))
                at += sizes[q]

    def upload(self):
        for f, q, a in self.up:
            self.sim.upload(f, a, q)

    def download(self):
        for f, q, b in self.down:
            self.sim.download(f, q, out=b)
        out = {}
        for f, t in self.flat.items():
            # the FP32 path's state as FP32, on the GPU (for analysis there); FP64 as it came
            out[f] = t.to("cuda", non_blocking=True).to(torch.float32) if self.precision == "fp32" else t
        return out

    def download_uniform(self):
        """The same with the blocks' interiors beside it (views): ghost corners no stencil reads hold old values."""
        out = self.download()
        return dict(out, **{"inner_" + f: t.view(-1, 8 if f == "U" else 2, 20, 20)[:, :, 2:18, 2:18] for f, t in out.items()})


def developed(case, seed):
    """Trees, time state and fields of the FP64 run after the develop steps (one rotor serves all copies), with the
    seed's factor on the momenta and its share added to the energy."""
    r = random.Random(1000003 * seed + 17)
    faster, hotter = 1 + 0.05 * (2 * r.random() - 1), 0.05 * r.random()
    cfgs = step_configs(case, "fp64")
    copies = case["ic"] != "blast"
    dev = amr.Simulation(cfgs[:1] if copies else cfgs).init()
    dev.run(case["develop"])
    out = []
    for q in range(1 if copies else len(cfgs)):
        s = {f: dev.download(f, q) for f in ("U", "Bi", "ff", "gg")}
        s["tree"], s["info"] = dev.tree(q), dev.info(q)
        U = s["U"]
        with np.errstate(all="ignore"):   # blocks that are no leaves may never have been written
            m2 = np.where(U[:, 0] > 0, (U[:, 1:4] ** 2).sum(1) / U[:, 0], 0.0)
        U[:, 4] += 0.5 * (faster ** 2 - 1) * m2 + hotter * U[:, 4]
        U[:, 1:4] *= faster
        out.append(s)
    return out * case["instances"] if copies else out


def smooth_flow(case, seed):
    """A smooth periodic state on [0, 1]^2 with every variable varying and the face field free of divergence:
    U [8, n, n], Bx, By."""
    r, n = random.Random(104729 * seed + 3), 16 * case["roots"]
    k = 2 * math.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n

    def wave(at=0.0):
        X, Y = torch.meshgrid(k + 2 * math.pi * at / n, k + 2 * math.pi * at / n, indexing="ij")
        return sum(r.uniform(0.3, 1.0) / 3 * torch.sin(a * X + b * Y + r.uniform(0, 2 * math.pi))
                   for a, b in ((1, 0), (0, 1), (1, 2), (2, -1), (3, 1)))
    A = 0.1 * wave(-0.5)                                     # vector potential at the corners (i-1/2, j-1/2)
    Bx, By = 0.2 + (torch.roll(A, -1, 1) - A) * n / 6, 0.1 - (torch.roll(A, -1, 0) - A) * n / 6
    rho, p = 1.5 + 0.4 * wave(0.5), 2.5 + 0.5 * wave(0.5)
    v = torch.stack([0.4 * wave(0.5), 0.4 * wave(0.5), 0.2 * wave(0.5)])
    b = torch.stack([0.5 * (Bx + torch.roll(Bx, -1, 0)), 0.5 * (By + torch.roll(By, -1, 1)), 0.1 * wave(0.5)])
    e = p / (5.0 / 3.0 - 1) + 0.5 * rho * (v * v).sum(0) + 0.5 * (b * b).sum(0)
    return torch.cat([rho[None], rho * v, e[None], b]), Bx, By


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cfl":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, e = case["blocks"], 16 + 2 * case["nghosts"]
        r = torch.rand(n, 8, e, e, dtype=torch.float64, device="cuda", generator=g)
        U = torch.empty_like(r)
        rho, v, b, p = 0.1 + 4 * r[:, 0], 2 * r[:, 1:4] - 1, 1.5 * (r[:, 5:8] - 0.3), 0.05 + 2 * r[:, 4]
        U[:, 0], U[:, 1:4], U[:, 5:8] = rho, v * rho[:, None], b
        U[:, 4] = p / (1.4 - 1) + 0.5 * rho * (v * v).sum(1) + 0.5 * (b * b).sum(1)
        level = torch.randint(0, 5, (n, 1), device="cuda", generator=g).expand(n, 2)
        dxdy = ((1 / 30.0) * 2.0 ** -level.double()).contiguous()
        return dict(kind=kind, U=U, dxdy=dxdy, out=torch.zeros(1, dtype=torch.float64, device="cuda"), n=n,
                    ng=case["nghosts"], lib=amr.load(), stream=torch.cuda.current_stream().cuda_stream)
    if kind == "riemann":
        wL, wR = face_states(case, seed)
        return dict(kind=kind, wL=wL, wR=wR, case=case)
    if kind == "program":
        r = random.Random(7919 * seed + 5)
        return dict(kind=kind, cfl=0.4 - 0.001 * r.random(), case=case)
    if kind == "steps":
        states = developed(case, seed)
        sim = amr.Simulation(step_configs(case, case["precision"]))
        for q, s in enumerate(states):
            lp, ic, lf = s["tree"]
            i = s["info"]
            sim.set_tree(lp, ic, lf, i["nb_leafs"], i["t"], i["dt"], i["dt_next"], i["steps"], instance=q)
        for q, s in enumerate(states):
            for f in ("U", "Bi", "ff", "gg"):
                sim.upload(f, s[f], q)
        sim.set_remesh(False)
        st = dict(kind=kind, run=Run(sim, states, case["precision"], case["steps"]))
    else:
        sim = amr.Simulation(kh_config(case, seed, case.get("precision", "fp64"))).init()
        if kind == "adjoint":
            U, Bx, By = smooth_flow(case, seed)
            state = dict(U=as_blocks(U, case["roots"]).numpy(), Bi=as_blocks(torch.stack([Bx, By]), case["roots"]).numpy())
        else:
            state = {f: sim.download(f) for f in ("U", "Bi")}
        st = dict(kind=kind, run=Run(sim, [state], case.get("precision", "fp64"), case["steps"]))
        if kind == "adjoint":
            st["lam"] = loss_weights(case, seed, sim.tree()[1])
    if case.get("tune"):
        sim.autotune(3)
    return st


def run(st):
    kind = st["kind"]
    if kind == "cfl":
        rc = st["lib"].amr_cfl_dt_static(ctypes.c_void_p(st["U"].data_ptr()), st["n"], st["ng"],
                                         ctypes.c_void_p(st["dxdy"].data_ptr()), 1.4,
                                         ctypes.c_void_p(st["out"].data_ptr()), ctypes.c_void_p(st["stream"]))
        if rc:
            raise amr.AmrError(rc, "amr_cfl_dt_static")
        return st["out"]
    if kind == "riemann":
        return amr.riemann(st["case"]["flux"], st["wL"], st["wR"], 1.4, bool(st["case"]["dir_y"]))
    if kind == "program":
        c = st["case"]
        sim = amr.Simulation(ic=c["ic"], limiter=c["limiter"], flux=c["flux"], cfl=st["cfl"], maxlevs=c["levels"],
                             nghosts=c["nghosts"]).init()
        sim.run(c["steps"])
        return sim.state()
    r = st["run"]
    r.upload()
    if kind != "adjoint":
        r.sim.run(r.steps)
        return r.download() if kind == "steps" else r.download_uniform()
    sim = r.sim
    sim.adjoint_enable(True)
    sim.run(r.steps)
    out = r.download_uniform()
    sim.adjoint_seed("U", st["lam"])
    for _ in range(r.steps):
        sim.adjoint_step()
    return dict(out, gU=sim.adjoint_read("U"), gBi=sim.adjoint_read("Bi"))


def work(case):
    kind = case["kind"]
    if kind == "cfl":
        e = 16 + 2 * case["nghosts"]
        return dict(bytes=case["blocks"] * 8 * 256 * 8 + case["blocks"] * 16 + 8, flops=case["blocks"] * 256 * 75)
    if kind == "riemann":
        return dict(bytes=case["n"] * (3 * 64 + 4), flops=case["n"] * FLUX_FLOPS[case["flux"]] / 2)
    if kind in ("frozen", "adjoint"):
        leaves, n, lim, fl = case["roots"] ** 2, 1, case["limiter"], "RUSA"
    else:
        leaves, n = LEAVES[(case["ic"], case["levels"])], case.get("instances", 1)
        lim, fl = case["limiter"], case["flux"]
    cells = 256 * leaves * n
    per_step = 2 * (RECON_FLOPS[recon_of(lim)] + FLUX_FLOPS[fl] + 60)
    io = cells * 10 * 8 * (1 if kind == "program" else 2)
    if kind == "adjoint":  # the seed and the gradient too; forward, recomputed and transposed steps
        return dict(bytes=io + cells * 18 * 8, flops=cells * case["steps"] * per_step * 4)
    return dict(bytes=io, flops=cells * case["steps"] * per_step)


# ------------------------------------------------------------- 64-bit results
def face_states(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]

    def side():
        w = np.empty((n, 8))
        w[:, 0] = rng.uniform(0.1, 4.0, n)
        w[:, 1:4] = rng.normal(0.0, 0.8, (n, 3))
        w[:, 4] = rng.uniform(0.05, 3.0, n)
        w[:, 5:8] = rng.normal(0.0, 0.6, (n, 3))
        return w
    wL, wR = side(), side()
    b = 6 if case["dir_y"] else 5
    wR[:, b] = wL[:, b]           # the normal field is the face's
    return wL, wR


def loss_weights(case, seed, icoord):
    """d loss / d U of a linear loss: random weights on every interior cell."""
    rng = np.random.default_rng(seed + 1)
    lam = np.zeros((len(icoord), 8, 20, 20))
    lam[:, :, 2:18, 2:18] = rng.normal(0.0, 1.0, (len(icoord), 8, 16, 16))
    return lam


SWAP = [0, 2, 1, 3, 4, 6, 5, 7]


def sides(w, g):
    """Conserved state, x flux, fast speed and total pressure of primitive states w [8, ...]."""
    rho, u, v, z, p, bx, by, bz = w
    b2 = bx * bx + by * by + bz * bz
    a2, c2, n2 = g * p / rho, b2 / rho, bx * bx / rho
    cf = torch.sqrt(0.5 * (c2 + a2 + torch.sqrt((c2 - a2) ** 2 + 4 * a2 * (c2 - n2))))
    e = p / (g - 1) + 0.5 * rho * (u * u + v * v + z * z) + 0.5 * b2
    pt = p + 0.5 * b2
    q = torch.stack([rho, rho * u, rho * v, rho * z, e, bx, by, bz])
    F = torch.stack([rho * u, rho * u * u + pt - bx * bx, rho * u * v - bx * by, rho * u * z - bx * bz,
                     u * (e + pt) - bx * (u * bx + v * by + z * bz), torch.zeros_like(rho), u * by - bx * v,
                     u * bz - bx * z])
    return q, F, cf, pt


def rusanov(l, r, g):
    qL, FL, cL, _ = sides(l, g)
    qR, FR, cR, _ = sides(r, g)
    s = torch.maximum(cL + l[1].abs(), cR + r[1].abs())
    return 0.5 * (FL + FR) - 0.5 * s * (qR - qL)


def hlld(l, r, g):
    """Miyoshi & Kusano's five-wave fan; both ** states are the left one, as in the scheme the framework has."""
    qL, FL, cL, ptL = sides(l, g)
    qR, FR, cR, ptR = sides(r, g)
    b = l[5]
    c = torch.maximum(cL, cR)
    SL, SR = torch.minimum(l[1], r[1]) - c, torch.maximum(l[1], r[1]) + c
    mL, mR = l[0] * (SL - l[1]), r[0] * (SR - r[1])
    SM = (mR * r[1] - mL * l[1] - ptR + ptL) / (mR - mL)
    pts = (mR * ptL - mL * ptR + mR * mL * (r[1] - l[1])) / (mR - mL)

    def star(w, q, pt, S):
        m = w[0] * (S - w[1])
        rho = m / (S - SM)
        den = m * (S - SM) - b * b
        k, h = b * (SM - w[1]) / den, (m * (S - w[1]) - b * b) / den
        v, z, by, bz = w[2] - w[6] * k, w[3] - w[7] * k, w[6] * h, w[7] * h
        e = ((S - w[1]) * q[4] - pt * w[1] + pts * SM + b * ((w[1:4] * w[5:8]).sum(0) - (SM * b + v * by + z * bz))) / (S - SM)
        return torch.stack([rho, rho * SM, rho * v, rho * z, e, b, by, bz]), v, z
    sL, vL, zL = star(l, qL, ptL, SL)
    sR, vR, zR = star(r, qR, ptR, SR)
    a, d = torch.sqrt(sL[0]), torch.sqrt(sR[0])
    S1, S2 = SM - b.abs() / a, SM + b.abs() / d
    sg = torch.sign(b)
    v = (a * vL + d * vR + (sR[6] - sL[6]) * sg) / (a + d)
    z = (a * zL + d * zR + (sR[7] - sL[7]) * sg) / (a + d)
    by = (a * sR[6] + d * sL[6] + a * d * (vR - vL) * sg) / (a + d)
    bz = (a * sR[7] + d * sL[7] + a * d * (zR - zL) * sg) / (a + d)
    vb = SM * b + v * by + z * bz
    eL = sL[4] - a * (SM * b + vL * sL[6] + zL * sL[7] - vb) * sg
    eR = sR[4] + d * (SM * b + vR * sR[6] + zR * sR[7] - vb) * sg
    mid = [sL[0], sL[0] * SM, sL[0] * v, sL[0] * z, eL, b, by, bz]
    midL = torch.stack(mid)
    midR = torch.stack(mid[:4] + [eR] + mid[5:])
    fan = [FL, FL + SL * (sL - qL), FL + S1 * midL - (S1 - SL) * sL - SL * qL,
           FR + S2 * midR - (S2 - SR) * sR - SR * qR, FR + SR * (sR - qR), FR]
    out = fan[5]
    for s, f in ((SR, fan[4]), (S2, fan[3]), (SM, fan[2]), (S1, fan[1])):
        out = torch.where(s >= 0, f, out)
    return torch.where(SL > 0, fan[0], out)


def limited(case, r):
    one = torch.ones_like(r)
    if case["limiter"] == "minmod":
        return torch.clamp(torch.minimum(one, r), min=0)
    return torch.clamp(torch.minimum(torch.minimum(2 * r, 0.5 * (1 + r)), 2 * one), min=0)


def uniform_step(case, U, Bx, By, dt, g, dx):
    """One RK2 step of the uniform periodic mesh, U [8, nx, ny], face fields at the left / lower faces."""
    def flux(U, Bx, By):
        rho, v = U[0], U[1:4] / U[0]
        p = (g - 1) * (U[4] - 0.5 * rho * (v * v).sum(0) - 0.5 * (U[5:8] ** 2).sum(0))
        W = torch.cat([rho[None], v, p[None], U[5:8]])
        out = []
        for d, bn in ((1, torch.roll(Bx, -1, 0)), (2, torch.roll(By, -1, 1))):
            Wp = torch.roll(W, -1, d)
            dA, dB, dC = W - torch.roll(W, 1, d), Wp - W, torch.roll(W, -2, d) - Wp
            l = W + 0.5 * limited(case, dB / (dA + 1e-15)) * dA
            r = Wp - 0.5 * limited(case, dB / (dC + 1e-15)) * dC
            if d == 2:
                l, r = l[SWAP], r[SWAP]
            l, r = (torch.cat([x[:5], bn[None], x[6:]]) for x in (l, r))
            f = rusanov(l, r, g)
            out.append(f[SWAP] if d == 2 else f)
        return out

    def update(base, F, G):
        return base - dt * ((F - torch.roll(F, 1, 1)) / dx + (G - torch.roll(G, 1, 2)) / dx)

    def transport(F, G, bx, by):
        G5, F6 = G[5], F[6]
        E = 0.25 * (torch.roll(G5, (1, 1), (0, 1)) + torch.roll(G5, 1, 1) - torch.roll(F6, (1, 1), (0, 1)) - torch.roll(F6, 1, 0))
        return bx - dt * (torch.roll(E, -1, 1) - E) / dx, by + dt * (torch.roll(E, -1, 0) - E) / dx

    def corrected(U, Bx, By):
        bx, by = 0.5 * (Bx + torch.roll(Bx, -1, 0)), 0.5 * (By + torch.roll(By, -1, 1))
        e = U[4] + 0.5 * (bx * bx + by * by - U[5] * U[5] - U[6] * U[6])
        return torch.stack([U[0], U[1], U[2], U[3], e, bx, by, U[7]])
    F, G = flux(U, Bx, By)
    bx, by = transport(F, G, Bx, By)
    Us = corrected(update(U, F, G), bx, by)
    F, G = flux(Us, bx, by)
    b2x, b2y = transport(F, G, bx, by)
    bx, by = 0.5 * (Bx + b2x), 0.5 * (By + b2y)
    return corrected(0.5 * (U + update(Us, F, G)), bx, by), bx, by


def kh_initial(c, n):
    """The perturbed shear layer on n x n cells of [0, 1]^2."""
    x = (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n
    X, Y = torch.meshgrid(x, x, indexing="ij")
    inside = (Y - 0.5).abs() <= 0.25
    rho, u = torch.where(inside, 2.0, 1.0).double(), torch.where(inside, 0.5, -0.5).double()
    env = torch.exp(-(Y - 0.25) ** 2 / 0.01) + torch.exp(-(Y - 0.75) ** 2 / 0.01)
    v = sum(c.ic_param[k] * torch.sin(2 * math.pi * (k + 1) * X) for k in range(16)) * env
    bx = torch.full_like(X, 0.1 / math.sqrt(4 * math.pi))
    zero = torch.zeros_like(X)
    e = 2.5 / (c.gamma - 1) + 0.5 * rho * (u * u + v * v) + 0.5 * bx * bx
    return torch.stack([rho, rho * u, rho * v, zero, e, bx, zero, zero]), bx, zero.clone()


def as_blocks(A, roots, ghosts=True):
    """[v, nx, ny] to blocks [root][v][20][20] ([j][i]), row by row, with periodic ghost cells (or zeros)."""
    n = 16 * roots
    i = torch.arange(20, device=A.device) - 2
    at = (16 * torch.arange(roots, device=A.device)[:, None] + i) % n          # [root, 20]
    B = A[:, at][:, :, :, at]                                                  # [v, rx, i, ry, j]
    B = B.permute(3, 1, 0, 4, 2).reshape(roots * roots, A.shape[0], 20, 20)
    if not ghosts:
        keep = ((i >= 0) & (i < 16)).double()
        B = B * keep[:, None] * keep
    return B.cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "cfl":
        s = prepare(case, seed)
        ng = case["nghosts"]
        U = s["U"][:, :, ng:ng + 16, ng:ng + 16].transpose(0, 1)
        v = U[1:4] / U[0]
        p = 0.4 * (U[4] - 0.5 * U[0] * (v * v).sum(0) - 0.5 * (U[5:8] ** 2).sum(0))
        W = torch.cat([U[:1], v, p[None], U[5:8]])
        lam = torch.maximum(W[0].abs() + sides(W, 1.4)[2], W[1].abs() + sides(W[SWAP], 1.4)[2])
        dt = s["dxdy"].amin(1) / lam.amax((1, 2))
        return torch.clamp(dt.amin(), max=1e6).reshape(1)
    if kind == "riemann":
        if case["flux"] not in ("RUSA", "HLLD"):
            return None
        l, r = (torch.from_numpy(w).T for w in face_states(case, seed))
        if case["dir_y"]:
            l, r = l[SWAP], r[SWAP]
        f = (rusanov if case["flux"] == "RUSA" else hlld)(l, r, 1.4)
        return (f[SWAP] if case["dir_y"] else f).T.contiguous().numpy(), None
    if kind not in ("frozen", "adjoint"):
        return None  # an adaptive mesh: a second implementation of the whole solver
    c = kh_config(case, seed, "fp64")
    n, roots = 16 * case["roots"], case["roots"]
    U0, Bx0, By0 = smooth_flow(case, seed) if kind == "adjoint" else kh_initial(c, n)
    if kind == "adjoint":
        for t in (U0, Bx0, By0):
            t.requires_grad_(True)
    U, Bx, By = U0, Bx0, By0
    for _ in range(case["steps"]):
        U, Bx, By = uniform_step(case, U, Bx, By, c.dt_fixed, c.gamma, 1.0 / n)
    out = dict(U=None, Bi=None, inner_U=as_blocks(U.detach(), roots)[:, :, 2:18, 2:18],
               inner_Bi=as_blocks(torch.stack([Bx, By]).detach(), roots)[:, :, 2:18, 2:18])
    if kind == "adjoint":
        icoord = [(16 * (b % roots), 16 * (b // roots)) for b in range(roots * roots)]
        lam = torch.from_numpy(loss_weights(case, seed, icoord)).cuda()[:, :, 2:18, 2:18]
        lam = lam.reshape(roots, roots, 8, 16, 16).permute(2, 1, 4, 0, 3).reshape(8, n, n)
        gU, gx, gy = torch.autograd.grad((lam * U).sum(), (U0, Bx0, By0))
        out["gU"] = as_blocks(gU, roots, ghosts=False)
        out["gBi"] = as_blocks(torch.stack([gx, gy]), roots, ghosts=False)
    return out
