"""The work that programs have this engine do, as cases that can be timed and checked.

A case is one call pattern of the public Python interface (qpgpu) at one size:

* ``step``   one 3D step of the fused path (Simulation.step3d: beam deposit, every
             slice, species renew) and the diagnostics a program reads after it:
             the on-axis wake, one plane of the force and of the plasma charge, and
             the transverse-B modes of the last slice;
* ``slices`` the same physics through the class interface, one reference call after
             another (Field2d, Species2d, Beam3d), for a number of slices, as a host
             code does that keeps its own slice loop;
* ``scan``   a parameter scan of independent instances (scan_run);
* ``grad``   forward and backward of the network that starts the B passes;
* ``train``  Adam steps of that network on pairs recorded from a simulation.

Grid sizes are powers of two (the engine's grids are); what is ragged is the
particle load: hollow and ring plasmas, 1 to 3 particles per cell and direction,
any number of beam particles, rectangular grids, image heights.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "quickpic-opensource_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import qpgpu  # noqa: E402

GAMMA = 20000.0


def listed():
    base = dict(kind="step", ppcx=2, ppcy=2, species=1, plasma=0, iter=2, tol=0.0, predict=0,
                beams=1, peak=4.0, sr=0.3, sz=0.6, dt=0.0, vpot=False, graphs=True)
    return [
        # the smallest call: the grid the parity tests use, direct launches
        # (the constructor's default); launch latency is all there is
        dict(base, name="step 64x64x32", ix=6, iy=6, iz=5, dz=0.3125, beam_np=32768,
             peak=2.0, sr=0.5, sz=0.5, graphs=False),
        # the reference's CPU-runnable configuration: 128^3, 262,144 beam particles
        dict(base, name="step 128x128x128", ix=7, iy=7, iz=7, dz=0.078125, beam_np=262144,
             peak=2.0, sz=0.5),
        # the medium transverse grid with the reference's two fixed passes
        dict(base, name="step 512x512x128", ix=9, iy=9, iz=7, dz=0.05, beam_np=262144),
        # the medium case as it is run: B to 1e-4, and each step ends with the beam
        # push; the host owns the beam, so its particles are copied in every step
        dict(base, name="step 512x512x128 to 1e-4", ix=9, iy=9, iz=7, dz=0.05,
             beam_np=300007, iter=16, tol=1e-4, dt=10.0),
        # the blow-out grid: narrow drive and witness bunches, 4.2 M electrons
        dict(base, name="step 1024x1024x64 two beams", ix=10, iy=10, iz=6, dz=0.08, beams=2,
             beam_np=200001, peak=20.0, sr=0.1, sz=0.4, iter=16, tol=1e-4),
        # rectangular grid, Gaussian ring plasma, 3 x 1 particles per cell, quadratic
        # start of the passes, vector potential kept
        dict(base, name="step 512x256x64 ring", ix=9, iy=8, iz=6, dz=0.1, ppcx=3, ppcy=1,
             plasma=11, beam_np=100003, iter=2, predict=2, vpot=True),
        # a hollow channel with mobile ions: two species, uneven tiles, one pass per slice
        dict(base, name="step 256x256x32 two species", ix=8, iy=8, iz=5, dz=0.2, species=2,
             plasma=10, iter=1, beam_np=65537),
        # the learned start of the passes (every layer of the network per slice)
        dict(base, name="step 256x256x64 learned", ix=8, iy=8, iz=6, dz=0.1, beam_np=131072,
             iter=16, tol=1e-4, predict=3),
        # a host code's own slice loop over the class interface
        dict(kind="slices", name="slices 256x256x16", ix=8, iy=8, iz=5, n=16, dz=0.2, ppcx=2,
             ppcy=2, iter=2, beam_np=65536, peak=2.0, sr=0.4, sz=0.5),
        # a parameter scan of small and middling instances on their own streams
        dict(kind="scan", name="scan of 6", n=6, ix=7, iz=5, dz=0.2, beam_np=32768),
        # one gradient of the network, 128 x 128 windows
        dict(kind="grad", name="network gradient 4", nb=4, h=128, w=128),
        # its training at the batch size it is trained with
        dict(kind="train", name="network training 32", batch=32, steps=16),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["slices"] * 2 + ["scan", "grad"])
    if kind == "grad":
        return dict(kind="grad", nb=rng.randint(1, 6), h=rng.randint(17, 160),
                    w=128 * rng.randint(1, 2))
    if kind == "scan":
        return dict(kind="scan", n=rng.randint(2, 7), ix=rng.choice([6, 7]), iz=rng.choice([4, 5]),
                    dz=round(rng.uniform(0.1, 0.3), 4),
                    beam_np=int(math.exp(rng.uniform(math.log(5e3), math.log(6e4)))))
    ix, iy = rng.randint(6, 9), rng.randint(6, 9)
    beam_np = int(math.exp(rng.uniform(math.log(1e4), math.log(3e5))))
    c = dict(kind=kind, ix=ix, iy=iy, dz=round(rng.uniform(0.08, 0.25), 4),
             ppcx=rng.randint(1, 3), ppcy=rng.randint(1, 2), beam_np=beam_np,
             peak=round(rng.uniform(1.0, 4.0), 3), sr=round(rng.uniform(0.25, 0.5), 3),
             sz=round(rng.uniform(0.4, 0.7), 3), iter=rng.randint(1, 3))
    if kind == "slices":
        return dict(c, iz=5, n=rng.randint(3, 20))
    c.update(iz=rng.randint(4, 7), species=1, plasma=rng.choice([0, 0, 0, 10, 11]), tol=0.0,
             predict=rng.choice([0, 0, 0, 1, 2]), beams=rng.choice([1, 1, 2]), dt=0.0,
             vpot=rng.random() < 0.2, graphs=rng.random() < 0.7)
    form = rng.choice(["fixed", "fixed", "tol", "species"])
    if form == "tol":
        c.update(tol=1e-4, iter=16, dt=rng.choice([0.0, 10.0]))
    elif form == "species":
        c.update(species=2, vpot=False, predict=0, iter=1)
    return c


# ---------------------------------------------------------------- inputs
def box_of(c):
    return [[-6.0, 6.0], [-6.0, 6.0], [0.0, c["dz"] * (1 << c["iz"])]]


def beam_specs(c):
    """Centre (xi), peak density and sigmas of each beam: the drive at 0.3 of the box,
    a witness of half its density at 0.75."""
    z = box_of(c)[2][1]
    s = [dict(center=0.3 * z, peak=c["peak"], sr=c["sr"], sz=min(c["sz"], 0.1 * z))]
    if c.get("beams", 1) == 2:
        s.append(dict(center=0.75 * z, peak=0.5 * c["peak"], sr=c["sr"],
                      sz=min(c["sz"], 0.07 * z)))
    return s


def beam_particles(c, seed):
    """part(7, np) of every beam, in cell units: a Gaussian sample of its own, slightly
    off axis, 1 % energy spread, normalised emittance 0.01."""
    rng = np.random.default_rng([seed, 17])
    box, out = box_of(c), []
    n = (1 << c["ix"], 1 << c["iy"], 1 << c["iz"])
    d = [(box[a][1] - box[a][0]) / n[a] for a in range(3)]
    for s in beam_specs(c):
        k = c["beam_np"]
        sig, mid = (s["sr"], s["sr"], s["sz"]), (0.05 * rng.standard_normal(), 0.0, s["center"])
        p = np.empty((7, k), dtype=np.float32, order="F")
        for a in range(3):
            x = (mid[a] + sig[a] * rng.standard_normal(k) - box[a][0]) / d[a]
            p[a] = np.clip(x, 1.01, n[a] - 1.01)
        p[3] = 0.01 / s["sr"] * rng.standard_normal(k)
        p[4] = 0.01 / s["sr"] * rng.standard_normal(k)
        p[5] = GAMMA + 0.01 * GAMMA * rng.standard_normal(k)
        p[6] = -s["peak"] * (2 * math.pi) ** 1.5 * s["sr"] ** 2 * s["sz"] / (d[0] * d[1] * d[2]) / k
        out.append(p)
    return out


def plasma_specs(c):
    """Keyword arguments of each Species2d; with two species the second is mobile ions."""
    shape = {0: {}, 10: dict(inner_radius=(0.9, 1.1), outer_radius=(4.6, 4.3)),
             11: dict(radius=1.5, width=1.2)}[c.get("plasma", 0)]
    e = dict(ppc=(c["ppcx"], c["ppcy"]), q=-1.0, m=1.0, profile=c.get("plasma", 0), **shape)
    return [e] + ([dict(e, q=1.0, m=1836.0)] if c.get("species", 1) == 2 else [])


def pinned(a):
    t = torch.empty(a.size, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()
    t = t.reshape(a.shape, order="F")
    t[...] = a
    return t


def net_params(seed):
    """Seeded weights of the network: He-initialised layers, a small last one."""
    rng = np.random.default_rng([seed, 23])
    out = []
    for cin, cout in ((16, 32), (32, 32), (32, 32), (32, 32), (32, 16)):
        std = math.sqrt(2.0 / (9 * cin)) * (1.0 if cout == 32 else 0.2)
        out += [std * rng.standard_normal(9 * cin * cout), 0.02 * rng.standard_normal(cout)]
    return np.concatenate(out).astype(np.float32)


class Held:
    """The handles and host arrays a program keeps, closed when it lets go of them."""

    def __init__(self, case):
        self.case, self.handles = case, []

    def keep(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        for h in reversed(self.handles):
            h.close()


def make_step(s, c, seed):
    ctx = s.keep(qpgpu.Context(c["ix"], c["iy"], c["iz"], box_of(c)))
    sp = [s.keep(qpgpu.Species2d(ctx, **k)) for k in plasma_specs(c)]
    parts = [pinned(p) for p in beam_particles(c, seed)]
    beams = []
    for b, p in zip(beam_specs(c), parts):
        # a beam of this many slots; the program's own particles replace the loader's
        beams.append(s.keep(qpgpu.Beam3d(
            ctx, (c["beam_np"], 1, 1), gamma=GAMMA, peak_density=b["peak"], quiet_start=False,
            center=(0.0, 0.0, b["center"]), sigma=(b["sr"], b["sr"], b["sz"]))))
        beams[-1].set_particles(p)
    ctx.sync()
    return ctx, sp, beams, parts


def prepare(case, seed):
    c, s = case, Held(case)
    if c["kind"] == "grad":
        rng = np.random.default_rng(seed)
        s.net = s.keep(qpgpu.Predictor(seed=1))
        s.net.set_params(net_params(seed))
        s.x = rng.standard_normal((c["nb"], 16, c["h"], c["w"]), dtype=np.float32)
        s.x[:, 12:] = 0.0
        s.t = 0.3 * rng.standard_normal((c["nb"], 2, c["h"], c["w"]), dtype=np.float32)
    elif c["kind"] == "train":
        rc = dict(ix=7, iy=7, iz=6, dz=0.15, ppcx=2, ppcy=2, beam_np=32768, peak=3.0, sr=0.3, sz=0.5)
        r = Held(rc)
        ctx, sp, beams, _ = make_step(r, rc, seed)
        sim = r.keep(qpgpu.Simulation(ctx, sp, beams, iter=16, tol=1e-4, store3d=False))
        s.data = s.keep(qpgpu.TrainingSet(ctx.nz))
        sim.record(s.data)
        sim.step3d()
        s.net = s.keep(qpgpu.Predictor(seed=1))
        s.params = net_params(seed)
        s.net.set_params(s.params)
    elif c["kind"] == "scan":
        s.sims = []
        for i in range(c["n"]):
            ci = scan_instance(c, i)
            ctx, sp, beams, _ = make_step(s, ci, seed + 1000 * i)
            s.sims.append(s.keep(qpgpu.Simulation(ctx, sp, beams, iter=2, use_graphs=True)))
    else:
        s.ctx, s.sp, s.beams, s.parts = make_step(s, c, seed)
        if c["kind"] == "slices":
            f = lambda dim: s.keep(qpgpu.Field2d(s.ctx, dim))  # noqa: E731
            s.f = dict(qb=f(1), qe=f(1), psi=f(1), psit=f(1), div=f(1), fxy=f(2), bxyz=f(3),
                       cu=f(3), dcu=f(2), amu=f(3), epw=f(2), epwb=f(2))
        else:
            s.sim = s.keep(qpgpu.Simulation(
                s.ctx, s.sp, s.beams, iter=c["iter"], use_graphs=c["graphs"], dt=c["dt"],
                tol=c["tol"], vpot=c["vpot"], predict=c["predict"]))
            if c["predict"] == 3:
                net = s.keep(qpgpu.Predictor(seed=1))
                net.set_params(np.load(os.path.join(PKG, "qpgpu", "predictor_weights.npy")))
                s.sim.set_predictor(net)
    return s


def scan_instance(c, i):
    """Instance i of a scan: density and size vary; every third one has a finer grid."""
    ind = c["ix"] + (1 if i % 3 == 2 else 0)
    return dict(kind="step", ix=ind, iy=ind, iz=c["iz"], dz=c["dz"], ppcx=2, ppcy=2, iter=2,
                tol=0.0, predict=0, beam_np=c["beam_np"], peak=1.0 + 0.5 * i, sr=0.3 + 0.03 * i,
                sz=0.5)


# ---------------------------------------------------------------- one pass
def plane_of(c):
    return 5 * (1 << c["iz"]) // 8


def run_slices(s):
    c, f, sp, beam = s.case, s.f, s.sp[0], s.beams[0]
    dex, dxi = s.ctx.dex, s.ctx.dxi
    qb, qe, psi, psit, div = f["qb"], f["qe"], f["psi"], f["psit"], f["div"]
    fxy, bxyz, cu, dcu, amu, epw, epwb = (f[k] for k in ("fxy", "bxyz", "cu", "dcu", "amu",
                                                         "epw", "epwb"))

    def magnetic():
        bxyz.mult(epw, [-dex, dex], dim=[1, 2], dim1=[2, 1])
        bxyz.mult(bxyz, [dex], dim=[3], dim1=[3])
        bxyz.sub(bxyz, epwb, dim=[1], dim1=[1], dim2=[2])
        bxyz.add(bxyz, epwb, dim=[2], dim1=[2], dim2=[1])
        bxyz.fftkr(2)

    def longitudinal():
        cu.div(div)
        div.pot(psit)
        psit.mult(psit, -dex)
        psit.fftkr(1)
        cu.bf(bxyz)

    beam.qdp()
    for h in (cu, epw):
        h.as_(0.0)
        h.fftrk(1)
    for j in range(1, c["n"] + 1):
        qb.as_(0.0)
        beam.qdp(qb, j + 1)
        qb.fftrk(1)
        qb.elf(epwb)
        qe.as_(0.0)
        sp.qdp(qe)
        qe.fftrk(1)
        qe.pot(psi)
        psi.grad(fxy)
        fxy.fftkr(1)
        psi.fftkr(1)
        sp.extpsi(psi, dex)
        longitudinal()
        for _ in range(c["iter"]):
            magnetic()
            for h in (cu, dcu, amu):
                h.as_(0.0)
            sp.amjdp(fxy, bxyz, psit, cu, amu, dcu, dex)
            for h, kind in ((cu, 1), (dcu, 1), (amu, 3)):
                h.mult(h, dex)
                h.fftrk(kind)
            cu.bfqp(dcu, amu, epw, dex * dex, dex)
            longitudinal()
        magnetic()
        fxy.mult(fxy, -1.0)
        fxy.add(fxy, bxyz, dim=[1], dim1=[1], dim2=[2])
        fxy.sub(fxy, bxyz, dim=[2], dim1=[2], dim2=[1])
        dcu.mult(dcu, dxi)
        cu.sub(cu, dcu, dim=[1, 2], dim1=[1, 2], dim2=[1, 2])
        sp.push(fxy, bxyz, psit, dex)
        sp.cbq(j + 1)
    out = dict(force=fxy.get_rs(), ez=psit.get_rs(), bperp=epw.get_ks(),
               charge=sp.get_q3(c["n"] + 1))
    sp.renew(0.0)
    return out


def read_step(sim, c):
    return dict(wake=sim.lineout(3), force=sim.get_plane("bexyz", plane_of(c)),
                charge=sim.get_plane("q3", plane_of(c)), bperp=sim.get_field("epw"))


def run(s):
    c = s.case
    if c["kind"] == "grad":
        loss, g = s.net.loss_grad(s.x, s.t)
        return dict(loss=loss, grad=g)
    if c["kind"] == "train":
        s.net.set_params(s.params)
        s.net.train(s.data, steps=c["steps"], batch=c["batch"], lr=1e-3)
        return dict(params=s.net.get_params())
    if c["kind"] == "scan":
        qpgpu.scan_run(s.sims, steps=1)
        return [read_step(sim, scan_instance(c, i)) for i, sim in enumerate(s.sims)]
    if c["kind"] == "slices":
        return run_slices(s)
    if c["dt"] > 0:
        for b, p in zip(s.beams, s.parts):
            b.set_particles(p)
    s.sim.step3d()
    out = read_step(s.sim, c)
    if c["dt"] > 0:
        out["beam"] = s.beams[0].get_particles()
    if c["vpot"]:
        out["vpot"] = s.sim.get_plane("vpot", plane_of(c))
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    if c["kind"] in ("grad", "train"):
        px = 128 * 128 * c["batch"] if c["kind"] == "train" else c["nb"] * c["h"] * c["w"]
        macs = 9 * (12 * 32 + 3 * 32 * 32 + 32 * 2)
        n = c["steps"] if c["kind"] == "train" else 1
        # forward, data gradient (not of the input) and weight gradient
        flops = 2.0 * px * n * (2 * macs + macs - 9 * 12 * 32)
        # features in (as bf16 once they are recorded), targets in
        return dict(bytes=float(px * n * ((24 if n > 1 else 48) + 8)), flops=flops)
    if c["kind"] == "scan":
        w = [work(scan_instance(c, i)) for i in range(c["n"])]
        return dict(bytes=sum(v["bytes"] for v in w), flops=sum(v["flops"] for v in w))
    nx, ny, nz = 1 << c["ix"], 1 << c["iy"], 1 << c["iz"]
    ns = c.get("n", nz) if c["kind"] == "slices" else nz
    share = {0: 1.0, 10: 0.42, 11: 1.0}[c.get("plasma", 0)]
    npl = (nx - 2) * (ny - 1) * c["ppcx"] * c["ppcy"] * share * c.get("species", 1)
    nodes = (nx + 1) * (ny + 1)
    passes = c["iter"] if not c.get("tol") else 2.0  # a converged start still needs two
    # beam in; per slice the plasma once in and once out (8 components) and the seven
    # 3D planes out
    byts = 28.0 * c["beam_np"] * c.get("beams", 1) + ns * (64.0 * npl + 28.0 * nodes)
    fft = 2.5 * nodes * (c["ix"] + c["iy"])  # one real transform of a plane in both axes
    flops = ns * (npl * (passes * 260.0 + 190.0) + fft * (9.0 + passes * 14.0)
                  + nodes * (40.0 + passes * 60.0))
    return dict(bytes=byts, flops=flops)


def tolerance(case):
    c = case
    if c["kind"] == "grad":
        # bf16 activations and output gradients: another order of the FP32 sums
        # moves values across a bf16 rounding
        return dict(rel=1e-2, max=0.3)
    if c["kind"] == "train":
        # the same, and Adam's step is the sign of a gradient that is nearly zero
        return dict(rel=2e-2, max=0.5)
    if c.get("tol"):
        # the passes stop at a relative change of 1e-4: where rounding moves a stop to
        # the next pass, fields move by about that, and later slices carry it
        return dict(rel=3e-3, max=0.3)
    # FP32 sums in any order, carried through the orbits of every later slice
    return dict(rel=6e-4, max=2e-2)


# ---------------------------------------------------------------- in 64 bits
class Exact:
    """The slice loop in float64 with plain torch: nodes [y][x], modes [ky][kx]."""

    def __init__(self, c, seed):
        self.c = c
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.nx, self.ny, self.nz = 1 << c["ix"], 1 << c["iy"], 1 << c["iz"]
        box = box_of(c)
        self.box = box
        self.dex, self.dxi = 12.0 / self.nx, box[2][1] / self.nz
        kx = 2 * math.pi / (2 * self.nx) * self.arange(self.nx + 1)[None, :]
        ky = 2 * math.pi / (2 * self.ny) * self.arange(self.ny + 1)[:, None]
        self.kx, self.ky = kx + 0 * ky, ky + 0 * kx
        k2 = kx * kx + ky * ky
        self.s = torch.exp(-0.5 * 0.912871 ** 2 * k2)
        self.g = torch.where(k2 > 0, self.s / torch.where(k2 > 0, k2, torch.ones_like(k2)),
                             torch.ones_like(k2))
        self.low = (self.arange(self.ny + 1)[:, None] < self.ny) & \
                   (self.arange(self.nx + 1)[None, :] < self.nx)
        self.inx = self.low & (self.kx > 0)
        self.iny = self.low & (self.ky > 0)
        self.inner = self.inx & self.iny
        self.sp = [self.plasma(k) for k in plasma_specs(c)]
        self.q3b = self.beam_charge(beam_particles(c, seed))

    def arange(self, n):
        return torch.arange(n, dtype=torch.float64, device=self.dev)

    # -- transforms: parity 0 sine, 1 cosine, unnormalised, along the last axis
    def line(self, a, parity):
        body = a[..., 1:-1].flip(-1)
        if parity:
            return torch.fft.rfft(torch.cat([a, body], -1)).real
        z = torch.zeros_like(a[..., :1])
        return -torch.fft.rfft(torch.cat([z, a[..., 1:-1], z, -body], -1)).imag

    def both(self, a, px, py):
        return self.line(self.line(a, px).transpose(-1, -2), py).transpose(-1, -2).contiguous()

    def rk(self, a, px, py):
        return self.both(a, px, py) * (0.25 / (self.nx * self.ny))

    def kr(self, a, px, py):
        r = self.both(a, px, py)
        r[self.ny] = r[0]
        return r

    # -- particles
    def plasma(self, k):
        c, d = self.c, self.dex
        px, py = k["ppc"]
        i, j = self.arange(self.nx)[1:-1], self.arange(self.ny)[1:]
        x = (i[:, None] + (self.arange(px)[None, :] + 0.5) / px).reshape(-1)
        y = (j[:, None] + (self.arange(py)[None, :] + 0.5) / py).reshape(-1)
        x, y = (v.reshape(-1) for v in torch.meshgrid(x, y, indexing="ij"))
        q = torch.full_like(x, math.copysign(1.0, k["q"]) / (px * py))
        u, v = x * d - 6.0, (y - self.ny / 2) * (12.0 / self.ny)
        if k["profile"] == 10:
            (ax, ay), (bx, by) = k["inner_radius"], k["outer_radius"]
            # radii enter in the cells of their own axis
            on = ((u / ax) ** 2 + (v / ay) ** 2 >= 1) & ((u / bx) ** 2 + (v / by) ** 2 <= 1)
            x, y, q = x[on], y[on], q[on]
        elif k["profile"] == 11:
            # the radius is in x cells, as the loader takes it
            r = torch.sqrt((x - self.nx / 2) ** 2 + (y - self.ny / 2) ** 2)
            q = q * torch.exp(-0.5 * ((r - k["radius"] / d) / (k["width"] / d)) ** 2)
        z = torch.zeros_like(x)
        s = dict(x=x, y=y, px=z, py=z, pz=z, p6=z + 1, p7=z + 1, q=q, qbm=k["q"] / k["m"])
        s["ion"] = -self.deposit(s, [q])[0]
        return s

    def corners(self, s):
        n, m = s["x"].floor(), s["y"].floor()
        dx, dy = s["x"] - n, s["y"] - m
        w = self.nx + 2
        o = m.long() * w + n.long()
        up = torch.where(m.long() + 1 == self.ny, n.long(), o + w)
        return ((o, (1 - dx) * (1 - dy)), (o + 1, dx * (1 - dy)), (up, (1 - dx) * dy),
                (up + 1, dx * dy)), (o, dx, dy)

    def deposit(self, s, values):
        at, _ = self.corners(s)
        out = []
        for v in values:
            p = torch.zeros((self.ny + 1) * (self.nx + 2), dtype=torch.float64, device=self.dev)
            for o, w in at:
                p.index_add_(0, o, w * v)
            out.append(p.reshape(self.ny + 1, self.nx + 2)[:, :-1].contiguous())
        return out

    def gather(self, s, planes):
        _, (o, dx, dy) = self.corners(s)
        w = self.nx + 2
        out = []
        for p in planes:
            p = torch.nn.functional.pad(p, (0, 1)).reshape(-1)
            out.append((1 - dy) * ((1 - dx) * p[o] + dx * p[o + 1])
                       + dy * ((1 - dx) * p[o + w] + dx * p[o + w + 1]))
        return out

    def beam_charge(self, parts):
        w, h = self.nx + 2, self.ny + 1
        q3 = torch.zeros((self.nz + 1) * w * h, dtype=torch.float64, device=self.dev)
        for p in parts:
            x, y, z, q = (torch.from_numpy(np.ascontiguousarray(p[i])).to(self.dev).double()
                          for i in (0, 1, 2, 6))
            n = [v.floor() for v in (x, y, z)]
            d = [x - n[0], y - n[1], z - n[2]]
            for k in range(8):
                a = [(k >> i) & 1 for i in range(3)]
                f = q
                for i in range(3):
                    f = f * (d[i] if a[i] else 1 - d[i])
                q3.index_add_(0, ((n[2].long() + a[2]) * h + n[1].long() + a[1]) * w
                              + n[0].long() + a[0], f)
        return q3.reshape(self.nz + 1, h, w)[:, :, :-1]

    # -- solves
    def smoothed(self, q):
        return self.kr(torch.where(self.inner, self.s * self.rk(q, 0, 0), 0 * q), 0, 0)

    def curl(self, cu):
        z, at = torch.zeros_like(self.g), self.g * self.s
        return [torch.where(self.inner, self.ky * at * cu[2], z),
                torch.where(self.inner, -self.kx * at * cu[2], z),
                torch.where(self.low, at * (self.kx * cu[1] - self.ky * cu[0]), z)]

    def fields(self, cu, epw, epwb):
        """psit and bxyz in real space from the current and the B iterate."""
        z = torch.zeros_like(self.g)
        psit = torch.where(self.inner, self.dex * self.g * (self.kx * cu[0] + self.ky * cu[1]), z)
        b = self.curl(cu)
        b = [-self.dex * epw[1] - epwb[1], self.dex * epw[0] + epwb[0], self.dex * b[2]]
        return self.kr(psit, 0, 0), [self.kr(b[0], 0, 1), self.kr(b[1], 1, 0), self.kr(b[2], 1, 1)]

    def moments(self, s, f, b, psit):
        """PPGRDCJPPOST2L_QP: the half push and the densities of cu, dcu, amu."""
        qtmh, dex = 0.5 * s["qbm"] * self.dxi, self.dex
        fx, fy, bx, by, bz, ez = self.gather(s, [*f, *b, psit])
        i7 = 1 / s["p7"]
        q1 = qtmh * i7
        q2 = q1 * s["p6"]
        ddx, ddy = -q2 * fx + qtmh * by, -q2 * fy - qtmh * bx
        acx, acy = s["px"] + ddx, s["py"] + ddy
        om = q1 * bz
        an, r1 = 2 / (1 + om * om), 0.5 * (1 - om * om)
        v1 = (r1 * acx + om * acy) * an + ddx
        v2 = (r1 * acy - om * acx) * an + ddy
        ox, oy = 0.5 * (v1 + s["px"]), 0.5 * (v2 + s["py"])
        oz = 0.5 * (1 + dex * dex * (ox * ox + oy * oy)) * i7 - 0.5 * s["p7"]
        s["p6"] = s["p7"] + oz
        oz = oz / dex
        vx, vy = (v1 - s["px"]) / self.dxi, (v2 - s["py"]) / self.dxi
        dz = s["qbm"] * (ez + (fx * ox + fy * oy) * dex * dex * i7)
        q = s["q"] * i7
        return self.deposit(s, [q * ox, q * oy, q * oz, q * (vx + ox * dz * i7),
                                q * (vy + oy * dz * i7), q * ox * ox * i7, q * oy * oy * i7,
                                q * ox * oy * i7])

    def push(self, s, f, b, psit):
        """PPGRBPPUSHF23L_QP and the periodic wrap."""
        dex = self.dex
        q1 = 0.5 * s["qbm"] * self.dxi / s["p7"]
        q2 = q1 * s["p6"]
        fx, fy, bx, by, bz, ez = self.gather(s, [*f, *b, psit])
        dx, dy, dz = q2 * fx, q2 * fy, q2 * ez / dex
        ax, ay, az = s["px"] + dx, s["py"] + dy, s["pz"] + dz
        ox, oy, oz = q1 * bx * dex, q1 * by * dex, q1 * bz
        om = ox * ox + oy * oy + oz * oz
        an, om = 2 / (1 + om), 0.5 * (1 - om)
        px = ((om + ox * ox) * ax + (oz + ox * oy) * ay + (ox * oz - oy) * az) * an + dx
        py = ((ox * oy - oz) * ax + (om + oy * oy) * ay + (ox + oy * oz) * az) * an + dy
        pz = ((oy + ox * oz) * ax + (oy * oz - ox) * ay + (om + oz * oz) * az) * an + dz
        s["px"], s["py"], s["pz"] = px, py, pz
        t = self.dxi / (torch.sqrt(1 + (px * px + py * py + pz * pz) * dex * dex) - pz * dex)
        s["x"], s["y"] = (s["x"] + px * t) % self.nx, (s["y"] + py * t) % self.ny

    def slices(self, n, keep=None):
        """n slices; the outputs of slice `keep` (default the last) and the on-axis Ez."""
        c, dex = self.c, self.dex
        z = torch.zeros_like(self.g)
        cu, epw, back1, back2 = [z, z, z], [z, z], [z, z], [z, z]
        wake, out = [0.0], {}
        for j in range(1, n + 1):
            qb = self.rk(self.q3b[j], 0, 0)
            epwb = [torch.where(self.inner, -self.g * self.s * k * qb, z)
                    for k in (self.kx, self.ky)]
            charge = [self.deposit(s, [s["q"]])[0] for s in self.sp]
            qe = sum(q + s["ion"] for q, s in zip(charge, self.sp))
            psi = torch.where(self.inner, self.g * self.rk(qe, 0, 0), z)
            f = [self.kr(self.kx * psi, 1, 0), self.kr(self.ky * psi, 0, 1)]
            psi = self.kr(psi, 0, 0)
            for s in self.sp:
                d = -self.gather(s, [psi])[0] * dex * dex * s["qbm"]
                s["p7"] = 1 + d
                s["p6"] = d + (dex * dex * (s["px"] ** 2 + s["py"] ** 2) - d * d - 2 * d) / \
                    (2 * (1 + d)) + 1
            if c.get("predict", 0):
                e1 = epw
                epw = [3 * (a - b) + e if c["predict"] == 2 else 2 * a - b
                       for a, b, e in zip(epw, back1, back2)]
                back1, back2 = e1, back1
            psit, b = self.fields(cu, epw, epwb)
            for _ in range(c["iter"]):
                per = [[dex * v for v in self.moments(s, f, b, psit)] for s in self.sp]
                m = [sum(v) for v in zip(*per)]
                par = [(1, 0), (0, 1), (0, 0), (1, 0), (0, 1), (0, 0), (0, 0), (1, 1)]
                k = [self.rk(v, *p) for v, p in zip(m, par)]
                cu, dc, (axx, ayy, axy) = k[:3], k[3:5], k[5:]
                d = [-dc[0] + self.kx * axx - self.ky * axy, -dc[1] - self.kx * axy + self.ky * ayy]
                at = self.g / (1 + dex * dex * self.g)
                epw = [torch.where(on, at * self.s * (d[i] - kk * cu[2] / dex)
                                   + dex * dex * at * epw[i], z)
                       for i, (on, kk) in enumerate(((self.iny, self.kx), (self.inx, self.ky)))]
                on = self.inx | self.iny
                dc = [torch.where(on, a, o) for a, o in zip(d, dc)]
                psit, b = self.fields(cu, epw, epwb)
            if j == (keep or n) and c.get("vpot"):
                at = self.g * self.s
                a = [torch.where(on, at * v, z) for on, v in zip((self.iny, self.inx, self.inner), cu)]
                out["vpot"] = [-dex * self.kr(a[0], 1, 0), -dex * self.kr(a[1], 0, 1),
                               -dex * self.kr(a[2], 0, 0)]
            if j == (keep or n):
                out["charge"] = self.smoothed(charge[0] + per[0][2])
            f = [-f[0] + b[1], -f[1] - b[0]]
            cu = [cu[0] - self.dxi * dc[0], cu[1] - self.dxi * dc[1], cu[2]]
            for s in self.sp:
                self.push(s, f, b, psit)
            wake.append(float(psit[self.ny // 2, self.nx // 2]))
            if j == (keep or n):
                out["force"], out["ez"] = f, psit
        return out, wake, epw

    # -- the layouts of the downloads
    def nodes(self, planes, rows):
        a = np.zeros((len(planes), self.nx + 2, rows))
        for i, p in enumerate(planes):
            a[i, : self.nx + 1, : self.ny + 1] = p.cpu().numpy().T
        return a

    def modes(self, planes):
        return np.stack([p.cpu().numpy() for p in planes])


def exact_step(c, seed):
    e = Exact(c, seed)
    o, wake, epw = e.slices(e.nz, plane_of(c))
    force = [e.dex * v for v in o["force"]] + [o["ez"]]
    out = dict(wake=np.array(wake), force=e.nodes(force, e.ny + 1),
               charge=e.nodes([o["charge"]], e.ny + 1)[0], bperp=e.modes(epw))
    if c.get("vpot"):
        out["vpot"] = e.nodes(o["vpot"], e.ny + 1)
    return out


def exact_grad(c, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((c["nb"], 16, c["h"], c["w"]), dtype=np.float32)
    x[:, 12:] = 0.0
    t = 0.3 * rng.standard_normal((c["nb"], 2, c["h"], c["w"]), dtype=np.float32)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    a, t = (torch.from_numpy(v).to(dev).double() for v in (x, t))
    p = torch.from_numpy(net_params(seed)).to(dev).double().requires_grad_(True)
    o = 0
    for cin, cout in ((16, 32), (32, 32), (32, 32), (32, 32), (32, 16)):
        w = p[o:o + 9 * cin * cout].reshape(3, 3, cin, cout).permute(3, 2, 0, 1)
        o += 9 * cin * cout
        pad = torch.nn.functional.pad(a, (1, 1, 1, 1))
        cols = torch.nn.functional.unfold(pad, 3)  # plain matrix product in float64
        y = torch.matmul(w.reshape(cout, -1), cols) + p[o:o + cout][None, :, None]
        o += cout
        a = y.reshape(a.shape[0], cout, *a.shape[2:])
        a = a.relu() if cout == 32 else a[:, :2]
    loss = ((a - t) ** 2).mean()
    loss.backward()
    return dict(loss=float(loss), grad=p.grad.cpu().numpy())


def exact(case, seed):
    c = case
    if c["kind"] == "grad":
        return exact_grad(c, seed)
    if c["kind"] == "train" or c.get("tol"):
        # Adam amplifies bf16 roundings of the gradients; a stop at a tolerance may
        # come one pass earlier or later: neither has one exact value
        return None
    if c["kind"] == "scan":
        return [exact_step(scan_instance(c, i), seed + 1000 * i) for i in range(c["n"])]
    if c["kind"] == "slices":
        e = Exact(c, seed)
        o, _, epw = e.slices(c["n"])
        return dict(force=e.nodes(o["force"], 2 * e.ny + 1), ez=e.nodes([o["ez"]], 2 * e.ny + 1),
                    bperp=e.modes(epw), charge=e.nodes([o["charge"]], e.ny + 1)[0])
    return exact_step(c, seed)
