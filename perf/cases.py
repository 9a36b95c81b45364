"""Workloads that time this library through its public entry points.

Four kinds of work, each as a program would call it:

* ``leg``       one leg of a simulation between two outputs: the compressed state goes up from page-locked host
                memory, a few whole steps run (update_x, the buffer calls, ext_pp_force and particle_mesh as the one
                call pp_particle_mesh, or particle_mesh alone where PP is off), and the new state comes back.
* ``species``   the same with a second, linked neutrino species (particle_mesh2).
* ``ensemble``  steps of a batch of independent boxes through its captured graph, the boxes' states read back.
* ``gradient``  the differentiable form: forward pass, final density, loss cotangent, density adjoint, backward pass;
                or the forward pass and the density alone.
* ``power``     the matter power spectrum of a resident state, the analysis call between steps.

Initial states are Zel'dovich realisations of the seed made on the device, evolved first where a case says so: the
clustered state of a late run is dearer for PP and the re-sort than the nearly uniform one of an early run.
"""
import gc
import math

import numpy as np
import torch
import torch.utils.checkpoint

from cafproject_gb300 import batch as B
from cafproject_gb300 import cosmology as cm
from cafproject_gb300 import cube as C
from cafproject_gb300 import dpm as D
from cafproject_gb300 import params as P

OMEGA_M, OMEGA_L, H0, S8, N_S = 0.3, 0.7, 0.7, 0.8, 0.96
DLNA = math.log(50.0) / 100.0  # step of the 100-step runs from z = 49 to 0
M_NU = 0.05                    # eV


def listed():
    leg = dict(kind="leg", np_nc=2, izipx=1, izipv=2, pp=True, evolve=0)
    return [
        # the smallest multi-tile box of the tests: launches and host latency count
        dict(leg, name="leg 48^3 pp", nc=24, nnt=2, cell=3.125, z=9.0, steps=4),
        # the PM-only configuration: 64^3 particles, 200 Mpc/h, one tile
        dict(leg, name="leg 64^3 pm", nc=32, nnt=1, cell=6.25, z=49.0, steps=4, pp=False),
        # two-byte positions, a mesh that is no power of two (nc 54, nf 216) over 3^3 tiles, large Zel'dovich moves
        dict(leg, name="leg 108^3 x2v2", nc=54, nnt=3, cell=2.5, z=2.0, steps=3, izipx=2),
        # the most compressed format, one byte for every component
        dict(leg, name="leg 208^3 x1v1", nc=104, nnt=2, cell=2.34375, z=5.0, steps=3, izipv=1),
        # a late run: 256^3 particles evolved to z = 0, haloes of thousands of particles
        dict(leg, name="leg 256^3 late", nc=128, nnt=2, cell=2.34375, z=0.1, steps=2, evolve=48),
        # the headline workload: 512^3 particles, 600 Mpc/h, fine mesh 1024^3, from z = 49
        dict(leg, name="leg 512^3 pp", nc=256, nnt=2, cell=2.34375, z=49.0, steps=3),
        # two species: CDM and eight times as many fast neutrinos, 4^3 tiles, moves of several cells
        dict(kind="species", name="species 128^3+256^3", nc=64, nnt=4, cell=3.90625, z=10.0, steps=2),
        # an ensemble of uneven small boxes in one graph launch per step
        dict(kind="ensemble", name="ensemble 12 boxes", boxes=12, largest=96, steps=2),
        # gradients of a small reconstruction, mesh not a power of two
        dict(kind="gradient", name="gradient 40^3", npd=40, ng=80, box=160.0, steps=6, ckpt=3, backward=True),
        # the differentiable workload: 128^3 particles, 256^3 mesh, ten steps
        dict(kind="gradient", name="gradient 128^3", npd=128, ng=256, box=256.0, steps=10, ckpt=2, backward=True),
        # a forward model without gradients, mesh three times the lattice
        dict(kind="gradient", name="forward 100^3", npd=100, ng=300, box=400.0, steps=8, ckpt=4, backward=False),
        # the power spectrum of an evolved state on the fine mesh
        dict(kind="power", name="power 512^3 mesh", nc=128, ng=512, cell=2.34375, z=1.0, evolve=12),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _tile(nnt, nt):
    """Coarse cells of a tile: at least twice the buffer depth, the whole mesh at least 16 and even."""
    nt = max(12 if nnt > 1 else 16, int(round(nt)))
    return nt + (nt * nnt) % 2


def draw(rng):
    kind = rng.choice(["leg"] * 6 + ["species", "ensemble", "gradient", "gradient", "gradient", "power"])
    if kind == "leg":
        nnt = rng.choice([1, 1, 2, 2, 3, 4])
        nc = nnt * _tile(nnt, _log(rng, 16, 200) / nnt)
        evolve = rng.choice([0, 0, rng.randint(8, 40)]) if nc <= 128 else 0
        z = math.expm1(math.log(20.0) - evolve * math.log(20.0) / 48.0) if evolve else rng.choice([49.0, 9.0, 2.0])
        return dict(kind="leg", nc=nc, nnt=nnt, np_nc=2, cell=round(_log(rng, 1.5, 6.25), 4),
                    izipx=rng.choice([1, 1, 2]), izipv=rng.choice([1, 2, 2]), pp=rng.random() < 0.8, z=round(z, 4),
                    evolve=evolve, steps=rng.randint(2, 4))
    if kind == "species":
        nnt = rng.choice([1, 2, 4])
        nc = nnt * _tile(nnt, _log(rng, 24, 72) / nnt)
        return dict(kind=kind, nc=nc, nnt=nnt, cell=round(rng.uniform(2.5, 6.0), 4), z=10.0, steps=rng.randint(1, 2))
    if kind == "ensemble":
        return dict(kind=kind, boxes=rng.randint(3, 12), largest=rng.choice([48, 64, 96]), steps=rng.randint(1, 4))
    if kind == "gradient":
        npd = 2 * int(round(_log(rng, 16, 128) / 2))
        ng = npd * rng.choice([1, 2, 2, 3] if npd <= 100 else [1, 2])
        steps = rng.randint(3, 10)
        return dict(kind=kind, npd=npd, ng=ng, box=round(npd * rng.uniform(1.5, 4.0), 2), steps=steps,
                    ckpt=rng.randint(1, min(4, steps)), backward=rng.random() < 0.7)
    nc = 2 * int(round(_log(rng, 24, 128) / 2))
    return dict(kind="power", nc=nc, ng=nc * rng.choice([1, 2, 4]), cell=round(_log(rng, 1.5, 6.25), 4), z=1.0,
                evolve=rng.choice([0, 12]))


# ------------------------------------------------------------------ states


def _params(case):
    return P.CubeParams(nc=case["nc"], nnt=case.get("nnt", 1), pp_on=bool(case.get("pp", True)), rsoft=0.1,
                        izipx=case.get("izipx", 1), izipv=case.get("izipv", 2), np_nc=case.get("np_nc", 2),
                        box=case["cell"] * case["nc"], omega_m=OMEGA_M, omega_l=OMEGA_L, h0=H0, s8=S8, n_s=N_S)


def _steps(z, n):
    """dt and a_mid of n steps from z, as long as those of a 100-step run."""
    a = math.log(1.0 / (1.0 + z)) + DLNA * n
    dt, a_mid, _ = cm.fixed_schedule(z, math.expm1(-a), n, OMEGA_M, OMEGA_L)
    return dt, a_mid


def _host(p, n):
    """Page-locked arrays for a state of up to n particles."""
    def pin(shape, dtype):
        return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()
    x = torch.int8 if p.izipx == 1 else torch.int16
    v = torch.int8 if p.izipv == 1 else torch.int16
    return dict(xp=pin((n, 3), x), vp=pin((n, 3), v), pid=pin((n,), torch.int32),
                rhoc=pin((p.nc ** 3,), torch.int32), vfield=pin((p.nc ** 3, 3), torch.float32))


def _take(g, p):
    """The context's state in page-locked arrays, and room for the one that comes back."""
    n = g.nplocal()
    state = g.download(_host(p, n))
    return state, _host(p, n + n // 64 + 4096)


def _evolve(g, p, vmax, z_end, n, z_init=19.0):
    dt, a_mid, _ = cm.fixed_schedule(z_init, z_end, n, OMEGA_M, OMEGA_L)
    vz, old = vmax[2], 0.0
    for i in range(n):
        g.update_x(old, dt[i], vz)
        pm = g.pp_particle_mesh(a_mid[i], dt[i])[1] if p.pp_on else g.particle_mesh(a_mid[i], dt[i])
        vz, old = pm["vmax"][2], dt[i]
    return g.get_sigma()[0], pm["vmax"]


def _start(g, p, case, seed):
    """A state at the case's redshift in the context; (sigma_vi, largest |v| per dimension)."""
    if case["evolve"]:
        _, vmax = g.ic_zeldovich(19.0, seed)
        return _evolve(g, p, vmax, case["z"], case["evolve"])
    return g.ic_zeldovich(case["z"], seed)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    {"leg": _prepare_leg, "species": _prepare_species, "ensemble": _prepare_ensemble, "gradient": _prepare_gradient,
     "power": _prepare_power}[s.kind](s, case, seed)
    return s


def run(s):
    return {"leg": _run_leg, "species": _run_species, "ensemble": _run_ensemble, "gradient": _run_gradient,
            "power": _run_power}[s.kind](s)


def _prepare_leg(s, case, seed):
    p = _params(case)
    s.p, s.g = p, C.CubeGPU(p)
    s.sigma, vmax = _start(s.g, p, case, seed)
    s.vz = vmax[2]
    s.dt, s.a_mid = _steps(case["z"], case["steps"])
    s.state, s.out = _take(s.g, p)


def _run_leg(s):
    g, n = s.g, len(s.dt)
    g.upload_begin(**s.state)
    g.set_sigma(s.sigma)
    vz, old, stats = s.vz, 0.0, []
    for i in range(n):
        up = g.update_x(old, s.dt[i], vz)
        g.buffer_grid()
        g.buffer_x()
        if i == n - 1:
            g.download_begin(s.out)
        if s.p.pp_on:
            pp, pm = g.pp_particle_mesh(s.a_mid[i], s.dt[i])
        else:
            pp, pm = None, g.particle_mesh(s.a_mid[i], s.dt[i])
        g.buffer_v()
        vz, old = pm["vmax"][2], s.dt[i]
        stats.append(_stats(up, pp, pm))
    out = g.download_finish()
    out["stats"] = np.array([x[0] for x in stats])
    out["counts"] = np.array([x[1] for x in stats])
    return out


def _stats(up, pp, pm):
    """What a driver takes from a step: the maxima its dt follows from, and the counts it checks."""
    real = [up["sigma_vi_new"], pm["f2_max_fine"], pm["f2_max_coarse"], pp["f2_max_pp"] if pp else 0.0] + pm["vmax"]
    whole = [up["nplocal"], up["nlost"], up["ndup"], up["max_disp"], pp["npairs"] if pp else 0]
    return np.array(real, np.float32), np.array(whole, np.int64)


def _prepare_species(s, case, seed):
    f_nu = M_NU / 93.14 / H0 ** 2 / OMEGA_M  # Omega_nu h^2 = m_nu / 93.14 eV
    geo = dict(nc=case["nc"], nnt=case["nnt"], box=case["cell"] * case["nc"], omega_m=OMEGA_M, omega_l=OMEGA_L)
    pc = P.CubeParams(pp_on=True, rsoft=0.1, np_nc=2, mass_p=8.0 * (1 - f_nu), **geo)
    pn = P.CubeParams(pp_on=False, np_nc=4, mass_p=f_nu, **geo)
    s.g = C.CubeGPU(pc)
    s.nu = C.CubeGPU(pn, owner=s.g)
    s.sigma, vc = s.g.ic_zeldovich(case["z"], seed)
    s.sigma_nu, vn = s.nu.ic_zeldovich_nu(case["z"], seed, M_NU, seed + 7)
    s.vz = max(vc[2], vn[2])
    s.dt, s.a_mid = _steps(case["z"], case["steps"])
    s.dt = np.minimum(s.dt, np.float32(18.0 / max(max(vc), max(vn))))  # the driver's dt_vmax
    s.state, s.out = _take(s.g, pc)
    s.state_nu, s.out_nu = _take(s.nu, pn)


def _run_species(s):
    g, nu = s.g, s.nu
    g.upload_begin(**s.state)
    nu.upload_begin(**s.state_nu)
    g.set_sigma(s.sigma)
    nu.set_sigma(s.sigma_nu)
    vz, old = s.vz, 0.0
    for i in range(len(s.dt)):
        up, upn = g.update_x(old, s.dt[i], vz), nu.update_x(old, s.dt[i], vz)
        pp = g.ext_pp_force(s.a_mid[i], s.dt[i])
        pm, pmn = g.particle_mesh2(nu, s.a_mid[i], s.dt[i])
        vz, old = max(pm["vmax"][2], pmn["vmax"][2]), s.dt[i]
    real, whole = _stats(up, pp, pm)
    return {"cdm": g.download(s.out), "nu": nu.download(s.out_nu), "stats": real, "counts": whole,
            "vmax_nu": np.array(pmn["vmax"], np.float32), "n_nu": upn["nplocal"]}


def _prepare_ensemble(s, case, seed):
    sizes = tuple(n for n in (32, 48, 64, 96, 128) if n <= case["largest"])
    # the mix of sizes belongs to the case, the realisations to the seed
    boxes = B.ensemble(case["boxes"], base_seed=1 + 1000 * (seed % 100003), sizes=sizes)
    s.b = B.Batch(boxes, z_init=19.0)
    n = 1600  # room for many passes of one ongoing run, z = 19 to 3
    dt, a_mid = np.zeros((len(boxes), n), np.float32), np.zeros((len(boxes), n), np.float32)
    a = np.exp(np.linspace(math.log(1 / 20.0), math.log(1 / 4.0), n + 1))
    mid = 0.5 * (a[1:] + a[:-1])
    for i, (p, _) in enumerate(boxes):
        # the Friedmann equation in the code's time unit, as the step's own expansion has it
        adot = 2.0 / 3.0 * np.sqrt(mid ** 3 * (1 + mid ** 3 * p.omega_l / p.omega_m
                                               + mid * (1 - p.omega_m - p.omega_l) / p.omega_m))
        dt[i], a_mid[i] = (a[1:] - a[:-1]) / adot, mid
    s.b._check(s.b.L.cube_batch_set_schedule(s.b.h, n, dt.ctypes.data, a_mid.ctypes.data))
    s.b.nsteps = n
    s.out = [_host(p, p.capacity()) for p, _ in boxes]
    s.done = 0


def _run_ensemble(s):
    n = s.case["steps"]
    s.b.step(n)
    s.done += n
    real, whole = [], []
    for h in s.b.history(s.done - 1):
        real.append([h["sigma_vi_new"], h["f2_max_fine"], h["f2_max_coarse"], h["f2_max_pp"]] + h["vmax"])
        whole.append([h["npairs"], h["itest1"], h["ndup"]])
    out = {"stats": np.array(real, np.float32), "counts": np.array(whole, np.int64)}
    for key in ("xp", "vp", "pid", "rhoc", "vfield"):
        out[key] = []
    for i, room in enumerate(s.out):
        st = s.b.box(i).download(room)
        for key in ("xp", "vp", "pid", "rhoc", "vfield"):
            out[key].append(st[key])
    return out


def _prepare_power(s, case, seed):
    p = _params(case)
    s.g = C.CubeGPU(p)
    _start(s.g, p, case, seed)
    s.g.synchronize()


def _run_power(s):
    return s.g.power_spectrum(s.case["ng"], s.case["cell"] * s.case["nc"])


def _noise(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed))
    return torch.randn(case["npd"] ** 3, generator=gen, device="cuda")


def _target(case, seed):
    """A smooth positive density of mean one, standing for the observed field."""
    gen = torch.Generator("cuda").manual_seed(int(seed) + 999983)
    n = case["ng"]
    f = torch.randn(n, n, n, generator=gen, device="cuda")
    for d in range(3):
        f = (torch.roll(f, 1, d) + f + torch.roll(f, -1, d)) / math.sqrt(3.0)
    r = torch.exp(0.5 * f)
    return (r / r.mean()).contiguous()


def _prepare_gradient(s, case, seed):
    s.sim = D.DiffPM(case["ng"], case["npd"], 9.0, 0.0, case["steps"], ckpt_every=case["ckpt"], box=case["box"],
                     omega_m=OMEGA_M, omega_l=OMEGA_L, h0=H0, s8=S8, n_s=N_S)
    s.noise = _noise(case, seed)
    if case["backward"]:
        s.target = _target(case, seed)
        s.zero = torch.zeros(case["npd"] ** 3, 3, device="cuda")


def _run_gradient(s):
    x, v = s.sim.forward(s.noise)
    rho = s.sim.density(x)
    if not s.case["backward"]:
        return {"x": x, "v": v, "rho": rho}
    gx = s.sim.density_adjoint(x, 2.0 * (rho - s.target))
    return {"x": x, "v": v, "rho": rho, "gnoise": s.sim.backward(gx, s.zero)}


# -------------------------------------------------------------------- work


def _pm_step(nc, n, code):
    """One step of the two-level PM: the state read and written once, the densities, spectra and three force
    components of both meshes once each way, and the kernels once; four transforms of each mesh."""
    b = f = 0.0
    for m in (nc, 4 * nc):
        b += 4.0 * m ** 3 * (2 + 2 + 6 + 6 + 1.5)
        f += 4 * 2.5 * m ** 3 * math.log2(m ** 3) + 8 * m ** 3
    b += 2.0 * n * (code + 4) + 2.0 * 16 * nc ** 3
    f += n * (2 * (3 * 8 * 4 + 40) + 2 * 40 + 60)
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("leg", "species"):
        n = (2.0 * case["nc"]) ** 3
        code = 3 * case.get("izipx", 1) + 3 * case.get("izipv", 2)
        b, f = _pm_step(case["nc"], n, code)
        if kind == "species":
            b += 2.0 * 8 * n * (code + 4) + 2.0 * 16 * case["nc"] ** 3
            f += 8 * n * 360
        elif case["pp"]:
            f += 2 * n * 25
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "ensemble":
        b = f = 0.0
        sizes = tuple(n for n in (32, 48, 64, 96, 128) if n <= case["largest"])
        for p, _ in B.ensemble(case["boxes"], sizes=sizes):
            x, y = _pm_step(p.nc, float(p.npglobal), 9)
            b, f = b + x, f + y + 50.0 * p.npglobal
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "gradient":
        n, m = float(case["npd"]) ** 3, float(case["ng"]) ** 3
        fft = 2 * 2.5 * m * math.log2(m)
        fwd_b, fwd_f = 48 * n + 4 * m * (2 + 2 + 2 + 0.5), n * 200 + fft
        b, f = case["steps"] * fwd_b + 36 * n + 4 * m, case["steps"] * fwd_f + n * 40
        if case["backward"]:
            # the potentials again, then the adjoint of each step, about a forward step's traffic each
            b += case["steps"] * 2 * fwd_b + 24 * n + 8 * m
            f += case["steps"] * (2 * fwd_f + n * 200)
        return {"bytes": b, "flops": f}
    n, m = (2.0 * case["nc"]) ** 3, float(case["ng"]) ** 3
    return {"bytes": 3 * n + 4.0 * case["nc"] ** 3 + 4 * m * 4, "flops": n * 60 + 2.5 * m * math.log2(m) + 15 * m}


# ------------------------------------------------- the same answers in 64 bits


def exact(case, seed):
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "power":
        return _exact_power(case, seed)
    # the state's codes are whole numbers; the velocity field and the maxima
    # after several kicks have no value of their own apart from those codes
    return None


def _exact_power(case, seed):
    """powerspectrum.f90's auto power of the CIC density contrast, in float64."""
    p = _params(case)
    g = C.CubeGPU(p)
    _start(g, p, case, seed)
    st = g.download()
    g.close()
    nc, ng = case["nc"], case["ng"]
    dev = torch.device("cuda")
    cell = torch.repeat_interleave(torch.arange(nc ** 3, device=dev), torch.as_tensor(st["rhoc"], device=dev).long())
    xp = torch.as_tensor(st["xp"], device=dev)
    bits = 8 * xp.element_size()
    frac = ((xp.long() & ((1 << bits) - 1)).double() + 0.5) / (1 << bits)
    nt, nnt = p.nt, p.nnt
    dims = []
    tile = cell // nt ** 3
    for d in range(3):
        dims.append((cell // nt ** d) % nt + nt * ((tile // nnt ** d) % nnt))
    pos = (torch.stack(dims, 1).double() + frac) * (ng / nc) - 0.5
    del cell, xp, frac, dims
    lo = torch.floor(pos)
    w = pos - lo
    lo = lo.long()
    rho = torch.zeros(ng ** 3, dtype=torch.float64, device=dev)
    for k in range(8):
        o = [k & 1, k >> 1 & 1, k >> 2]
        c = [(lo[:, d] + o[d]) % ng for d in range(3)]
        wt = 1.0
        for d in range(3):
            wt = wt * (w[:, d] if o[d] else 1 - w[:, d])
        rho.index_add_(0, (c[2] * ng + c[1]) * ng + c[0], wt)
    del pos, lo, w
    delta = (rho / rho.mean() - 1).view(ng, ng, ng)
    del rho
    ck = torch.fft.rfftn(delta) / ng ** 3
    del delta
    nyq = ng // 2
    ky = (torch.arange(ng, device=dev) + nyq) % ng - nyq
    kx = (torch.arange(nyq + 1, device=dev) + nyq) % ng - nyq
    nbin = int(round(nyq * math.sqrt(3.0)))
    acc = torch.zeros(7, nbin + 2, dtype=torch.float64, device=dev)
    sinc = lambda q: torch.where(q == 0, torch.ones_like(q), torch.sin(math.pi * q / ng) / (math.pi * q / ng))  # noqa: E731
    j = torch.arange(ng, device=dev)
    i = torch.arange(nyq + 1, device=dev)
    edge = (i == 0) | (i == nyq)
    for z in range(ng):  # one plane of modes at a time
        kr = torch.sqrt((kx[None, :] ** 2 + ky[:, None] ** 2 + ky[z] ** 2).double())
        s2 = (sinc(kx.double())[None, :] * sinc(ky.double())[:, None] * sinc(ky[z].double())) ** 2
        keep = ~(edge[None, :] & (j > nyq)[:, None])
        if z > nyq:
            keep &= ~(edge[None, :] & ((j == 0) | (j == nyq))[:, None])
        if z == 0:
            keep[0, 0] = False
        a = ck[z].abs() ** 2 * (4 * math.pi) * kr ** 3 / s2 ** 2
        b = torch.floor(kr + 0.5).long().clamp(max=nbin + 1)[keep]
        for q, x in enumerate((torch.ones_like(kr), kr, a, a, a, 1 / s2, 1 / s2 ** 2)):
            acc[q].index_add_(0, b, x[keep])
    v = acc[:, 1:nbin + 1].cpu().numpy()
    o = np.zeros((nbin, 10))
    with np.errstate(all="ignore"):
        o[:, 0] = v[0]
        o[:, 1] = v[1] / v[0] * 2 * math.pi / (case["cell"] * nc)
        o[:, 2:7] = (v[2:] / v[0]).T
        o[:, 7] = o[:, 4] / np.sqrt(o[:, 2] * o[:, 3])
        o[:, 8] = np.sqrt(o[:, 3] / o[:, 2])
        o[:, 9] = o[:, 7] ** 4 / o[:, 8] ** 2 * o[:, 3]
    return o


def _growth(a):
    h = OMEGA_M / a ** 3 + (1 - OMEGA_M - OMEGA_L) / a ** 2 + OMEGA_L
    def g(om, ol):
        return 2.5 * om / (om ** (4.0 / 7) - ol + (1 + om / 2) * (1 + ol / 70))
    return a * g(OMEGA_M / (a ** 3 * h), OMEGA_L / h) / g(OMEGA_M, OMEGA_L)


def _noise_filter(n, box, a, dev):
    """White noise to potential on an n^3 lattice: Eisenstein & Hu's no-wiggle spectrum normalised to sigma_8, times
    the discrete Laplacian's inverse with its short-range part taken from -1/r."""
    ob = 0.049
    k = np.logspace(-4, 2, 1000)
    theta, omh2, fb = 2.7255 / 2.7, OMEGA_M * H0 ** 2, ob / OMEGA_M
    s = 44.5 * np.log(9.83 / omh2) / np.sqrt(1 + 10 * (ob * H0 ** 2) ** 0.75)
    alpha = 1 - 0.328 * np.log(431 * omh2) * fb + 0.38 * np.log(22.3 * omh2) * fb ** 2
    q = k * theta ** 2 / (OMEGA_M * H0 * (alpha + (1 - alpha) / (1 + (0.43 * k * H0 * s) ** 4)))
    l0 = np.log(2 * math.e + 1.8 * q)
    t = l0 / (l0 + (14.2 + 731 / (1 + 62.5 * q)) * q * q)
    d2 = t ** 2 * k ** (3 + N_S) / (2 * math.pi ** 2)
    dk = np.empty_like(k)
    dk[0], dk[1:-1], dk[-1] = k[1] / 2, (k[2:] - k[:-2]) / 2, k[-1] - k[-2]
    x = 8 * k
    w = 3 * (np.sin(x) - np.cos(x) * x) / x ** 3
    d2 *= S8 ** 2 / np.sum((d2 * w * w * dk / k)[k <= 2 * math.pi * math.sqrt(3) * (n // 2) / box]) * _growth(a) ** 2
    f = torch.fft.fftfreq(n, d=1.0 / n, device=dev, dtype=torch.float64)
    kz, ky, kx = f.view(n, 1, 1), f.view(1, n, 1), torch.arange(n // 2 + 1, device=dev, dtype=torch.float64)
    kr = torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2).clamp_min(1.0)
    lk = torch.log(2 * math.pi / box * kr).cpu().numpy()
    spec = torch.as_tensor(np.exp(np.interp(lk, np.log(k), np.log(d2))), device=dev)
    hat = sum((2 * torch.sin(math.pi * c / n)) ** 2 for c in (kx, ky, kz)).clamp_min(1.0 / n ** 2)
    ker = -4 * math.pi / hat
    ker[0, 0, 0] = 0
    r = torch.fft.irfftn(ker.to(torch.complex128), s=(n, n, n))
    phi8 = (r[0, 0, 8] + r[0, 8, 0] + r[8, 0, 0] + r[0, 0, n - 8] + r[0, n - 8, 0] + r[n - 8, 0, 0]) / 6
    rr = torch.sqrt(f.view(n, 1, 1) ** 2 + f.view(1, n, 1) ** 2 + f.view(1, 1, n) ** 2)
    r = torch.where(rr > 8, r - (phi8 + 0.125), torch.where(rr > 0, -1 / rr.clamp_min(1e-30), torch.full_like(r, -2.5)))
    out = torch.sqrt(spec / (4 * math.pi) * (n / kr)) * (n / kr) * torch.fft.rfftn(r).real
    out[0, 0, 0] = 0
    return out


def _exact_gradient(case, seed):
    dev = torch.device("cuda")
    ng, npd, f64 = case["ng"], case["npd"], torch.float64
    a0, step = 0.1, ng // npd
    drift, kick, _ = D.schedule(9.0, 0.0, case["steps"], OMEGA_M, OMEGA_L)  # inputs of the pass, not its result
    vf = a0 ** 2 * 2 / (3 * math.sqrt(a0 ** 3)) * math.sqrt(1 + a0 * (1 - OMEGA_M - OMEGA_L) / OMEGA_M
                                                            + a0 ** 3 * OMEGA_L / OMEGA_M)
    mass = float(ng) ** 3 / float(npd) ** 3
    filt = _noise_filter(npd, case["box"], a0, dev)
    s = (2 * torch.sin(math.pi * torch.arange(ng, device=dev, dtype=f64) / ng)) ** 2
    k2 = s[: ng // 2 + 1].view(1, 1, -1) + s.view(1, -1, 1) + s.view(-1, 1, 1)
    green = -4 * math.pi / k2
    green[0, 0, 0] = 0
    lat = torch.arange(npd ** 3, device=dev)
    lat = torch.stack([lat % npd, lat // npd % npd, lat // npd ** 2], 1) * step

    def corners(x):
        fl = torch.floor(x).detach()
        w, c = x - fl, lat + fl.long()
        for k in range(8):
            o = (k & 1, k >> 1 & 1, k >> 2)
            wt = 1.0
            for d in range(3):
                wt = wt * (w[:, d] if o[d] else 1 - w[:, d])
            i = [(c[:, d] + o[d]) % ng for d in range(3)]
            yield (i[2] * ng + i[1]) * ng + i[0], wt

    def density(x):
        rho = torch.zeros(ng ** 3, dtype=f64, device=dev)
        for i, wt in corners(x):
            rho = rho.index_add(0, i, mass * wt)
        return rho.view(ng, ng, ng)

    def advance(x, v, dr, kk):
        x = x + dr * v
        phi = torch.fft.irfftn(torch.fft.rfftn(density(x)) * green, s=(ng, ng, ng))
        force = torch.stack([(torch.roll(phi, 1, d) - torch.roll(phi, -1, d)).reshape(-1) / 2 for d in (2, 1, 0)], 1)
        f = 0
        for i, wt in corners(x):
            f = f + wt[:, None] * force[i]
        return x, v + kk * f

    noise = _noise(case, seed).double()
    if case["backward"]:
        noise.requires_grad_(True)
    with torch.set_grad_enabled(case["backward"]):
        phi = torch.fft.irfftn(torch.fft.rfftn(noise.view(npd, npd, npd)) * filt, s=(npd, npd, npd))
        x = torch.stack([(torch.roll(phi, 1, d) - torch.roll(phi, -1, d)).reshape(-1) for d in (2, 1, 0)], 1)
        x = x * (step / (8 * math.pi))
        v = x * vf
        for dr, kk in zip(drift, kick):
            x, v = torch.utils.checkpoint.checkpoint(advance, x, v, float(dr), float(kk), use_reentrant=False)
        rho = density(x)
        out = {"x": x.detach(), "v": v.detach(), "rho": rho.detach()}
        if case["backward"]:
            ((rho - _target(case, seed).double()) ** 2).sum().backward()
            out["gnoise"] = noise.grad
    gc.collect()
    return out
