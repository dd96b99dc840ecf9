"""What the speed of this framework is measured on.

Each case is one call (or one cycle of calls) of a program that drives the
force path: forces of a configuration, a cycle of molecular dynamics between
two frames of a trajectory, a batch of small boxes, Widom insertions, the
adjoint.  The sizes are those of the configurations in
macsimus_gb300/configs.py and the tests (216, 864, 4352 and 32768 molecules;
256 ionic boxes), with ragged ones beside them.

Inputs come from the seed alone: molecules on an fcc lattice with vacancies,
displaced at random, with random orientations and Maxwell velocities, as a
run that starts from a crystal has them (cook's init="crystal").

The mixed path computes forces and moves sites with single-precision force
arithmetic; its results leave run() in single precision (forces as the
float32 tensor a learned or coarse-grained model takes, trajectories as the
float32 playback frames cook writes).  The FP64 path's results leave it in
double precision.
"""
import math

import numpy as np
import torch

import macsimus_gb300 as M
from macsimus_gb300 import configs, forcefield as ff


def listed():
    return [
        # the smallest box of the tests: a force call of a small program, energies
        # every time; launches and latency are what it pays for
        dict(name="forces_216", kind="forces", species="WAT", counts="216", density=0.997,
             cutoff=9.0, alpha=0.35, kn=7, measure=True),
        # cook itself with this library in place of forces(): host arrays in and
        # out on every call, 864 waters in L = 29.65 A
        dict(name="cook_864", kind="cook", species="WAT", counts="864", density=0.9916,
             cutoff=12.0, alpha=0.26, kn=8, measure=True),
        # the same box as device-resident MD, a cycle of 20 steps between two
        # frames, with the kernels the autotuner picks for it
        dict(name="md_864", kind="md", species="WAT", counts="864", density=0.9916, cutoff=12.0,
             alpha=0.26, kn=8, steps=20, pair_variant=10),
        # NaCl brine at 298 K: 4096 waters and 256 ions, thermostatted
        dict(name="md_brine", kind="md", species="WAT,NA,CL", counts="4096,128,128",
             density=1.06, cutoff=10.0, alpha=0.31, kn=12, steps=20, thermostat="bussi",
             pair_variant=9, cells=2),
        # a ragged brine evaluated with every option left at its default
        dict(name="forces_ragged", kind="forces", species="WAT,NA,CL", counts="2741,37,37",
             density=1.02, cutoff=10.0, alpha=0.31, kn=10, measure=True),
        # the headline: 32768 SPC/E waters (98304 sites), tuned, a cycle of 20 steps
        dict(name="md_32768", kind="md", species="WAT", counts="32768", density=0.997,
             cutoff=12.0, alpha=0.26, kn=20, steps=20, pair_variant=10, cells=2, serial=1),
        # forces of a large box for a program that never called the autotuner
        dict(name="forces_20011", kind="forces", species="WAT", counts="20011", density=0.997,
             cutoff=12.0, alpha=0.26, kn=17, measure=False),
        # Drude-polarizable water: ASPC k = 2 and one SCF iteration per step
        dict(name="md_drude", kind="md", species="WATD", counts="32768", density=0.997,
             cutoff=12.0, alpha=0.26, kn=20, steps=5, pair_variant=9, cells=2, serial=1),
        # 256 ionic-fluid boxes of 500 to 4000 sites stepped together
        dict(name="batch_256", kind="batch", nbox=256, nmin=500, nmax=4000, steps=20, sizes=0),
        # Widom insertions of a neutral probe into a batch of such boxes
        dict(name="widom_48", kind="widom", nbox=48, nmin=500, nmax=4000, insertions=100000,
             sizes=1),
        # the plain FP64 path on 864 waters with the tight SHAKE tolerance
        dict(name="fp64_864", kind="md", species="WAT", counts="864", density=0.9916,
             cutoff=12.0, alpha=0.26, kn=8, steps=5, precision="fp64", epsc=1e-10),
        # gradients with respect to the force field, FP64, on the brine
        dict(name="adjoint_brine", kind="adjoint", species="WAT,NA,CL", counts="4096,128,128",
             density=1.06, cutoff=10.0, alpha=0.31, kn=12),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces", "forces", "cook", "md", "md", "md", "drude", "tip4p", "batch",
                       "widom", "fp64", "adjoint"])
    if kind in ("batch", "widom"):
        nmin = _logint(rng, 500, 1500)
        c = dict(kind=kind, nbox=_logint(rng, 4, 128 if kind == "batch" else 32), nmin=nmin,
                 nmax=rng.randint(nmin + 100, 4000), sizes=rng.randint(2, 10 ** 6))
        c.update(steps=20) if kind == "batch" else c.update(insertions=_logint(rng, 2000, 100000))
        return c
    top = {"fp64": 900, "adjoint": 4000, "tip4p": 8000, "drude": 24000}.get(kind, 32000)
    n = _logint(rng, 220, top)
    density = rng.uniform(0.96, 1.06)
    if kind in ("drude", "tip4p"):
        species, counts = {"drude": "WATD", "tip4p": "T4P"}[kind], [n]
    elif rng.random() < 0.4 or kind == "adjoint":
        ions = max(1, int(n * rng.uniform(0.005, 0.04)))
        species, counts = "WAT,NA,CL", [n - 2 * ions, ions, ions]
    else:
        species, counts = "WAT", [n]
    L = _box(species, counts, density)
    cutoff = round(min(rng.uniform(9.0, 12.0), 0.485 * L), 3)
    alpha = round(3.12 / cutoff, 4)
    kn = max(5, int(math.ceil(rng.uniform(0.77, 0.95) * alpha * L)))
    if L / cutoff > 5.5:
        kn = min(kn, 20)
    c = dict(kind={"fp64": "md", "drude": "md", "tip4p": "md"}.get(kind, kind), species=species,
             counts=",".join(map(str, counts)), density=density, cutoff=cutoff, alpha=alpha,
             kn=kn)
    if c["kind"] == "md":
        c["steps"] = 5 if kind in ("fp64", "drude") else rng.choice([10, 20])
        if kind == "fp64":
            c.update(precision="fp64", epsc=1e-10)
        elif kind == "tip4p":
            c["thermostat"] = "nose"
        else:
            c["thermostat"] = rng.choice(["none", "none", "berendsen", "bussi"])
    if c["kind"] in ("forces", "cook"):
        c["measure"] = rng.random() < 0.5
    if kind in ("md", "forces") and n > 700:
        c["pair_variant"] = rng.choice([0, 9, 10, 10])
    if kind == "drude":
        c["pair_variant"] = 9
    if c.get("pair_variant") and n > 3000:
        c.update(cells=2, serial=1 if n > 8000 else 0)
    return c


# ----------------------------------------------------------------- inputs --

def _box(species, counts, density):
    return configs.box_length(species.split(","), counts, density)


def _crystal(species, counts, L, seed, T=298.0, h=0.002, jitter=0.12):
    """system, r, r1: whole molecules on a randomly occupied fcc lattice"""
    rng = np.random.default_rng(seed)
    system = ff.build_system(species, counts)
    nmol = sum(counts)
    n = 1
    while 4 * n ** 3 < nmol:
        n += 1
    i = np.arange(n)
    cells = np.stack(np.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 1, 3)
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    sites = ((cells + base[None]).reshape(-1, 3) + 0.25) * (L / n)
    x = sites[rng.permutation(len(sites))[:nmol]] + rng.normal(scale=jitter, size=(nmol, 3))
    r = np.zeros((system.ns, 3))
    v = np.zeros((system.ns, 3))
    mol = 0
    for s, cnt in zip(species, counts):
        sp = ff.SPECIES[s]()
        geo = np.asarray(sp.geometry) - sp.geometry[0]
        k = len(geo)
        a = system.mol_first[mol]
        m = system.mass[a:a + k]
        q = rng.normal(size=(cnt, 4))
        w, qx, qy, qz = (q / np.linalg.norm(q, axis=1)[:, None]).T
        R = np.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qz * w), 2 * (qx * qz + qy * w),
                      2 * (qx * qy + qz * w), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qx * w),
                      2 * (qx * qz - qy * w), 2 * (qy * qz + qx * w),
                      1 - 2 * (qx * qx + qy * qy)], -1).reshape(cnt, 3, 3)
        p = x[mol:mol + cnt, None] + np.einsum("nij,kj->nki", R, geo)
        vel = np.repeat(rng.normal(size=(cnt, 1, 3)) * math.sqrt(T / m.sum()), k, axis=1)
        if k > 1:
            d = p - (m[None, :, None] * p).sum(1, keepdims=True) / m.sum()
            inertia = (m[None, :, None] * d * d).sum((1, 2)) * 2 / 3
            omega = rng.normal(size=(cnt, 3)) * np.sqrt(T / inertia)[:, None]
            vel = vel + np.cross(omega[:, None], d)
        r[a:a + cnt * k] = p.reshape(-1, 3)
        v[a:a + cnt * k] = vel.reshape(-1, 3)
        mol += cnt
    v -= (system.mass[:, None] * v).sum(0) / system.mass.sum()
    r1 = h * v
    if system.polar:
        # shells start on their sites
        r, r1 = np.vstack([r, np.zeros_like(r)]), np.vstack([r1, np.zeros_like(r1)])
    return system, r, r1


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).pin_memory().numpy()


def _inputs(case, seed):
    species, counts = case["species"].split(","), [int(n) for n in case["counts"].split(",")]
    L = _box(case["species"], counts, case["density"])
    return (L, (case["kn"] + 1e-6) / L) + _crystal(species, counts, L, seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "widom"):
        # the boxes' sizes and parameters are the case's, their ions the seed's
        boxes = configs.ionic_boxes(case["nbox"], seed=case["sizes"], nmin=case["nmin"],
                                    nmax=case["nmax"])
        rng = np.random.default_rng(seed)
        for w in boxes:
            n = len(w["r"])
            w["r"] = w["r"][rng.permutation(n)] + rng.normal(scale=0.1, size=(n, 3))
            w["r1"] = w["r1"][rng.permutation(n)] * rng.choice([-1.0, 1.0], size=(n, 1))
        b = M.Batch([dict(system=w["system"], L=w["L"], cutoff=w["cutoff"], alpha=w["alpha"],
                          kappa=w["kappa"], h=w["h"]) for w in boxes])
        st = dict(case=case, batch=b, r=[_pinned(w["r"]) for w in boxes],
                  r1=[_pinned(w["r1"]) for w in boxes])
        if kind == "widom":
            # insertions go into the configuration of the last force evaluation
            for fp, r in zip(b.box, st["r"]):
                fp.forces(r)
            st["seed"] = 1 + seed
        return st
    L, kappa, system, r, r1 = _inputs(case, seed)
    kw = dict(precision=case.get("precision", "mixed"), epsc=case.get("epsc", 1e-7),
              pair_variant=case.get("pair_variant", 0), cells_per_cutoff=case.get("cells", 0),
              kspace_serial=case.get("serial", 0), thermostat=case.get("thermostat", "none"),
              seed=seed)
    if kind == "adjoint":
        kw["precision"] = "fp64"
    fp = M.ForcePath(system, [L] * 3, case["cutoff"], case["alpha"], kappa, **kw)
    st = dict(case=case, fp=fp)
    if kind == "forces":
        st["stream"] = torch.cuda.Stream()
        fp.set_stream(st["stream"].cuda_stream)
        st["r"] = torch.from_numpy(r.reshape(-1)).cuda()
        st["f"] = torch.empty_like(st["r"])
    else:
        st["r"], st["r1"] = _pinned(r), _pinned(r1)
    if kind == "adjoint":
        st["g"] = _pinned(np.random.default_rng(seed + 1).normal(scale=1e-3, size=r.shape))
    return st


# -------------------------------------------------------------------- run --

def _energies(en):
    # the parts, each of the size of the Ewald sums (el cancels almost to nothing
    # between molecules of random orientation)
    return dict(er=en["er"], ek=en["ek"], lj=en["lj"], vir=en["vir"],
                Pvir=np.array(en["Pvir"], np.float32))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forces":
        # a program that keeps its configuration in device tensors, on its own stream
        en = state["fp"].forces_device(state["r"].data_ptr(), state["f"].data_ptr(),
                                       measure=case["measure"])
        with torch.cuda.stream(state["stream"]):
            out = dict(f=state["f"].float())
        return dict(out, **_energies(en)) if en else out
    if kind == "cook":
        f, en = state["fp"].forces(state["r"], measure=case["measure"])
        f = f.astype(np.float32)
        return dict(f=f, **_energies(en)) if en else dict(f=f)
    if kind == "md":
        fp = state["fp"]
        fp.md_set_state(state["r"], state["r1"])
        en = fp.md_steps(case["steps"])
        sums = [en["er"], en["ek"], en["lj"], en["ekin"], en["vir"], en["virc"]]
        if case.get("precision") == "fp64":
            r, r1 = fp.md_get_state()
            return dict(r=r, r1=r1, sums=np.array(sums))
        frames = ["plb", "vlb"] + (["dlb"] if fp.polar else [])
        return dict({w: fp.playback_frame(w)[1] for w in frames},
                    sums=np.array(sums, np.float32))
    if kind == "batch":
        b = state["batch"]
        for fp, r, r1 in zip(b.box, state["r"], state["r1"]):
            fp.md_set_state(r, r1)
        en = b.md_steps(case["steps"])
        return dict(
            plb=np.concatenate([fp.playback_frame("plb")[1] for fp in b.box]),
            vlb=np.concatenate([fp.playback_frame("vlb")[1] for fp in b.box]),
            sums=np.array([[e["er"], e["ek"], e["lj"], e["ekin"], e["vir"]] for e in en], np.float32))
    if kind == "widom":
        # the third type of an ionic system is the neutral LJ probe
        res = state["batch"].widom([2], n=case["insertions"], seed=state["seed"], T=298.0)
        return dict(raw=np.array([w["raw"] for w in res], np.float32),
                    widom=np.array([w["widom"] for w in res], np.float32))
    if kind == "adjoint":
        return state["fp"].adjoint(state["r"], state["g"])
    raise ValueError(kind)


def work(case):
    """bytes: positions (and velocities) in, forces or frames out; flops: 45
    per pair of sites within the cutoff and 8 per (k-vector, charge) in each
    of the two Ewald sums, per force evaluation"""
    kind = case["kind"]
    if kind in ("batch", "widom"):
        n = 0.5 * (case["nmin"] + case["nmax"])
        ns = n * case["nbox"]
        if kind == "widom":
            # 2.5 sigma spheres at reduced density 0.8: 52 sites per probe
            return dict(bytes=16 * ns, flops=52.0 * 20 * case["insertions"] * case["nbox"])
        kn = 1.08 * 3.1 / (2.5 * 4.0) * (n * 3.75 ** 3 / 0.8) ** (1 / 3)
        per = 45 * n * 33 + 16 * n * 2 / 3 * math.pi * kn ** 3
        return dict(bytes=72 * ns, flops=per * case["nbox"] * case["steps"])
    counts = [int(n) for n in case["counts"].split(",")]
    L = _box(case["species"], counts, case["density"])
    size = {"WAT": (3, 3), "WATD": (3, 4), "T4P": (4, 3), "NA": (1, 1), "CL": (1, 1)}
    names = case["species"].split(",")
    ns = sum(size[s][0] * c for s, c in zip(names, counts))
    nq = sum(size[s][1] * c for s, c in zip(names, counts))
    pairs = 0.5 * ns * ns * 4 / 3 * math.pi * case["cutoff"] ** 3 / L ** 3
    nk = 2 / 3 * math.pi * case["kn"] ** 3
    flops = 45 * pairs + 16 * nk * nq
    if kind == "md":
        return dict(bytes=(48 + 24) * ns, flops=flops * case["steps"])
    return dict(bytes=(24 + 12) * ns if kind != "adjoint" else 64 * ns, flops=flops)


# ------------------------------------------------------------ exact values --

def _smooth_lj(eps, rmin, c2):
    """the switch radius c1 at which LJ (depth eps, minimum at rmin) meets
    a (r^2 - c2^2)^2 with equal value and slope"""
    def u(r):
        x = (rmin / r) ** 6
        return eps * (x * x - 2 * x)

    def fr(r):
        x = (rmin / r) ** 6
        return 12 * eps * (x * x - x) / (r * r)
    # f/r of a (r^2 - c2^2)^2 is 4 a (c2^2 - r^2) with a = u / (r^2 - c2^2)^2
    c1 = 0.775 * c2
    for _ in range(500):
        c1 = c2 / math.sqrt(1 + 4 * u(c1) / (c1 * c1 * fr(c1)))
    return c1, u(c1) / (c2 * c2 - c1 * c1) ** 2


def _hyperbolic(alpha, cutoff, grid=256, margin=2.5):
    """the path's r-space functions, erfc(alpha r)/r and its -d/dr / r as
    A + B / (C + r^2) on intervals of alpha^2 r^2, slopes continuous, shifted
    to zero at the cutoff: [n, 6] and the intervals per A^2"""
    n = int(((cutoff + margin) * alpha) ** 2 * grid) + 1
    h = 1.0 / grid
    x = np.arange(n + 3) * h
    s = np.sqrt(np.maximum(x, 1e-300))
    er = torch.erfc(torch.from_numpy(s)).numpy() / s
    fn = [er.copy(), (2 / math.sqrt(math.pi) * np.exp(-x) + er) / np.maximum(x, 1e-300)]
    tab = np.zeros((n, 6))
    for m, f in enumerate(fn):
        f[0] = 9e9
        D = (-f[n + 2] + 8 * f[n + 1] - 8 * f[n - 1] + f[n - 2]) / (12 * h)
        for i in range(n - 1, -1, -1):
            d = f[i + 1] - f[i]
            Cc = (x[i] * d - x[i + 1] * D * h) / (D * h - d)
            B = -D * (Cc + x[i + 1]) ** 2
            tab[i, 3 * m:3 * m + 3] = (f[i + 1] + D * (Cc + x[i + 1])) * alpha ** (1 + 2 * m), \
                B * alpha ** (2 * m - 1), Cc / alpha ** 2
            D = -B / (Cc + x[i]) ** 2
    sg = grid * alpha * alpha
    c2 = cutoff * cutoff
    row = tab[int(c2 * sg)].copy()
    tab[:, 0] -= row[1] / (row[2] + c2) + row[0]
    tab[:, 3] -= row[4] / (row[5] + c2) + row[3]
    return tab, sg


def exact(case, seed):
    if case["kind"] not in ("forces", "cook"):
        return None
    L, kappa, system, r, _ = _inputs(case, seed)
    dev, f64 = "cuda", torch.float64
    cutoff, alpha, ns = case["cutoff"], case["alpha"], system.ns
    x = torch.from_numpy(r).to(dev)
    q = torch.from_numpy(system.q).to(dev)
    typ = torch.from_numpy(system.type).to(dev).long()
    mol = torch.from_numpy(system.mol).to(dev)
    nt = len(system.typeE)
    lj = np.zeros((nt, nt, 4))     # eps, rmin, c1, a
    for a in range(nt):
        for b in range(nt):
            e = math.sqrt(system.typeE[a] * system.typeE[b])
            if e:
                rm = system.typeR[a] + system.typeR[b]
                lj[a, b] = (e, rm) + _smooth_lj(e, rm, cutoff)
    lj = torch.from_numpy(lj.reshape(nt * nt, 4)).to(dev)
    tab, sg = _hyperbolic(alpha, cutoff)
    tab = torch.from_numpy(tab).to(dev)
    f = torch.zeros(ns, 3, dtype=f64, device=dev)
    er = elj = vir = 0.0
    P = torch.zeros(3, 3, dtype=f64, device=dev)
    step = max(1, int(1.2e8) // ns)
    for i0 in range(0, ns, step):
        r2 = torch.zeros(min(step, ns - i0), ns, dtype=f64, device=dev)
        for d in range(3):
            dx = x[i0:i0 + step, d, None] - x[None, :, d]
            dx -= torch.round(dx / L) * L
            r2 += dx * dx
        i, j = torch.nonzero(r2 < cutoff * cutoff, as_tuple=True)
        del r2, dx
        i = i + i0
        keep = i != j
        i, j = i[keep], j[keep]
        d = x[i] - x[j]
        d -= torch.round(d / L) * L
        r2 = (d * d).sum(1)
        qq = q[i] * q[j]
        same = mol[i] == mol[j]
        # between molecules: LJ and the splined erfc terms
        t = tab[(r2 * sg).long().clamp(max=len(tab) - 1)]
        u = qq * (t[:, 1] / (t[:, 2] + r2) + t[:, 0])
        fr = qq * (t[:, 4] / (t[:, 5] + r2) + t[:, 3])
        p = lj[typ[i] * nt + typ[j]]
        s6 = (p[:, 1] ** 2 / r2) ** 3
        near = r2 < p[:, 2] ** 2
        gap = cutoff * cutoff - r2
        ul = torch.where(near, p[:, 0] * (s6 * s6 - 2 * s6), p[:, 3] * gap * gap)
        fl = torch.where(near, 12 * p[:, 0] * (s6 * s6 - s6) / r2, 4 * p[:, 3] * gap)
        ul, fl = (torch.where(same, torch.zeros_like(v), v) for v in (ul, fl))
        # within a molecule: minus the smooth part of the Ewald sum
        rr = r2.sqrt()
        ex = -torch.erf(alpha * rr) / rr
        fx = (ex + 2 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2)) / r2
        u, fr = torch.where(same, qq * ex, u), torch.where(same, qq * fx, fr)
        er += 0.5 * u.sum().item()
        elj += 0.5 * ul.sum().item()
        vir += 0.5 * (fl * r2).sum().item()
        fv = (fr + fl)[:, None] * d
        f.index_add_(0, i, fv)
        P += 0.5 * d.T @ fv
    # k-space over the whole sphere |k| <= kappa; k = n / L
    K = int(L * kappa)
    n = torch.arange(-K, K + 1, dtype=f64, device=dev)
    ph = torch.exp(2j * math.pi / L * n[:, None, None] * x.T[None])    # [2K+1, 3, ns]
    X, Y, Z = ph[:, 0], ph[:, 1], ph[:, 2]
    kk = (n[:, None, None] ** 2 + n[None, :, None] ** 2 + n[None, None, :] ** 2) / L ** 2
    w = torch.where((kk > 0) & (kk <= kappa * kappa),
                    torch.exp(-(math.pi / alpha) ** 2 * kk) / (2 * math.pi * L ** 3)
                    / kk.clamp(min=1e-300), torch.zeros_like(kk))
    S = torch.stack([(X[a] * q * Y) @ Z.T for a in range(2 * K + 1)])
    A = w * (S.real ** 2 + S.imag ** 2)
    ek = A.sum().item()
    P += ek * torch.eye(3, dtype=f64, device=dev)
    g = 2 * A * (1 / kk.clamp(min=1e-300) + (math.pi / alpha) ** 2)
    g[K, K, K] = 0
    nn = [n[:, None, None] / L, n[None, :, None] / L, n[None, None, :] / L]
    for a in range(3):
        for b in range(3):
            P[a, b] -= (g * nn[a] * nn[b]).sum()
    # f_j = -grad of the energy: 4 pi q_j sum w Im(conj(S) exp(2 pi i k r_j)) k
    W = w * S.conj()
    for a in range(2 * K + 1):
        H, Hz = W[a] @ Z, (W[a] * n) @ Z                   # [2K+1 (ky), ns]
        e = X[a] * Y
        c = 4 * math.pi / L * q
        f[:, 0] += c * n[a] * (e * H).sum(0).imag
        f[:, 1] += c * (e * n[:, None] * H).sum(0).imag
        f[:, 2] += c * (e * Hz).sum(0).imag
    out = dict(f=f.reshape(-1) if case["kind"] == "forces" else f)
    if case["measure"]:
        out.update(er=er, ek=ek, lj=elj, vir=vir,
                   Pvir=np.array([P[0, 0].item(), P[1, 1].item(), P[2, 2].item(),
                                  P[1, 2].item(), P[2, 0].item(), P[0, 1].item()]))
    return out
