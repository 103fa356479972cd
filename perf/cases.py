"""Timing cases of the SCF hot path, through the calls a program makes.

Kinds (the ranges that draw() covers are those of the configurations, the
training families and the density-file grids of this repository):

  post      the non-eigensolver part of a short SCF: LDA, potential update and
            msecant1 mixing, eight iterations on one grid
  step      one SCF iteration as solver.run_rsdft_calculation runs it:
            chefsi1, occupations, density, Hartree solve, LDA, update, mixing
  filter    the Chebyshev filter of a block (mode 1: first_filt's slim filter
            of a random block, mode 0: chefsi1's scaled filter)
  hx        H @ X for a block
  hartree   the Hartree solve (plain CG, or preconditioned with cg_prec = 1)
  setup     what every SCF does before its first iteration: grid context, SAD
            density and potentials, projector tables
  net_fwd   the learned start's network, forward
  net_grad  forward, loss and backward of one training step

Inputs are drawn from the seed alone: geometries are a configuration's atoms
displaced by 0.05 A, the local potential is a sum of smooth wells at the
atoms, blocks are box modes with noise (or random, for first_filt).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from parsec_python_b200 import gpu, learned, workloads
from parsec_python_b200._lib import F32, F64
from parsec_python_b200.inputs import ElementTable, pseudo_tables
from parsec_python_b200.models import A0_ANG

BOHR = 1.0 / A0_ANG
POST_ITERATIONS = 8
# FD second-derivative weights of -d2/dx2 by order: centre, then distance 1..4
FD = {2: (2.0, -1.0), 4: (5.0 / 2, -4.0 / 3, 1.0 / 12), 6: (49.0 / 18, -3.0 / 2, 3.0 / 20, -1.0 / 90),
      8: (205.0 / 72, -8.0 / 5, 1.0 / 5, -8.0 / 315, 1.0 / 560)}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # small density-file grid (24^3, as the ML-grid inputs): launch latency is everything
        {"name": "post_24", "kind": "post", "nx": 24, "ny": 24, "nz": 24, "h": 0.25},
        # the H2O configuration with default options: FP64, plain CG, 27 columns
        {"name": "step_h2o_f64", "kind": "step", "system": "h2o", "nx": 52, "ny": 52, "nz": 52, "h": 0.2, "nev": 12,
         "deg": 10, "dtype": "f64", "cg_prec": 0, "late": 0},
        # the C10H8 configuration, FP64 with the preconditioned Hartree solve
        {"name": "step_c10h8_f64", "kind": "step", "system": "c10h8", "nx": 78, "ny": 78, "nz": 78, "h": 0.18,
         "nev": 40, "deg": 12, "dtype": "f64", "cg_prec": 1, "late": 0},
        # the benchmark's chosen form at its own size: mixed precision, early phase
        {"name": "step_si87h76_mixed", "kind": "step", "system": "si87h76", "nx": 90, "ny": 90, "nz": 90, "h": 0.25,
         "nev": 292, "deg": 16, "dtype": "f32", "cg_prec": 1, "late": 0},
        # first filter of the Si35H36 configuration in FP32 on the sphere-masked domain
        {"name": "filter_si35h36_f32_sphere", "kind": "filter", "system": "si35h36", "nx": 74, "ny": 74, "nz": 74,
         "h": 0.25, "k": 143, "deg": 10, "mode": 1, "dtype": "f32", "mask": 1, "order": 8},
        # the filter of a later iteration at the largest configuration, FP32
        {"name": "filter_si87h76_f32", "kind": "filter", "system": "si87h76", "nx": 90, "ny": 90, "nz": 90, "h": 0.25,
         "k": 307, "deg": 16, "mode": 0, "dtype": "f32", "mask": 0, "order": 8},
        # H X on a density-file grid with odd, unequal sides
        {"name": "hx_odd_f64", "kind": "hx", "system": "water", "geom": 3, "nx": 61, "ny": 55, "nz": 67, "h": 0.2,
         "k": 31, "dtype": "f64", "mask": 0, "order": 8},
        # the default Hartree solve on the C10H8 grid (stops at its 200 iterations)
        {"name": "hartree_c10h8_plain", "kind": "hartree", "nx": 78, "ny": 78, "nz": 78, "h": 0.18, "prec": 0,
         "order": 8},
        # the preconditioned one on the water training grid
        {"name": "hartree_water_prec", "kind": "hartree", "nx": 92, "ny": 92, "nz": 92, "h": 0.2, "prec": 1,
         "order": 8},
        # setup of the largest configuration (163 atoms)
        {"name": "setup_si87h76", "kind": "setup", "system": "si87h76", "nx": 90, "ny": 90, "nz": 90, "h": 0.25},
        # the learned start on the benchmark's grid
        {"name": "net_fwd_90", "kind": "net_fwd", "nx": 90, "ny": 90, "nz": 90},
        # gradient of one training step on the Si-H family's grid
        {"name": "net_grad_82", "kind": "net_grad", "nx": 82, "ny": 82, "nz": 82},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """Sides of a drawn grid: a cube with an even side (an .in file's domain),
    or the unequal sides of a density file."""
    if rng.random() < 0.5:
        n = 2 * rng.randint(lo // 2, hi // 2)
        return {"nx": n, "ny": n, "nz": n}
    return {"nx": rng.randint(lo, hi), "ny": rng.randint(lo, hi), "nz": rng.randint(lo, hi)}


def _geometry(rng):
    return {"system": rng.choice(["water", "sih"]), "geom": rng.randint(0, 500)}


def draw(rng):
    kind = rng.choice(["post", "step", "filter", "hx", "hartree", "setup", "net_fwd", "net_grad"])
    h = round(rng.uniform(0.18, 0.27), 4)
    if kind == "post":
        return {"kind": kind, **_grid(rng, 20, 92), "h": h}
    if kind == "setup":
        return {"kind": kind, **_geometry(rng), **_grid(rng, 48, 92), "h": h}
    if kind == "hartree":
        prec = rng.randint(0, 1)
        return {"kind": kind, **_grid(rng, 24, 92 if prec else 80), "h": h, "prec": prec,
                "order": rng.choice([8, 8, 8, 6, 4])}
    if kind in ("net_fwd", "net_grad"):
        return {"kind": kind, **_grid(rng, 32, 88)}
    g = _grid(rng, 44, 90)
    n = g["nx"] * g["ny"] * g["nz"]
    dtype = rng.choice(["f64", "f32"])
    size = 8 if dtype == "f64" else 4
    if kind == "step":
        # FP64 blocks on top of an FP32-sized budget: columns bounded by the block's bytes
        k = min(_log_int(rng, 24, 300), int(4e8 / (n * size)), 160)
        return {"kind": kind, **_geometry(rng), **g, "h": h, "nev": max(9, k - 15), "deg": rng.randint(8, 16),
                "dtype": dtype, "cg_prec": rng.randint(0, 1), "late": rng.randint(0, 1)}
    k = max(4, min(_log_int(rng, 8, 307), int(8e8 / (n * size))))
    case = {"kind": kind, **_geometry(rng), **g, "h": h, "k": k, "dtype": dtype,
            "mask": 1 if rng.random() < 0.25 else 0, "order": rng.choice([8, 8, 8, 6, 4])}
    if kind == "filter":
        case.update(deg=rng.randint(8, 16), mode=rng.randint(0, 1))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _h(case):
    return case.get("h", 0.25) * BOHR


def _domain(case):
    h = _h(case)
    return {"nx": case["nx"], "ny": case["ny"], "nz": case["nz"], "h": h, "radius": 0.5 * h * (case["nx"] - 1)}


def _atoms(case, seed):
    """The system's atoms in bohr, displaced by 0.05 A, in the frame of the
    grid (point i of an axis at i h - radius, radius that of x)."""
    name = case["system"]
    if name == "water":
        atoms = workloads.water_cluster(case["geom"])
    elif name == "sih":
        atoms = workloads.sih_random_cluster(case["geom"], nmax=20)
    else:
        atoms = workloads.CONFIGS[name]["atoms"]()
    rng = np.random.default_rng(int(seed))
    h = _h(case)
    shift = 0.5 * h * (np.array([case["nx"], case["ny"], case["nz"]]) - case["nx"])
    out = []
    for a in atoms:
        c = np.asarray(a["coord"], dtype=float).reshape(-1, 3)
        out.append({"typ": a["typ"], "coord": (c + 0.05 * rng.standard_normal(c.shape)) * BOHR + shift})
    return out


def _axes(case):
    h = _h(case)
    ax = [torch.arange(case[d], dtype=torch.float64, device="cuda") * h for d in ("nx", "ny", "nz")]
    return ax


def _gaussians(case, centres, weights, widths):
    """sum_a w_a exp(-|r - c_a|^2 / (2 s_a^2)) on the grid, x fastest; centres
    from the first grid point."""
    x, y, z = _axes(case)
    out = torch.zeros(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device="cuda")
    for c, w, s in zip(centres, weights, widths):
        ex = torch.exp(-(x - c[0]) ** 2 / (2 * s * s))
        ey = torch.exp(-(y - c[1]) ** 2 / (2 * s * s))
        ez = torch.exp(-(z - c[2]) ** 2 / (2 * s * s))
        out += (w * ez)[:, None, None] * (ey[:, None] * ex[None, :])[None]
    return out.reshape(-1)


def _smooth(case, rng, count=12, scale=1.0):
    """A random smooth field: Gaussians of either sign inside the grid."""
    h = _h(case)
    ext = h * (np.array([case["nx"], case["ny"], case["nz"]]) - 1)
    return _gaussians(case, rng.uniform(0.2, 0.8, (count, 3)) * ext, scale * rng.standard_normal(count),
                      rng.uniform(0.08, 0.2, count) * ext.min())


def _centres(case, atoms):
    pts = np.vstack([a["coord"] for a in atoms])
    return pts + 0.5 * _h(case) * (case["nx"] - 1)


def _potential(case, atoms):
    """Smooth attractive wells (Hartree), deeper at the heavy atoms."""
    w, s = [], []
    for a in atoms:
        m = len(a["coord"])
        w += [-(0.7 if a["typ"] == "H" else 1.6)] * m
        s += [1.0 if a["typ"] == "H" else 1.5] * m
    return _gaussians(case, _centres(case, atoms), w, s)


def _density(case, atoms, electrons):
    """Smooth positive density in electrons per point with the given count."""
    w = [1.0 if a["typ"] == "H" else 4.0 for a in atoms for _ in range(len(a["coord"]))]
    rho = _gaussians(case, _centres(case, atoms), w, [1.6] * len(w)) + 1e-9
    return rho * (electrons / rho.sum())


def _modes(case, k, gen, dtype):
    """k box modes of lowest kinetic energy with 1 % noise, and their energies."""
    h = _h(case)
    dims = (case["nx"], case["ny"], case["nz"])
    m = 12
    q = [np.pi * np.arange(1, min(m, d) + 1) / (h * (d + 1)) for d in dims]
    e = 0.5 * (q[2][:, None, None] ** 2 + q[1][None, :, None] ** 2 + q[0][None, None, :] ** 2)
    order = np.argsort(e, axis=None, kind="stable")[:k]
    iz, iy, ix = np.unravel_index(order, e.shape)
    s = [torch.sin(torch.arange(1, d + 1, dtype=torch.float64, device="cuda")[None, :] *
                   torch.arange(1, min(m, d) + 1, dtype=torch.float64, device="cuda")[:, None] * (np.pi / (d + 1)))
         * math.sqrt(2.0 / (d + 1)) for d in dims]
    n = dims[0] * dims[1] * dims[2]
    X = torch.empty(k, n, dtype=dtype, device="cuda")
    for c in range(k):
        X[c] = (s[2][iz[c]][:, None, None] * s[1][iy[c]][None, :, None] * s[0][ix[c]][None, None, :]).reshape(-1)
    noise = torch.randn(k, n, dtype=dtype, device="cuda", generator=gen)
    X.add_(noise, alpha=0.01 / math.sqrt(n))
    return X, e.reshape(-1)[order]


def _kinetic_top(h, order):
    """Upper bound of 0.5 A: three axes of the stencil's largest symbol."""
    c = FD[order]
    return 1.5 * (c[0] + 2 * sum(abs(v) for v in c[1:])) / (h * h)


def _hamiltonian(case, seed):
    ctx = gpu.GridContext(_domain(case), case.get("order", 8), seed=int(seed) & 0xFFFF)
    if case.get("mask"):
        ctx.set_sphere_mask(0.5 * ctx.h * (min(ctx.nx, ctx.ny, ctx.nz) - 1))
    atoms = _atoms(case, seed)
    gpu.projector_setup(ctx, atoms, ElementTable(), pseudo_tables())
    pot = _potential(case, atoms)
    return ctx, atoms, pot, gpu.Hamiltonian(ctx, pot)


def _net_inputs(case, ctx, net, seed):
    rng = np.random.default_rng(int(seed))
    h = _h(case)
    ext = h * (np.array([case["nx"], case["ny"], case["nz"]]) - 1)
    c = rng.uniform(0.25, 0.75, (20, 3)) * ext
    rho = _gaussians(case, c, [0.3] * 20, [1.5] * 20)
    vloc = _gaussians(case, c, [-1.5] * 20, [1.2] * 20)
    delta = _gaussians(case, c + 0.3 * rng.standard_normal(c.shape), 0.03 * rng.standard_normal(20), [1.3] * 20)
    net.scales = {"a0": 1.0 / float(rho.std()), "a1": 1.0 / float(vloc.std()), "at": 1.0 / float(delta.std())}
    return rho, vloc, (delta * net.scales["at"]).float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    st = {"case": case, "seed": int(seed)}
    if kind == "post":
        rng = np.random.default_rng(int(seed))
        ctx = gpu.GridContext(_domain(case), 8)
        rho = torch.exp(_smooth(case, rng)) * 0.05
        st.update(ctx=ctx, ppot=_smooth(case, rng), hpot0=_smooth(case, rng), rho=[], hpot=[], pot=[])
        base, target = _smooth(case, rng, scale=0.3), st["ppot"] + st["hpot0"]
        for i in range(POST_ITERATIONS):
            w = 0.5 ** i
            st["rho"].append(rho * (1.0 + 0.1 * w * torch.tanh(_smooth(case, rng))))
            st["hpot"].append(base + 0.2 * w * _smooth(case, rng))
            st["pot"].append(target + base - 0.2 + w * _smooth(case, rng))
    elif kind == "step":
        ctx, atoms, pot, H = _hamiltonian(case, seed)
        dt = torch.float64 if case["dtype"] == "f64" else torch.float32
        nev = case["nev"]
        X, e = _modes(case, nev + 15, gen, dt)
        nelec = 2 * max(1, int(0.72 * nev))
        rng = np.random.default_rng(int(seed) + 1)
        rho0 = _density(case, atoms, nelec)
        lam = torch.from_numpy(np.sort(e - 0.6)).to("cuda")
        hpot0 = 0.1 * _smooth(case, rng)
        st.update(ctx=ctx, H=H, A=gpu.Laplacian(ctx), X=X, lam=lam, pot=pot, rho0=rho0, nelec=float(nelec),
                  hpot=torch.zeros_like(pot), hpot0=hpot0, ppot=pot - hpot0)
        if case["dtype"] == "f32":   # the solver's phases of mixed precision
            for name in ("psc_set_gemm_impl", "psc_set_gram_impl"):
                ctx.call(name, 0 if case["late"] else 1)
    elif kind in ("filter", "hx"):
        ctx, atoms, pot, H = _hamiltonian(case, seed)
        dt = torch.float64 if case["dtype"] == "f64" else torch.float32
        if kind == "filter" and case["mode"] == 1:
            X = torch.rand(case["k"], ctx.n, dtype=dt, device="cuda", generator=gen)
        else:
            X, _ = _modes(case, case["k"], gen, dt)
        st.update(ctx=ctx, H=H, pot=pot, X=ctx.mask_block(X))
        if kind == "filter":
            top = _kinetic_top(_h(case), case["order"]) + 1.0
            bounds = [-0.8, 1.2, top] if case["mode"] == 0 else [0.0, 0.3 * top, top]
            st.update(W=torch.empty_like(X), T=torch.empty_like(X),
                      bounds=torch.tensor(bounds, dtype=torch.float64, device="cuda"))
    elif kind == "hartree":
        rng = np.random.default_rng(int(seed))
        ctx = gpu.GridContext(_domain(case), case["order"])
        drho = _smooth(case, rng, scale=0.02)
        st.update(ctx=ctx, A=gpu.Laplacian(ctx), rhs=4 * np.pi * (drho - drho.mean()),
                  x0=0.01 * _smooth(case, rng))
    elif kind == "setup":
        st.update(atoms=_atoms(case, seed), elem=ElementTable(), tables=pseudo_tables())
    else:
        ctx = gpu.GridContext(_domain(case), 8)
        net = learned.UNet3D(ctx, seed=int(seed) & 0xFFFF)
        rho, vloc, target = _net_inputs(case, ctx, net, seed)
        st.update(ctx=ctx, net=net, rho=rho, vloc=vloc, target=target)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    ctx = st.get("ctx")
    if kind == "post":
        mixer = gpu.Mixer(ctx, POST_ITERATIONS + 2)
        out = {}
        for i in range(POST_ITERATIONS):
            vxc, xc = gpu.lda_xc(ctx, st["rho"][i])
            pot_new, f, sums = gpu.scf_update(ctx, st["ppot"], vxc, st["hpot"][i], st["hpot0"], st["rho"][i],
                                              st["pot"][i])
            mixed, used = mixer(st["pot"][i], f)
            out[f"xc{i}"], out[f"sums{i}"], out[f"mixed{i}"] = xc, sums, mixed
        out.update(vxc=vxc, pot_new=pot_new, f=f, used=used)
        return out
    if kind == "step":
        nev = case["nev"]
        H = st["H"]
        H.set_potential(st["pot"])
        # the filter works in place: the block of the last iteration is kept for the next pass
        W, lam = gpu.chefsi1(st["X"].clone(), st["lam"], case["deg"], nev, H)
        ef, occ = gpu.occupations(ctx, lam[:nev], 500.0, st["nelec"], 1e-6)
        rho, hrhs = gpu.density(ctx, W, nev, occ, st["rho0"])
        prec = ("spectral", "precLU") if case["cg_prec"] else ()
        hpot, its = gpu.pcg(st["A"], hrhs, st["hpot"], 200, 1e-5, *prec)
        vxc, xc = gpu.lda_xc(ctx, rho)
        pot_new, f, sums = gpu.scf_update(ctx, st["ppot"], vxc, hpot, st["hpot0"], rho, st["pot"])
        mixed, _ = gpu.Mixer(ctx, 42)(st["pot"], f)
        # the eigenvectors are not returned: their signs (and rotations of
        # close pairs) are free; the density is what they determine
        return {"lam": lam, "occ": occ, "ef": ef, "rho": rho, "hrhs": hrhs, "hpot": hpot, "its": its, "vxc": vxc,
                "xc": xc, "pot_new": pot_new, "f": f, "sums": sums, "mixed": mixed}
    if kind == "filter":
        st["W"].copy_(st["X"])
        Y, _ = gpu.cheb_filter(st["H"], st["W"], st["T"], case["deg"], st["bounds"], case["mode"])
        return Y
    if kind == "hx":
        return st["H"] @ st["X"]
    if kind == "hartree":
        prec = ("spectral", "precLU") if case["prec"] else ()
        x, its = gpu.pcg(st["A"], st["rhs"], st["x0"], 200, 1e-5, *prec)
        return {"x": x, "its": its}
    if kind == "setup":
        ctx = gpu.GridContext(_domain(case), 8)
        rho0, hpot0, ppot, info = gpu.sad_setup(ctx, st["atoms"], st["elem"], st["tables"])
        proj = gpu.projector_setup(ctx, st["atoms"], st["elem"], st["tables"])
        return {"rho0": rho0, "hpot0": hpot0, "ppot": ppot, "electrons": info["electron_count_initial"],
                "normalized": info["electron_count_normalized"], "atoms": proj.n_atoms, "points": proj.n_points,
                "touched": proj.n_touched}
    net = st["net"]
    out = net.forward(net.pack(st["rho"], st["vloc"]))
    if kind == "net_fwd":
        return out
    loss, grad = net.loss_and_grad(out, st["target"])
    net.backward(grad)
    return {"out": out, "loss": loss, "grad": net.grad}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _hx_flops(order):
    return 2 * (3 * order + 1) + 5


def work(case):
    kind = case["kind"]
    n = case["nx"] * case["ny"] * case["nz"]
    size = 8 if case.get("dtype", "f64") == "f64" else 4
    if kind == "post":
        # per iteration: rho, hpot, pot, x and f in, vxc, pot_new and f, x out; the history once
        m = POST_ITERATIONS
        return {"bytes": 8.0 * n * (12 * m + m * (m - 1)), "flops": 60.0 * n * m}
    if kind == "setup":
        return {"bytes": 3 * 8.0 * n, "flops": 60.0 * n}
    if kind == "hartree":
        its = 3 if case["prec"] else 200
        mm = 12.0 * n * (case["nx"] + case["ny"] + case["nz"]) / 3 if case["prec"] else 0.0
        return {"bytes": 3 * 8.0 * n, "flops": its * (n * (2.0 * (3 * case["order"] + 1) + 10) + mm)}
    if kind in ("hx", "filter"):
        steps = case.get("deg", 1)
        frac = 1.0
        if case["mask"]:
            m = min(case["nx"], case["ny"], case["nz"])
            frac = math.pi / 6 * m ** 3 / n
        k = case["k"]
        if kind == "hx":
            return {"bytes": size * frac * n * (2 * k + 1), "flops": frac * n * k * _hx_flops(case["order"])}
        # every step reads two blocks and writes one (the first reads one)
        return {"bytes": size * frac * n * ((3 * steps - 1) * k + steps),
                "flops": steps * frac * n * k * _hx_flops(case["order"])}
    if kind == "step":
        k = case["nev"] + 15
        d = case["deg"]
        # filter, H W, one read of W and H W for the Gram pair, W in and out of the block product, density
        b = size * n * ((3 * d - 1) * k + d + 2 * k + 2 * k + 2 * k + case["nev"]) + 8.0 * n * 16
        f = (d + 1.0) * n * k * _hx_flops(8) + 4.0 * n * k * k
        return {"bytes": b, "flops": f}
    dims = {"in": (case["nx"], case["ny"], case["nz"])}
    macs, b = 0.0, 8.0 * 2 * n
    for l in learned.LAYERS:
        src = dims[l.src]
        out = dims[l.skip] if l.up else (tuple((v + 1) // 2 for v in src) if l.stride == 2 else src)
        dims[l.name] = out
        nv = float(np.prod(out))
        macs += nv * l.ksize ** 3 * (l.ca + l.cs) * l.cout
        b += 2.0 * (nv * l.cout + float(np.prod(src)) * l.ca + (nv * l.cs if l.skip else 0))
    if kind == "net_fwd":
        return {"bytes": b + 32.0 * n, "flops": 2 * macs}
    # backward: activations again, FP32 gradients written and read once
    return {"bytes": 4 * b + 64.0 * n, "flops": 6 * macs}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _lap(x, dims, h, order):
    """A x for a (k, n) block, zero outside the cube."""
    nx, ny, nz = dims
    v = x.reshape(-1, nz, ny, nx)
    c = FD[order]
    y = v * (3 * c[0])
    for d in range(1, len(c)):
        for ax in (1, 2, 3):
            m = v.shape[ax]
            if m > d:
                y.narrow(ax, d, m - d).add_(v.narrow(ax, 0, m - d), alpha=c[d])
                y.narrow(ax, 0, m - d).add_(v.narrow(ax, d, m - d), alpha=c[d])
    return (y / (h * h)).reshape(x.shape)


class _ExactH:
    def __init__(self, st):
        case, ctx = st["case"], st["ctx"]
        self.case, self.pot = case, st["pot"]
        self.dims, self.h, self.order = (ctx.nx, ctx.ny, ctx.nz), ctx.h, case["order"]
        off, idx, u, w = ctx.projectors.tables()
        self.parts = [(torch.from_numpy(idx[a:b].astype(np.int64)).cuda(), torch.from_numpy(u[:, a:b].copy()).cuda(),
                       float(w[i])) for i, (a, b) in enumerate(zip(off[:-1], off[1:]))]
        self.keep = None
        if case["mask"]:
            g = [(torch.arange(d, dtype=torch.float64, device="cuda") - 0.5 * (d - 1)) * self.h for d in self.dims]
            r2 = (0.5 * self.h * (min(self.dims) - 1)) ** 2
            d2 = g[2][:, None, None] ** 2 + g[1][None, :, None] ** 2 + g[0][None, None, :] ** 2
            self.keep = (d2 <= r2).reshape(-1).double()

    def __call__(self, X):
        Y = _lap(X, self.dims, self.h, self.order).mul_(0.5)
        Y += self.pot * X
        for idx, u, w in self.parts:
            Y.index_add_(1, idx, ((X[:, idx] @ u.T) * w) @ u)
        return Y if self.keep is None else Y * self.keep


def _exact_filter(st):
    case = st["case"]
    H, X = _ExactH(st), st["X"].double()
    lam1, lo, hi = (float(v) for v in st["bounds"].cpu())
    e, c = (hi - lo) / 2, (hi + lo) / 2
    if case["mode"] == 0:
        s1 = e / (lam1 - c)
        s = s1
        Y = (H(X) - c * X) * (s1 / e)
        for _ in range(1, case["deg"]):
            sn = 1.0 / (2.0 / s1 - s)
            X, Y = Y, (H(Y) - c * Y) * (2 * sn / e) - X * (s * sn)
            s = sn
    else:
        Y = -(H(X) - c * X) / e
        for _ in range(1, case["deg"]):
            X, Y = Y, -(H(Y) - c * Y) * (2 / e) - X
    return Y


def _exact_pcg(st):
    case, ctx = st["case"], st["ctx"]
    dims, h, order = (ctx.nx, ctx.ny, ctx.nz), ctx.h, case["order"]

    def A(v):
        return _lap(v[None], dims, h, order)[0]

    if case["prec"]:
        S, lam = [], []
        c = FD[order]
        for m in dims:
            j = torch.arange(1, m + 1, dtype=torch.float64, device="cuda")
            S.append(torch.sin(j[:, None] * j[None, :] * (math.pi / (m + 1))) * math.sqrt(2.0 / (m + 1)))
            lam.append(sum((c[d] if d == 0 else 2 * c[d] * torch.cos(d * math.pi * j / (m + 1)))
                           for d in range(len(c))) / (h * h))
        den = lam[2][:, None, None] + lam[1][None, :, None] + lam[0][None, None, :]

        def both(v):
            return torch.einsum("zyx,xa,yb,zc->cba", v, S[0], S[1], S[2])

        def M(v):
            return both(both(v.reshape(dims[2], dims[1], dims[0])) / den).reshape(-1)
    x = st["x0"].clone()
    r = st["rhs"] - A(x)
    z = M(r) if case["prec"] else r
    p = z.clone()
    ro = torch.dot(z, r)
    tol1 = 1e-10 * ro
    its = 0
    while its < 200 and float(ro) > float(tol1):
        its += 1
        Ap = A(p)
        alpha = ro / torch.dot(p, Ap)
        x = x + alpha * p
        r = r - alpha * Ap
        z = M(r) if case["prec"] else r
        ro1 = torch.dot(z, r)
        # the plain solve's first direction aliases r (Eigensolvers/pcg.py): p = r + beta r
        p = z + (ro1 / ro) * (r if not case["prec"] and its == 1 else p)
        ro = ro1
    return {"x": x, "its": None}


def _exact_xc(rho, h3):
    g, b1, b2 = -0.2846, 1.0529, 0.3334
    c1, c2, c3, c4, c5 = 0.0622, 0.096, 0.004, 0.0232, 0.0192
    third = 1.0 / 3.0
    a0 = (4.0 / (9.0 * math.pi)) ** third
    rs = (0.75 / math.pi / rho) ** third
    vx = -2.0 / (math.pi * a0) / rs
    sq, al = torch.sqrt(rs), torch.log(rs)
    e1 = g / (1.0 + b1 * sq + b2 * rs)
    v1 = e1 ** 2 * (1.0 + 3.5 * b1 * sq * third + 4.0 * b2 * rs * third) / g
    e2 = c1 * al - c2 + (c3 * al - c4) * rs
    v2 = e2 - (c1 + (c3 * al - c5) * rs) * third
    ec, vc = torch.where(rs >= 1.0, e1, e2), torch.where(rs >= 1.0, v1, v2)
    exc = (0.75 * rho * vx + rho * ec).sum() * h3
    return vx + vc, torch.stack([exc, rho.max(), rho.min()])


def _exact_post(st):
    h3 = st["ctx"].h ** 3
    out, DX, DF, last = {}, [], [], None
    mix = 0.5
    for i in range(POST_ITERATIONS):
        rho, x1 = st["rho"][i], st["pot"][i]
        vxc, xc = _exact_xc(rho, h3)
        hsum = st["hpot"][i] + st["hpot0"]
        pot_new = st["ppot"] + 0.5 * vxc + hsum
        f1 = pot_new - x1
        sums = torch.stack([f1.dot(f1), pot_new.dot(pot_new), rho.dot(hsum), rho.dot(vxc)])
        m, fn = len(DX), float(f1.norm())
        if m == 0:
            new, used = x1 + mix * f1, 0
            DX, DF = [x1], [f1]
            last = fn
        elif m >= 2 and last < 0.1 * fn:
            new, used = DX[-1] + mix * DF[-1], 0
            DX, DF = [DX[-1]], [DF[-1]]
        else:
            dx, df = x1 - DX[-1], f1 - DF[-1]
            d, new, nv = dx + mix * df, x1 + mix * f1, -mix * dx
            for a, b in zip(DX[:-1], DF[:-1]):
                d = d - a * b.dot(df)
                new = new - a * b.dot(f1)
                nv = nv + b * a.dot(dx)
            M = nv.dot(df)
            new = new - d * (nv.dot(f1) / M)
            DX, DF = DX[:-1] + [d, x1], DF[:-1] + [nv / M, f1]
            used, last = m, fn
        out[f"xc{i}"], out[f"sums{i}"], out[f"mixed{i}"] = xc, sums, new
    out.update(vxc=vxc, pot_new=pot_new, f=f1, used=None)
    return out


def _exact_net(st):
    """FP64 convolutions and gradients between the network's own BF16
    roundings (weights, input and every stored activation)."""
    case, net = st["case"], st["net"]
    want = case["kind"] == "net_grad"
    bf = torch.bfloat16

    def stored(v):   # rounded to BF16, gradient passed through
        return v + (v.detach().to(torch.float32).to(bf).double() - v.detach())

    dims = {"in": (case["nz"], case["ny"], case["nx"])}
    s = net.scales
    x = torch.zeros(1, 8, *dims["in"], dtype=torch.float64, device="cuda")
    x[0, 0] = (s["a0"] * st["rho"]).float().to(bf).double().reshape(dims["in"])
    x[0, 1] = (s["a1"] * st["vloc"]).float().to(bf).double().reshape(dims["in"])
    w64 = net.w.to(bf).double()
    acts, params = {"in": x}, []
    with torch.set_grad_enabled(want):
        for l in learned.LAYERS:
            o, nw, ob, nb = net.offsets[l.name]
            w = w64[o:o + nw].clone().requires_grad_(want)
            b = net.w[ob:ob + nb].double().clone().requires_grad_(want)
            params += [w, b]
            ks = l.ksize
            wt = w.reshape(ks, ks, ks, l.ca + l.cs, l.cout).permute(4, 3, 0, 1, 2)
            a = acts[l.src]
            if l.up:
                sk = acts[l.skip]
                for ax in (2, 3, 4):
                    a = a.repeat_interleave(2, ax).narrow(ax, 0, sk.shape[ax])
                a = torch.cat([a, sk], 1)
            y = torch.nn.functional.conv3d(a, wt, b, stride=l.stride, padding=ks // 2)
            if l.act == 2:
                y = torch.where(y > 0, y, 0.0625 * y)
            acts[l.name] = y if l.name == "out" else stored(y)
        out = acts["out"][0].reshape(8, -1).T
        if not want:
            return out.contiguous()
        loss = ((out[:, 0] - st["target"].double()) ** 2).mean()
        g = torch.autograd.grad(loss, params)
    return {"out": out.detach().contiguous(), "loss": loss.detach().reshape(1),
            "grad": torch.cat([v.reshape(-1) for v in g])}


def exact(case, seed):
    kind = case["kind"]
    # step: chefsi1 draws its Lanczos start inside the call; setup: spline
    # tables and NumPy's summation order are the library's own
    if kind in ("step", "setup"):
        return None
    st = prepare(case, seed)
    if kind == "hx":
        return _ExactH(st)(st["X"].double())
    if kind == "filter":
        return _exact_filter(st)
    if kind == "hartree":
        return _exact_pcg(st)
    if kind == "post":
        return _exact_post(st)
    return _exact_net(st)
