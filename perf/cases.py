"""The engine's performance cases: the calls a user of the package makes.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges;
``prepare`` makes what a program has in hand before the call (an engine whose
chains are mid-run, host buffers), ``run`` is one call through the public
entry points with its outputs, ``work`` the bytes and flops the call cannot
do without and ``exact`` the outputs in 64 bits where they are a function of
the inputs alone (a Monte Carlo sweep has no such value).

Kinds of case
    run      the reference's run! through pimc.run: System, updates, Density
             and Energy measurements
    chain    Engine.run on one chain, then beads, permutation, observables
    io       a batch's beads from a pinned host buffer, sweeps, beads and
             energies back (Engine.run_io)
    batch    sweeps of a resident batch (Engine.run_batched), then its beads
    adjoint  Engine.adjoint: per-bead forces and parameter derivatives
    adjoints Engine.batch_adjoint over a batch
    table    contact_table: the tabulated contact propagator
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "pimc.jl_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)


def listed():
    return [
        # the first thing every user runs: 10 trapped ideal bosons, the
        # reference's own small test system, ten sweeps with density and energy
        dict(name="run_ideal_n10", kind="run", N=10, M=20, beta=1.0, L=5.0, ell=8, nbins=64,
             sweeps=10),
        # a periodic free gas under the physical rules, measured every sweep
        dict(name="chain_free_n64", kind="chain", N=64, M=32, beta=2.0, L=10.0, ell=16, omega=0.0,
             V0=0.0, g=-1.0, sigma=0.5, r_a=0.0, physical=True, nbins=0, contact=False, hard=0.0,
             beams=False, sweeps=4),
        # the interacting trap with a 128 x 128 density, the reference's rules
        dict(name="chain_pair_n256", kind="chain", N=256, M=64, beta=2.0, L=8.0, ell=16, omega=1.0,
             V0=0.0, g=1.0, sigma=0.5, r_a=1.5, physical=False, nbins=128, contact=False, hard=0.0,
             beams=False, sweeps=2),
        # hard spheres with the contact propagator in a quasicrystal lattice
        # (odd sizes; every move is decided from exact pair sums)
        dict(name="chain_contact_n33", kind="chain", N=33, M=40, beta=1.0, L=6.0, ell=13, omega=1.0,
             V0=0.0, g=0.0, sigma=0.5, r_a=1.5, physical=False, nbins=0, contact=True, hard=0.0432,
             beams=True, sweeps=1),
        # the largest single chain: lattice, trap and pair, physical rules
        dict(name="chain_lattice_n1024", kind="chain", N=1024, M=64, beta=4.0, L=16.0, ell=16,
             omega=0.1, V0=4.0, g=1.0, sigma=0.3, r_a=0.9, physical=True, nbins=0, contact=False,
             hard=0.0, beams=False, sweeps=1),
        # many replicas of small chains on the default launch shape, the way
        # errors are estimated without an autocorrelation model
        dict(name="batch_replicas_768", kind="batch", chains=768, Nlo=8, Nhi=48, Mlo=16, Mhi=32,
             physical=False, contact=False, split=False, measure_every=1, sweeps=4),
        # the headline batch: 4096 uneven chains end to end through host
        # buffers, the launch shape the tuner keeps for it
        dict(name="io_4096", kind="io", chains=4096, Nlo=8, Nhi=512, Mlo=16, Mhi=128,
             physical=False, contact=False, split=True, measure_every=10, sweeps=1),
        # the same list's first chains under the physical rules (pair action in
        # every move)
        dict(name="io_physical_512", kind="io", chains=512, Nlo=8, Nhi=512, Mlo=16, Mhi=128,
             physical=True, contact=False, split=True, measure_every=10, sweeps=1),
        # contact-propagator chains sharing one table (one temperature, M = 64)
        dict(name="batch_contact_256", kind="batch", chains=256, Nlo=8, Nhi=512, Mlo=64, Mhi=64,
             physical=False, contact=True, split=False, measure_every=10, sweeps=1),
        # forces and parameter derivatives of the differentiated configuration
        dict(name="adjoint_n1024", kind="adjoint", N=1024, M=64, beta=4.0, L=16.0, omega=0.1, V0=4.0,
             g=1.0, sigma=0.3, r_a=0.9),
        # gradients of a parameter scan, with every bead's force
        dict(name="adjoints_60", kind="adjoints", chains=60, Nlo=8, Nhi=512, Mlo=16, Mhi=128),
        # the contact propagator of a new temperature: the reference's 600 x 600
        # grid
        dict(name="table_600", kind="table", n=600, g0=1.16, tau=1.0 / 32, range=12.0),
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "chain", "chain", "chain", "batch", "io", "io", "adjoint", "adjoints",
                       "table"])
    if kind == "run":
        N, M = _loguni(rng, 2, 64), rng.randint(8, 40)
        return dict(kind=kind, N=N, M=M, beta=round(rng.uniform(0.5, 3.0), 3), L=5.0,
                    ell=rng.randint(2, min(16, M - 2)), nbins=rng.choice([17, 64, 100]),
                    sweeps=rng.randint(1, 20))
    if kind == "chain":
        pair = rng.random() < 0.7
        contact = pair and rng.random() < 0.25
        physical = rng.random() < 0.5
        N = _loguni(rng, 2, 100 if contact else 1000)
        M = rng.randint(9, 64)
        return dict(kind=kind, N=N, M=M, beta=round(rng.uniform(0.5, 4.0), 3),
                    L=round(rng.uniform(7.0, 12.0), 2), ell=rng.randint(3, min(20, M - 2)),
                    omega=rng.choice([0.0, 0.3, 1.0]), V0=rng.choice([0.0, 2.5]),
                    g=round(rng.uniform(0.0, 2.0), 3) if pair and not contact else (0.0 if contact else -1.0),
                    sigma=0.5, r_a=1.5 if pair else 0.0, physical=physical,
                    nbins=rng.choice([0, 33, 128]), contact=contact,
                    hard=0.02 if contact and rng.random() < 0.5 and N < 50 else 0.0,
                    beams=rng.random() < 0.2, sweeps=rng.randint(1, 2))
    if kind in ("batch", "io"):
        Nhi = _loguni(rng, 16, 512)
        physical = rng.random() < 0.4
        contact = kind == "batch" and rng.random() < 0.3
        M = rng.choice([16, 24, 64, 100])
        most = 256 if physical or contact else 2000
        return dict(kind=kind, chains=_loguni(rng, 8, most), Nlo=min(8, Nhi), Nhi=Nhi,
                    Mlo=M if contact else 16, Mhi=M if contact else rng.choice([16, 64, 128]),
                    physical=physical, contact=contact, split=kind == "io",
                    measure_every=rng.choice([1, 4, 10]), sweeps=1)
    if kind == "adjoint":
        N = _loguni(rng, 4, 1024)
        return dict(kind=kind, N=N, M=rng.randint(8, 64), beta=round(rng.uniform(0.5, 4.0), 3),
                    L=round(rng.uniform(6.0, 16.0), 2), omega=rng.choice([0.1, 1.0]),
                    V0=rng.choice([0.0, 4.0]), g=round(rng.uniform(0.1, 2.0), 3), sigma=0.4, r_a=1.2)
    if kind == "adjoints":
        return dict(kind=kind, chains=rng.randint(2, 60), Nlo=4, Nhi=_loguni(rng, 16, 512), Mlo=9,
                    Mhi=rng.choice([16, 50, 128]))
    return dict(kind=kind, n=_loguni(rng, 40, 600), g0=rng.choice([0.5, 1.16, 2.0, 20.0]),
                tau=1.0 / rng.choice([16, 32, 40, 100]), range=round(rng.uniform(5.0, 13.0), 2))


# --------------------------------------------------------------------- inputs
def _paths(gen, N, M, beta, omega, L, spread):
    """[2][N][M] closed paths with the thermal fluctuations of the primitive
    action in the trap (free about a uniform or Gaussian centre without one),
    the centres widened by `spread`; wrapped into the box.  On the GPU."""
    tau = beta / M
    dev = gen.device
    k = torch.arange(M, device=dev, dtype=torch.float64)
    om = max(omega, 0.5)
    prec = 4.0 * torch.sin(math.pi * k / M) ** 2 / tau + tau * om * om
    z = torch.randn((2, N, M), generator=gen, device=dev, dtype=torch.float64)
    x = torch.fft.ifft(torch.fft.fft(z) / torch.sqrt(prec)).real
    c = torch.randn((2, N, 1), generator=gen, device=dev, dtype=torch.float64) * spread
    if omega == 0.0:
        c = (torch.rand((2, N, 1), generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * L
    x = x + c
    return (x + L) % (2 * L) - L


def _gen(seed):
    g = torch.Generator(device="cuda" if torch.cuda.is_available() else "cpu")
    g.manual_seed(int(seed))
    return g


def _mix(N, M, ell, L, measure_every):
    from pimc.engine import Mix
    return Mix(stage_slices=ell, stage_min=2, stage_max=ell, stage_minacc=0.0, stage_maxacc=1.0,
               swaps_per_sweep=N if N > 1 else 0, swap_slices=ell, swap_min=2, swap_max=ell,
               swap_minacc=0.0, swap_maxacc=1.0, com_phases=1, com_step=1.0, com_minstep=0.1,
               com_maxstep=L / 2, adapt=1, measure_every=measure_every)


def _chain_params(case, seed):
    from pimc.engine import ChainParams
    pair = case["g"] >= 0.0 or case["contact"]
    return ChainParams(dim=2, N=case["N"], M=case["M"], L=case["L"], T=1.0 / case["beta"], lam=0.5,
                       harmonic_omega=case["omega"], lattice_V0=case["V0"], lattice_a=1.0,
                       interactions=pair, pair_g=max(case["g"], 0.0), pair_sigma=case["sigma"],
                       r_a=case["r_a"], hardcore_a=case["hard"], semantics=int(case["physical"]),
                       density_nbins=case["nbins"], seed=1000003 * (seed + 1))


def _batch_shapes(case, seed=None):
    """(N, M, beta, g) of a batch's chains.  A case's chains are the same list
    for every seed: what a program repeats is the batch, with other beads."""
    rng = np.random.default_rng(4096)
    n = case["chains"]
    Ms = [m for m in (9, 16, 24, 32, 64, 100, 128) if case["Mlo"] <= m <= case["Mhi"]]
    if case["Mlo"] == 16 and case["Mhi"] == 128:
        Ms = [16, 32, 64, 128]
    N = rng.integers(case["Nlo"], case["Nhi"] + 1, size=n)
    M = rng.choice(Ms, size=n)
    beta = rng.uniform(0.5, 4.0, size=n)
    g = rng.uniform(0.0, 2.0, size=n)
    if case.get("contact"):
        beta[:] = 2.0 * M[0] / 64
    return [(int(N[i]), int(M[i]), float(beta[i]), float(g[i])) for i in range(n)]


def _batch(case, seed):
    """engine of a batch, the mixes set, and its beads in host layout"""
    from pimc.engine import ChainParams, Engine
    shapes = _batch_shapes(case)
    ps = [ChainParams(dim=2, N=N, M=M, L=8.0, T=1.0 / b, lam=0.5, harmonic_omega=1.0,
                      interactions=True, pair_g=g, pair_sigma=0.5, r_a=1.5,
                      semantics=int(case.get("physical", False)), seed=1000003 * (seed + 1) + i)
          for i, (N, M, b, g) in enumerate(shapes)]
    eng = Engine(ps)
    gen = _gen(seed)
    flat = torch.empty(eng.beads_all_size(), dtype=torch.float64, device=gen.device)
    at = 0
    for N, M, b, g in shapes:
        # the repulsive cloud is wider than the ideal one
        x = _paths(gen, N, M, b, 1.0, 8.0, 0.5 + 0.2 * (g * N / 30.0) ** 0.25)
        flat[at:at + x.numel()] = x.reshape(-1)
        at += x.numel()
    return eng, ps, flat


def prepare(case, seed):
    import pimc
    from pimc.engine import Engine
    pimc.load()
    kind = case["kind"]
    st = {"case": case}
    if kind == "run":
        N, M = case["N"], case["M"]
        s = pimc.System(pimc.Harmonic(1.0), M=M, N=N, L=case["L"], T=1.0 / case["beta"], λ=0.5,
                        length_measurement_cycle=1, seed=1000003 * (seed + 1))
        s.set_world(_paths(_gen(seed), N, M, case["beta"], 1.0, case["L"], 0.3).cpu().numpy())
        k = -(-M // case["ell"])
        frozen = dict(minacc=0.0, maxacc=1.0)
        st["s"] = s
        st["updates"] = [(1, pimc.ReshapeLinear(s, case["ell"], **frozen)),
                         (k, pimc.ReshapeSwapLinear(s, case["ell"], **frozen)),
                         (k, pimc.SingleCenterOfMass(s, 1.0))]
        st["n"] = N * (k + 2) * case["sweeps"]
        pimc.run(s, st["n"], st["updates"], Zmeasurements=[pimc.Density(s, case["nbins"]),
                                                           pimc.Energy(s, 1000)])
    elif kind in ("chain", "adjoint"):
        c = dict(case)
        if kind == "adjoint":
            c.update(physical=True, nbins=0, contact=False, hard=0.0, beams=False)
        e = Engine(_chain_params(c, seed))
        if c["contact"]:
            e.set_contact_propagator(2.0, 12.0)
        if c["beams"]:
            e.set_beams(pimc.lattice_angles("l25"), 0.6, -3.0)
        if c["hard"] == 0.0:  # hard spheres keep init_world's placement
            e.set_beads(_paths(_gen(seed), c["N"], c["M"], c["beta"], c["omega"], c["L"],
                               0.5 + 0.08 * math.sqrt(c["N"])).cpu().numpy())
        if kind == "adjoint":
            e.set_next(np.random.default_rng(seed).permutation(c["N"]))
            st["x"], st["next"] = e.get_beads(), e.get_next()
        else:
            e.set_mix(_mix(c["N"], c["M"], c["ell"], c["L"], 1))
            e.run(1)
        st["e"] = e
    elif kind in ("io", "batch", "adjoints"):
        eng, ps, flat = _batch(case, seed)
        if kind == "adjoints":
            eng.set_beads_all(flat.cpu().numpy())
            st["e"] = eng
            return st
        for i, p in enumerate(ps):
            eng.set_mix(_mix(p.N, p.M, min(16, p.M // 2), 8.0, case["measure_every"]), chain=i)
        if case["contact"]:
            eng.set_contact_propagator(1.16, 12.0)
        if case["split"]:
            # what the tuner keeps for such a batch: a launch per phase, row scans
            eng.set_launch(block=64, sweeps_per_launch=1, state_smem_bytes=0, split_phases=1,
                           phase_block=(128, 64, 256 if case["physical"] else 128), cell_lists=1)
        buf = torch.empty(flat.numel(), dtype=torch.float64, pin_memory=torch.cuda.is_available())
        buf.copy_(flat)
        st["buf"], st["x"], st["e"] = buf, buf.numpy(), eng
        if kind == "io":
            eng.run_io(st["x"], 2)
        else:
            eng.set_beads_all(st["x"])
            eng.run_batched(2)
    else:
        st["seed"] = seed
        # another coupling a seed, the same work
        st["g0"] = case["g0"] * (1.0 + 0.001 * (seed % 97))
    return st


def run(st):
    import pimc
    from pimc.engine import contact_table
    case = st["case"]
    kind = case["kind"]
    if kind == "run":
        s = st["s"]
        dens, en = pimc.Density(s, case["nbins"]), pimc.Energy(s, 1000)
        pimc.run(s, st["n"], st["updates"], Zmeasurements=[dens, en])
        return {"density": dens.dens, "energy": np.array(en.energy[s.N]),
                "virial": np.array(en.energy_virial[s.N]), "x": s.engine.get_beads(),
                "next": s.engine.get_next()}
    e = st["e"] if "e" in st else None
    if kind == "chain":
        e.run(case["sweeps"])
        out = {"x": e.get_beads(), "next": e.get_next(), "sums": e.observable_sums()[0]}
        if case["nbins"]:
            out["density"] = e.density()[0]
        return out
    if kind == "io":
        x = e.run_io(st["x"], case["sweeps"])
        s, _, cnt = e.energy_sums_all()
        return {"x": x, "energy": s, "count": cnt.astype(np.int64)}
    if kind == "batch":
        e.run_batched(case["sweeps"])
        s, _, cnt = e.energy_sums_all()
        return {"x": e.get_beads_all(st["x"]), "energy": s, "count": cnt.astype(np.int64)}
    if kind == "adjoint":
        g, th, ex = e.adjoint()
        return {"force": g, "theta": th, "extra": ex}
    if kind == "adjoints":
        g, th, ex = e.batch_adjoint(want_beads=True)
        return {"force": g, "theta": th, "extra": ex}
    return {"table": contact_table(st["g0"], case["tau"], case["range"], case["n"])}


# --------------------------------------------------------------------- work
def _sweep_work(N, M, ell, pair, physical, measured, sweeps):
    """bytes and flops of sweeps of one chain: the beads and the permutation
    in and out once; per proposed bead a bridge point, its potential and its
    share of the decision (about 30 flops), a swap's weights over every
    partner (8), and with a pair action the terms with the partners in reach
    (a quarter of the slice, 15 flops, old and new) where the rules ask for
    them; a measurement visits every pair in reach once"""
    k = -(-M // ell)
    half = max(1.0, 0.5 * ell)
    staged, swapped = N * k * half, 2.0 * N * half
    f = 30.0 * (staged + swapped) + 8.0 * N * N
    if pair:
        f += 2 * 15.0 * 0.25 * N * (swapped + (staged if physical else 0.0))
    if measured:
        f += 30.0 * N * M + (20.0 * 0.125 * N * N * M if pair else 0.0)
    return 2.0 * (16.0 * N * M + 4.0 * N), f * sweeps


def work(case):
    kind = case["kind"]
    if kind == "run":
        b, f = _sweep_work(case["N"], case["M"], case["ell"], False, False, True, case["sweeps"])
        return {"bytes": b + 8.0 * case["nbins"] ** 2, "flops": f}
    if kind == "chain":
        b, f = _sweep_work(case["N"], case["M"], case["ell"], case["g"] >= 0.0, case["physical"], True,
                           case["sweeps"])
        return {"bytes": b + 8.0 * case["nbins"] ** 2, "flops": f}
    if kind in ("io", "batch"):
        b = f = 0.0
        for N, M, _, _ in _batch_shapes(case):
            bi, fi = _sweep_work(N, M, min(16, M // 2), True, case["physical"],
                                 case["measure_every"] == 1, case["sweeps"])
            b += bi
            f += fi
        return {"bytes": b, "flops": f}
    if kind == "table":
        # two Bessel functions (about 40 flops each) per radius and node, four
        # products per entry of the triangle and node
        nodes = 8.0 * (33 + math.sqrt(41.5 / case["tau"]) * 4 * case["range"] / math.pi)
        return {"bytes": 8.0 * case["n"] ** 2,
                "flops": nodes * (80.0 * case["n"] + 4.0 * case["n"] ** 2)}
    shapes = [(case["N"], case["M"])] if kind == "adjoint" else [s[:2] for s in _batch_shapes(case)]
    b = sum(32.0 * N * M for N, M in shapes)
    return {"bytes": b, "flops": sum(30.0 * N * M + 30.0 * 0.125 * N * N * M for N, M in shapes)}


# --------------------------------------------------------------------- exact
def _exact_adjoint(x, nxt, beta, L, omega, V0, g, sigma, r_a):
    """the potential action's gradient and its parameter derivatives, S = tau
    sum V + tau/2 sum over links and pairs within reach at the link's start of
    v(r) at both ends; x [2][N][M] on a device, in FP64"""
    N, M = x.shape[1], x.shape[2]
    tau = beta / M
    rc2 = (2 * L / math.floor(2 * L / r_a)) ** 2
    c = 1.0 / (2 * sigma * sigma)
    h = 0.5 * tau
    pi = math.pi
    grad = tau * (omega ** 2 * x + V0 * pi * torch.sin(2 * pi * x))
    sin2 = (torch.sin(pi * x) ** 2).sum()
    r2 = (x * x).sum()
    s_ext = tau * (0.5 * omega ** 2 * r2 + V0 * sin2)
    r_ge = (x * grad).sum()
    s_pair = torch.zeros((), dtype=x.dtype, device=x.device)
    vir = torch.zeros_like(s_pair)
    iu = torch.ones((N, N), dtype=torch.bool, device=x.device).triu(1)
    step = max(1, (1 << 24) // max(N * N, 1))
    idx = torch.arange(N, device=x.device)

    def rel(p):
        d = p[:, :, None, :] - p[:, None, :, :]  # [2][N][N][s]
        return d - 2 * L * torch.round(d / (2 * L))

    for j0 in range(0, M, step):
        j = torch.arange(j0, min(j0 + step, M), device=x.device)
        cur = x[:, :, j]
        nx = torch.empty_like(cur)
        rows = torch.empty((len(j), N), dtype=torch.long, device=x.device)
        jn = (j + 1) % M
        for q in range(len(j)):
            rows[q] = nxt if int(j[q]) == M - 1 else idx
            nx[:, :, q] = x[:, rows[q], int(jn[q])]
        d1, d2 = rel(cur), rel(nx)
        r1, r2b = (d1 * d1).sum(0), (d2 * d2).sum(0)
        on = ((r1 <= rc2) & ~torch.eye(N, dtype=torch.bool, device=x.device)[:, :, None]).to(x.dtype)
        v1, v2 = on * g * torch.exp(-r1 * c), on * g * torch.exp(-r2b * c)
        up = iu[:, :, None].to(x.dtype)
        s_pair = s_pair + h * ((v1 + v2) * up).sum()
        vir = vir - 2 * c * h * ((r1 * v1 + r2b * v2) * up).sum()
        g1 = (-2 * c * h) * (v1 * d1).sum(2)
        g2 = (-2 * c * h) * (v2 * d2).sum(2)
        for q in range(len(j)):
            grad[:, :, int(j[q])] += g1[:, :, q]
            grad[:, rows[q], int(jn[q])] += g2[:, :, q]
    theta = torch.stack([tau * sin2 if V0 else torch.zeros_like(s_pair), tau * omega * r2, s_pair / g])
    extra = torch.stack([s_ext, s_pair, (s_ext + 0.5 * r_ge + s_pair + 0.5 * vir) / beta,
                         (x * grad).sum()])
    return grad, theta, extra


def _bessel0(x):
    """J0 and Y0 in FP64: the power series below 2, backward recurrence with
    Neumann's series for Y0 up to 25, Hankel's expansion beyond"""
    gamma = 0.5772156649015329
    lo, hi = x < 2.0, x > 25.0
    # power series
    xs = torch.where(lo, x, torch.ones_like(x))
    q = 0.25 * xs * xs
    term, J, S, hk = torch.ones_like(x), torch.ones_like(x), torch.zeros_like(x), 0.0
    for k in range(1, 20):
        term = term * (-q) / (k * k)
        hk += 1.0 / k
        J, S = J + term, S - hk * term
    Y = (2 / math.pi) * ((torch.log(0.5 * xs) + gamma) * J + S)
    # backward recurrence, normalised by J0 + 2 sum J_2k = 1
    xm = torch.where(lo | hi, torch.full_like(x, 10.0), x)
    a, b = torch.zeros_like(x), torch.full_like(x, 1e-150)  # J_(n+1), J_n up to the norm
    norm, neum = torch.zeros_like(x), torch.zeros_like(x)
    for n in range(90, 0, -1):
        if n % 2 == 0:
            norm = norm + 2 * b
            neum = neum + (b if (n // 2) % 2 == 0 else -b) / (n // 2)
        a, b = b, (2.0 * n / xm) * b - a
    norm = norm + b
    Jm = b / norm
    Ym = (2 / math.pi) * (torch.log(0.5 * xm) + gamma) * Jm - (4 / math.pi) * neum / norm
    # Hankel
    xh = torch.where(hi, x, torch.full_like(x, 30.0))
    P, Q, t = torch.ones_like(x), torch.zeros_like(x), torch.ones_like(x)
    for k in range(1, 24):
        t = t * (-((2 * k - 1) ** 2)) / (8.0 * k * xh)
        if k % 2:
            Q = Q + (t if k % 4 == 1 else -t)
        else:
            P = P + (t if k % 4 == 0 else -t)
    c, s = torch.cos(xh), torch.sin(xh)
    amp = torch.sqrt(1.0 / (math.pi * xh))
    # cos(x - pi/4) = (c + s)/sqrt 2, sin(x - pi/4) = (s - c)/sqrt 2
    Jh, Yh = amp * (P * (c + s) - Q * (s - c)), amp * (P * (s - c) + Q * (c + s))
    return (torch.where(lo, J, torch.where(hi, Jh, Jm)), torch.where(lo, Y, torch.where(hi, Yh, Ym)))


def _exact_table(n, g0, tau, rng_, dev):
    """the Bessel integrals on the radii 1e-20 .. range as products of the
    node values: Gauss-Legendre panels half as long as the engine's"""
    r = 1e-20 + torch.arange(n, device=dev, dtype=torch.float64) * ((rng_ - 1e-20) / (n - 1))
    gx, gw = np.polynomial.legendre.leggauss(12)
    edges = [1e-10 * 2.0 ** p for p in range(33) if 1e-10 * 2.0 ** p < 0.5] + [0.5]
    K = math.sqrt(44.0 / tau)
    nu = int(math.ceil((K - 0.5) / (math.pi / rng_ / 8)))
    edges += [0.5 + (K - 0.5) * (i + 1) / nu for i in range(nu)]
    e = np.array(edges)
    a, b = e[:-1, None], e[1:, None]
    k = torch.from_numpy((0.5 * (a + b) + 0.5 * (b - a) * gx).reshape(-1)).to(dev)
    w = torch.from_numpy((0.5 * (b - a) * gw * np.ones_like(a)).reshape(-1)).to(dev)
    s = (2 / math.pi) * (0.5772156649015329 + torch.log(0.5 * k)) - 4.0 / g0
    base = w * k * torch.exp(-tau * k * k) / (1 + s * s) / (2 * math.pi)
    J, Y = _bessel0(r[:, None] * k)
    return (Y * base) @ Y.T - (J * base) @ J.T - (J * (base * s)) @ Y.T - (Y * (base * s)) @ J.T


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "table":
        t = _exact_table(case["n"], case["g0"] * (1.0 + 0.001 * (seed % 97)), case["tau"],
                         case["range"], dev)
        return {"table": t.cpu().numpy()}
    if kind == "adjoint":
        x = _paths(_gen(seed), case["N"], case["M"], case["beta"], case["omega"], case["L"],
                   0.5 + 0.08 * math.sqrt(case["N"]))
        nxt = torch.from_numpy(np.random.default_rng(seed).permutation(case["N"])).to(x.device)
        f, th, ex = _exact_adjoint(x, nxt, case["beta"], case["L"], case["omega"], case["V0"],
                                   case["g"], case["sigma"], case["r_a"])
        return {"force": f.cpu().numpy(), "theta": th.cpu().numpy(), "extra": ex.cpu().numpy()}
    if kind == "adjoints":
        gen = _gen(seed)
        out = {"force": [], "theta": [], "extra": []}
        for N, M, b, g in _batch_shapes(case):
            x = _paths(gen, N, M, b, 1.0, 8.0, 0.5 + 0.2 * (g * N / 30.0) ** 0.25)
            f, th, ex = _exact_adjoint(x, torch.arange(N, device=x.device), b, 8.0, 1.0, 0.0, g, 0.5, 1.5)
            out["force"].append(f.cpu().numpy())
            out["theta"].append(th.cpu().numpy())
            out["extra"].append(ex.cpu().numpy())
        out["theta"], out["extra"] = np.array(out["theta"]), np.array(out["extra"])
        return out
    return None
