"""The fast kernels at the sizes where they can go wrong: tile and warp edges,
remainders, the smallest and the largest of their ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 65])
def test_contact_table_tile_edges(n, engine_lib):
    """table sizes around the product's 32 x 32 tiles against adaptive
    quadrature, with the golden test's tolerance"""
    pytest.importorskip("scipy")
    from oracle import contact_table as CT
    from pimc.engine import contact_table
    g0, tau, rng_ = 2.0, 1.0 / 16, 4.0
    tab = contact_table(g0, tau, rng_, n)
    np.testing.assert_array_equal(tab, tab.T)
    r = CT.grid(rng_, n)
    big = np.abs(tab).max()
    idx = sorted({0, 1, n // 2, max(n - 2, 0), n - 1})
    for i in idx:
        for j in idx:
            if i <= j:
                v = CT.entry(float(r[i]), float(r[j]), g0, tau)
                assert abs(tab[i, j] - v) <= 1e-10 * abs(v) + 1e-13 * big, (i, j, tab[i, j], v)


def test_contact_table_in_several_ranges_of_nodes(engine_lib):
    """a table whose node rows outgrow the scratch (38 k nodes x 608 radii) has
    the entries of a small table of the same quadrature: the 601 grid's every
    200th radius.  Both sum the same terms, |terms| within a few times the
    largest entry, in another order: 38 k rounding errors of 1.1e-16 stay
    below 1e-11 of it"""
    from pimc.engine import contact_table
    big = contact_table(2.0, 1.0 / 2000, 13.0, 601)
    small = contact_table(2.0, 1.0 / 2000, 13.0, 4)
    np.testing.assert_allclose(big[::200, ::200], small, rtol=0, atol=1e-11 * np.abs(small).max())


def _adjoint_reference(x, nxt, T, L, omega, V0, g, sigma, r_a, pair):
    """dS/dr and dS/d(V0, omega, g) of the potential action in FP64 numpy"""
    dim, N, M = x.shape
    tau, h, c = 1.0 / (T * M), 0.5 / (T * M), 0.5 / sigma ** 2
    grad = tau * (omega ** 2 * x + V0 * np.pi * np.sin(2 * np.pi * x))
    th = np.array([tau * np.sum(np.sin(np.pi * x) ** 2) if V0 else 0.0, tau * omega * np.sum(x * x), 0.0])
    if pair:
        rc = 2 * L / np.floor(2 * L / r_a)
        for j in range(M):
            jn, own = (j + 1) % M, nxt if j == M - 1 else np.arange(N)
            for a, rows in ((x[:, :, j], None), (x[:, own, jn], own)):
                d = a[:, :, None] - a[:, None, :]
                d -= 2 * L * np.round(d / (2 * L))
                first = x[:, :, j][:, :, None] - x[:, :, j][:, None, :]
                first -= 2 * L * np.round(first / (2 * L))
                on = (np.sum(first ** 2, 0) <= rc * rc) & ~np.eye(N, dtype=bool)
                e = on * np.exp(-c * np.sum(d * d, 0))
                th[2] += 0.5 * h * e.sum()
                f = (-2 * c * h * g) * np.sum(e * d, axis=2)
                if rows is None:
                    grad[:, :, j] += f
                else:
                    np.add.at(grad, (slice(None), rows, jn), f)
    return grad, th


@pytest.mark.parametrize("N,M,dim,pair", [(1, 4, 2, True), (2, 5, 2, True), (7, 9, 1, True), (8, 6, 2, False),
                                          (9, 33, 2, True), (31, 8, 2, True), (32, 8, 1, True),
                                          (33, 40, 2, True), (200, 65, 2, True), (300, 70, 1, True)])
def test_adjoint_gather_edges(N, M, dim, pair, engine_lib):
    """the adjoint around its blocks of particles and rings of 32 pairs, crowded
    and sparse, alone (a warp per particles of a slice) and in a batch of at
    least 700 slices (a CTA per slice), against FP64 numpy.  A force sums at most 2 N terms no larger than the largest force's
    scale, each with a few rounding errors: 1e-12 of that scale"""
    from pimc.engine import ChainParams, Engine
    rng = np.random.default_rng(N * 100 + M)
    kw = dict(dim=dim, N=N, M=M, L=4.0, T=0.5, lam=0.5, harmonic_omega=0.7, lattice_V0=1.5,
              lattice_a=1.0, interactions=pair, pair_g=1.3, pair_sigma=0.5, r_a=1.2, semantics=1)
    for spread in (0.4, 2.0):
        x = np.clip(rng.normal(scale=spread, size=(dim, N, M)), -3.99, 3.99)
        nxt = rng.permutation(N).astype(np.int32)
        e = Engine([ChainParams(**kw)] + [ChainParams(**dict(kw, N=3)) for _ in range(700 // M + 1)])
        e.set_beads(x)
        e.set_next(nxt)
        want, th_want = _adjoint_reference(x, nxt, 0.5, 4.0, 0.7, 1.5, 1.3, 0.5, 1.2, pair)
        scale = np.abs(want).max()
        g, th, _ = e.adjoint(0)
        gb, thb, _ = e.batch_adjoint(want_beads=True)
        for got, t in ((g, th), (gb[0], thb[0])):
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * scale)
            np.testing.assert_allclose(t, th_want, rtol=1e-12, atol=1e-13)
        e.close()


def test_batch_adjoint_follows_a_new_trap(engine_lib):
    """dS/domega after set_potential uses the new frequency"""
    from pimc.engine import ChainParams, Engine
    e = Engine([ChainParams(dim=2, N=5, M=8, L=4.0, T=1.0, lam=0.5, harmonic_omega=1.0, seed=i) for i in range(2)])
    e.batch_adjoint()
    e.set_potential(0.0, 0.5, 0.0, chain=1)
    _, th, _ = e.batch_adjoint()
    _, one, _ = e.adjoint(1)
    np.testing.assert_allclose(th[1], one, rtol=1e-13)


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("ell,M", [(5, 9), (17, 40), (18, 36), (31, 40), (32, 40), (33, 70), (64, 70)])
def test_sweep_paths_decide_as_exact_sums(sem, ell, M, engine_lib):
    """sweeps around the windows' edges (half-warp and warp bridges, the longest
    swap of a warp, the longest window), crowded and sparse, one and two
    dimensions: bracketed decisions give the beads, permutations and
    acceptance counts of exact FP64 ones, bit for bit"""
    from pimc.engine import ChainParams, Engine, Mix, OPT_EXACT_DECISIONS
    ps = [ChainParams(dim=dim, N=N, M=M, L=L, T=1.0, lam=0.5, harmonic_omega=om, interactions=pair,
                      pair_g=g, pair_sigma=0.4, r_a=1.0, semantics=sem, seed=900 + i)
          for i, (N, dim, L, om, pair, g) in enumerate(
              [(2, 2, 4.0, 1.0, True, 1.5), (31, 2, 3.0, 1.0, True, 1.0), (32, 1, 6.0, 0.5, True, 2.0),
               (33, 2, 8.0, 0.0, True, 1.0), (70, 2, 3.0, 2.0, True, 0.7), (64, 2, 5.0, 1.0, False, 0.0),
               (20, 2, 3.0, 1.0, True, 0.0)])]
    out = []
    for exact in (0, 1):
        e = Engine(ps)
        for i, p in enumerate(ps):
            e.set_mix(Mix(stage_slices=ell, stage_min=2, stage_max=ell, stage_minacc=0.0, stage_maxacc=1.0,
                          swaps_per_sweep=p.N + 40, swap_slices=ell, swap_min=2, swap_max=ell,
                          swap_minacc=0.0, swap_maxacc=1.0, com_phases=1, com_step=0.5,
                          com_minstep=0.1, com_maxstep=2.0), chain=i)
        e.set_option(OPT_EXACT_DECISIONS, exact)
        e.run_batched(6)
        out.append([(e.get_beads(c), e.get_next(c), e.stats(c).accepts) for c in range(len(ps))])
        e.close()
    for (xa, na, aa), (xb, nb, ab) in zip(*out):
        np.testing.assert_array_equal(xa, xb)
        np.testing.assert_array_equal(na, nb)
        assert aa == ab and np.isfinite(xa).all()


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 6.0])
def test_contact_sweeps_decide_as_exact_sums(sem, scale, engine_lib):
    """contact chains, dense and sparse, with separations past a short table's
    end and (scale 6) pairs on the -mu branch: bracketed decisions give the beads
    and acceptance counts of exact FP64 ones, bit for bit"""
    from pimc.engine import ChainParams, Engine, Mix, OPT_EXACT_DECISIONS, contact_table
    M = 20
    tab = scale * contact_table(1.16, 1.0 / M, 3.0, 200)
    ps = [ChainParams(dim=dim, N=N, M=M, L=L, T=1.0, lam=0.5, mu=0.3, harmonic_omega=om, interactions=True,
                      r_a=1.0, semantics=sem, seed=40 + i)
          for i, (N, dim, L, om) in enumerate([(2, 2, 3.0, 2.0), (33, 2, 3.0, 1.5), (40, 1, 6.0, 1.0), (64, 2, 5.0, 1.0)])]
    out = []
    for exact in (0, 1):
        e = Engine(ps)
        e.set_contact_table(tab, 3.0)
        for i, p in enumerate(ps):
            e.set_mix(Mix(stage_slices=9, stage_max=9, stage_minacc=0.0, stage_maxacc=1.0, swaps_per_sweep=60,
                          swap_slices=9, swap_max=9, swap_minacc=0.0, swap_maxacc=1.0, com_maxstep=2.0), chain=i)
        e.set_option(OPT_EXACT_DECISIONS, exact)
        e.run_batched(8)
        out.append([(e.get_beads(c), e.get_next(c), e.stats(c).accepts) for c in range(len(ps))])
        e.close()
    for (xa, na, aa), (xb, nb, ab) in zip(*out):
        np.testing.assert_array_equal(xa, xb)
        np.testing.assert_array_equal(na, nb)
        assert aa == ab and np.isfinite(xa).all()


@pytest.mark.parametrize("N,M,dim", [(2, 4, 2), (31, 9, 2), (33, 20, 1), (200, 17, 2), (300, 24, 2)])
def test_measurement_launches_agree(N, M, dim, engine_lib):
    """a sweep's measurement in its own CTA, in launches of its own (a split
    sweep; a lone large chain) and by pimc_measure after the sweep: the same
    observables, density counts and pair histogram; the pair columns within the
    FP32 terms' 2e-7, the rest to rounding"""
    from pimc.engine import ChainParams, Engine, Mix
    kw = dict(dim=dim, N=N, M=M, L=5.0, T=0.5, lam=0.5, harmonic_omega=1.0, interactions=True, pair_g=1.0,
              pair_sigma=0.5, r_a=1.5, density_nbins=16, energy_capacity=4, seed=5)
    mix = Mix(stage_slices=3, stage_max=3, swaps_per_sweep=N, swap_slices=3, swap_max=3, com_maxstep=2.0,
              measure_every=2)
    out = []
    for shape in ("plain", "fused", "split"):
        e = Engine([ChainParams(**kw), ChainParams(**dict(kw, N=3, seed=6))], mix)
        e.set_radial(12)
        if shape == "plain":
            e.run_plain(4)
        else:
            e.set_launch(128, split_phases=int(shape == "split"))
            e.run_batched(4)
        out.append((e.observables(), e.density()[0], e.radial()[0], e.get_beads()))
        if shape == "split":
            e.reset_measurements()
            e.measure()
            exact = e.observables()[0]
        e.close()
    for o in out[1:]:
        np.testing.assert_array_equal(o[3], out[0][3])
        np.testing.assert_allclose(o[0], out[0][0], rtol=1e-12, atol=1e-12)
        np.testing.assert_array_equal(o[1], out[0][1])
        np.testing.assert_array_equal(o[2], out[0][2])
    last = out[2][0][-1]
    scale = np.maximum(np.abs(exact), 1.0)
    assert np.all(np.abs(last - exact)[[0, 1, 4, 5, 6]] <= 1e-10 * scale[[0, 1, 4, 5, 6]])
    assert np.all(np.abs(last - exact)[[2, 3]] <= 2e-7 * scale[[2, 3]])


@pytest.mark.parametrize("helical", [False, True])
@pytest.mark.parametrize("scale,K", [(0.5, 1), (0.6, 12), (3.0, 16), (1e15, 5)])
def test_beam_phases_around_the_table(scale, K, helical, engine_lib):
    """links of beads whose phases lie on, halfway between and beside the entries
    of the table of a turn, across many turns and beyond the table's range,
    against extended precision from the same rounded half turns z.  An entry,
    the polynomials and the turn by them are a few roundings of numbers below
    1, z two of its last places: I within 8 ulp + 4 pi |z| ulp"""
    from pimc.engine import ChainParams, Engine
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision")
    N, M, L = 16, 16, 4.0
    ang = np.linspace(0.0, 2.0, K) if K > 1 else np.array([0.0])
    k = np.arange(N * M)
    y = ((k % 9 - 4) / 512.0 + (k * 37 % 256 - 128) / 128.0) / (2.0 * scale) * (1.0 + (k % 5 - 2) * 2.0 ** -40)
    y[np.abs(y) > L * 0.99] *= 0.25
    x = np.zeros((2, N, M))
    x[1] = y.reshape(N, M)
    if K > 1:
        x[0] = np.random.default_rng(4).uniform(-3.9, 3.9, (N, M))
    e = Engine(ChainParams(dim=2, N=N, M=M, L=L, T=1.0, lam=0.5, semantics=1))
    e.set_beams(ang, scale, 1.0, helical)
    e.set_beads(x)
    got = np.asarray(e.get_links())  # -tau/2 (I_j + I_j+1)
    e.close()
    if scale > 1e6:  # the phases themselves carry no digits: finite and in range
        assert np.all(np.isfinite(got)) and np.all(got <= 0.0) and np.all(got >= -1.0 / M * (1 + 1e-12))
        return
    q = np.longdouble
    ph = [2 * q(scale) * (q(1) * x[0] * np.sin(q(a)) + q(1) * x[1] * np.cos(q(a))) for a in ang]
    off = [q(a) if helical else q(0) for a in ang]
    pi = q("3.14159265358979323846264338327950288")
    S = sum(np.sin(pi * np.fmod(z, 2) + o) for z, o in zip(ph, off)) / K
    Cc = sum(np.cos(pi * np.fmod(z, 2) + o) for z, o in zip(ph, off)) / K
    I = S * S + Cc * Cc
    want = np.asarray(-0.5 / M * (I + np.roll(I, -1, axis=1)), dtype=float)
    zmax = float(max(np.abs(z).max() for z in ph))
    np.testing.assert_allclose(got.reshape(want.shape), want, rtol=0, atol=(8 + 4 * np.pi * zmax) * 2.0 ** -52 / M)


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("N,L", [(257, 9.0), (513, 9.0), (1100, 16.0), (1300, 20.0)])
def test_long_chains_decide_as_exact_sums(N, L, sem, engine_lib):
    """lone chains, split sweeps with swaps in CTAs of 64 threads and warps at lengths
    where the kernels change over (staging in CTAs of 512 threads, the partner
    ratio's particles past the kept ones, swaps bracketed from the cell lists):
    bracketed decisions, with lists and with row scans, give the beads,
    permutations and acceptance counts of exact FP64 ones, bit for bit"""
    from pimc.engine import ChainParams, Engine, Mix, OPT_EXACT_DECISIONS
    p = ChainParams(dim=2, N=N, M=9, L=L, T=1.0, lam=0.5, harmonic_omega=0.3, interactions=True, pair_g=1.0,
                    pair_sigma=0.4, r_a=1.0, semantics=sem, seed=61)
    out = []
    for exact, mode, split in ((1, 0, 0), (0, 0, 0), (0, 2, 0), (0, 0, 1), (0, 2, 1), (0, 0, 2), (0, 2, 2)):
        e = Engine(p, Mix(stage_slices=4, stage_max=4, stage_minacc=0.0, stage_maxacc=1.0, swaps_per_sweep=200,
                          swap_slices=5, swap_max=5, swap_minacc=0.0, swap_maxacc=1.0, com_maxstep=2.0))
        e.set_option(OPT_EXACT_DECISIONS, exact)
        e.set_cells(mode)
        if split:  # 2: a warp per chain
            e.set_launch(64, split_phases=split % 2, warp_per_chain=split == 2)
            e.run_batched(3)
        else:
            e.run_plain(3)
        out.append((e.get_beads(), e.get_next(), e.stats(0).accepts))
        e.close()
    assert out[0][2][1] > 20
    for x, n, acc in out[1:]:
        np.testing.assert_array_equal(x, out[0][0])
        np.testing.assert_array_equal(n, out[0][1])
        assert acc == out[0][2]


def test_longest_chains_stage_alike(engine_lib):
    """a chain past the lengths where staging goes from stage_slot to the cell lists
    (split sweeps, the fused kernel): lists and row scans, in split sweeps, whole
    sweeps in one launch and lone launches, move the same beads"""
    from pimc.engine import ChainParams, Engine, Mix
    p = ChainParams(dim=2, N=6200, M=6, L=48.0, T=1.0, lam=0.5, interactions=True, pair_g=1.0, pair_sigma=0.4,
                    r_a=1.0, semantics=1, seed=29)
    out = []
    for how, mode in (("plain", 0), ("split", 0), ("split", 2), ("fused", 0), ("fused", 2)):
        e = Engine(p, Mix(stage_slices=3, stage_max=3, stage_minacc=0.0, stage_maxacc=1.0, swaps_per_sweep=20,
                          swap_slices=3, swap_max=3, swap_minacc=0.0, swap_maxacc=1.0, com_phases=0))
        e.set_cells(mode)
        if how == "plain":
            e.run_plain(1)
        else:
            e.set_launch(256, split_phases=int(how == "split"))
            e.run_batched(1)
        out.append((e.get_beads(), e.stats(0).accepts, e.stats(0).bead_updates))
        e.close()
    assert out[0][1][0] > 6200
    for x, acc, beads in out[1:]:
        np.testing.assert_array_equal(x, out[0][0])
        assert acc == out[0][1] and beads == out[0][2]


def test_128_register_swaps_stay_a_choice(engine_lib):
    """phase_regs 128 names a kernel: it is reported as chosen, unlike 0, which
    leaves the choice open, and where no other is offered it is 0; all give the
    same chains"""
    from pimc.engine import ChainParams, Engine, Mix
    ps = [ChainParams(dim=2, N=N, M=12, L=5.0, T=1.0, lam=0.5, harmonic_omega=1.0, interactions=True, pair_g=1.0,
                      pair_sigma=0.4, r_a=1.0, semantics=1, seed=N) for N in (9, 40, 300)]
    out = []
    for block, regs in ((64, 128), (64, 0), (64, 170), (64, 255), (128, 128)):
        e = Engine(ps, Mix(stage_slices=4, stage_max=4, swaps_per_sweep=40, swap_slices=4, swap_max=4))
        e.set_launch(block, split_phases=1, state_smem_bytes=0, phase_regs=(0, regs, 0))
        assert e.launch["phase_regs"] == [0, regs if block == 64 else 0, 0]
        e.run_batched(3)
        out.append([e.get_beads(c) for c in range(3)])
        e.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("sem", [0, 1])
@pytest.mark.parametrize("e", [-90, 80])
def test_chains_in_any_unit_of_length(e, sem, engine_lib):
    """the same chains with every length times 2^e (beyond the square roots of
    FP32's range): positions times 2^e and the same decisions and observables,
    bit for bit, since a power of two scales every product exactly"""
    from pimc.engine import ChainParams, Engine, Mix
    out = []
    for k in (0, e):
        u = 2.0 ** k
        kw = dict(dim=2, M=16, L=4.0 * u, T=1.0, lam=0.5 * u * u, harmonic_omega=1.0 / u, interactions=True,
                  pair_g=1.0, pair_sigma=0.5 * u, r_a=1.0 * u, semantics=sem, seed=3)
        eng = Engine([ChainParams(N=N, **kw) for N in (7, 40, 160)],
                     Mix(stage_slices=6, stage_max=6, swaps_per_sweep=60, swap_slices=6, swap_max=6,
                         com_step=0.5 * u, com_minstep=0.1 * u, com_maxstep=2.0 * u, measure_every=1))
        eng.run_batched(4)
        s, _, cnt = eng.energy_sums_all()
        eng.set_launch(64, split_phases=1)
        eng.run_batched(2)
        s2, _, _ = eng.energy_sums_all()
        out.append(([eng.get_beads(c) / u for c in range(3)], [eng.stats(c).accepts for c in range(3)], s, s2, cnt))
        eng.close()
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
    assert out[0][1] == out[1][1]
    for k in (2, 3, 4):
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert np.all(out[0][2][:, 2] != 0.0)


def test_measurement_of_chains_too_long_to_stage(engine_lib):
    """a chain of more particles than the measurement launches stage: a split
    sweep's and a lone chain's observables as pimc_measure's, within the bounds of
    test_measurement_launches_agree (the sums of 2100 particles' positive terms
    round within 1e-10 as well)"""
    from pimc.engine import ChainParams, Engine, Mix
    p = ChainParams(dim=2, N=2100, M=4, L=20.0, T=0.5, lam=0.5, harmonic_omega=0.2, interactions=True, pair_g=1.0,
                    pair_sigma=0.5, r_a=1.5, energy_capacity=4, seed=5)
    for split in (0, 1):
        e = Engine(p, Mix(stage_slices=2, stage_max=2, swaps_per_sweep=20, swap_slices=2, swap_max=2, com_maxstep=2.0,
                          measure_every=1))
        if split:
            e.set_launch(128, split_phases=1)
            e.run_batched(1)
        else:
            e.run_plain(1)
        got = e.observables()[-1]
        e.reset_measurements()
        e.measure()
        want = e.observables()[0]
        e.close()
        scale = np.maximum(np.abs(want), 1.0)
        assert np.all(np.abs(got - want)[[0, 1, 4, 5, 6]] <= 1e-10 * scale[[0, 1, 4, 5, 6]])
        assert np.all(np.abs(got - want)[[2, 3]] <= 2e-7 * scale[[2, 3]]) and want[2] > 0.0


def test_adjoint_of_one_chain_by_slices(engine_lib):
    """a lone chain of enough slices for a CTA each, against FP64 numpy with the
    bound of test_adjoint_gather_edges"""
    from pimc.engine import ChainParams, Engine
    N, M = 9, 700
    rng = np.random.default_rng(8)
    x = np.clip(rng.normal(scale=1.0, size=(2, N, M)), -3.99, 3.99)
    nxt = rng.permutation(N).astype(np.int32)
    e = Engine(ChainParams(dim=2, N=N, M=M, L=4.0, T=0.5, lam=0.5, harmonic_omega=0.7, lattice_V0=1.5, lattice_a=1.0,
                           interactions=True, pair_g=1.3, pair_sigma=0.5, r_a=1.2, semantics=1))
    e.set_beads(x)
    e.set_next(nxt)
    g, th, _ = e.adjoint()
    e.close()
    want, th_want = _adjoint_reference(x, nxt, 0.5, 4.0, 0.7, 1.5, 1.3, 0.5, 1.2, True)
    np.testing.assert_allclose(g, want, rtol=0, atol=1e-12 * np.abs(want).max())
    np.testing.assert_allclose(th, th_want, rtol=1e-12, atol=1e-13)
