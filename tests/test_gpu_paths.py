"""The kernels' size-dependent forms against the oracle, at the sizes where one
form gives way to another.

Tolerances: FP64 as in test_gpu_fp64_parity.py (1e-10 of the force scale and of
an energy); mixed forces 1e-5 rms as in test_gpu_mixed.py.  A Monte Carlo chain's
sums keep one order whatever number of blocks it takes: bit for bit."""
import dataclasses

import numpy as np
import pytest

from oracle import mlp_oracle as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _water(n_mol, stretch=(0.0, 0.0, 0.0), seed=5, **kw):
    """A water box, its edges lengthened (vacuum beside the water)."""
    from thecodecombo_7_gb300 import systems
    s = systems.water_box(n_mol, density=0.1, seed=seed)
    return dataclasses.replace(s, L=np.asarray(s.L, float) + np.asarray(stretch, float), **kw)


# grids: ragged factors of 2, 3 and 5; a factor of 7 (the library); a plane too
# large for shared memory
@pytest.mark.parametrize("n_mol,stretch,grid,order,switch", [
    (200, (0, 0, 0), (20, 24, 30), 4, 0.0),
    (200, (0, 3, 5), (16, 27, 25), 3, 8.0),
    (201, (2, 0, 1), (32, 18, 40), 5, 0.0),
    (223, (0, 0, 4), (21, 24, 28), 6, 0.0),
    (200, (0, 0, 0), (30, 30, 30), 7, 8.0),
    (200, (0, 0, 0), (24, 135, 128), 8, 0.0),
])
def test_fp64_forces_over_grids_orders_and_boxes(n_mol, stretch, grid, order, switch):
    from thecodecombo_7_gb300 import engine
    s = _water(n_mol, stretch, grid=grid, order=order, r_switch=switch)
    f_ref, en_ref = O.Oracle(s).forces(s.pos)
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        b.nblist()
        en = b.forces()
        f = b.get_forces()
    scale = np.abs(f_ref).max()
    assert np.abs(f - f_ref).max() <= 1e-10 * scale
    for k in ("nbond", "kewald", "rewald", "iewald", "bond", "bend"):
        assert abs(en[k] - en_ref[k]) <= 1e-10 * max(1.0, abs(en_ref[k])), (k, en[k], en_ref[k])


# list units of one site (to 7,499 sites) and of four, rows of the outer list (to
# 8,192) and of the inner one
@pytest.mark.parametrize("n_mol,stretch,switch", [
    (500, (0, 0, 0), 0.0), (500, (3, 0, 1), 8.0), (2431, (0, 2, 0), 0.0),
    (2433, (0, 0, 0), 8.0), (2433, (1, 0, 3), 0.0), (2731, (0, 0, 0), 0.0),
    (2731, (0, 4, 0), 8.0),
])
def test_mixed_forces_over_row_forms(n_mol, stretch, switch):
    from thecodecombo_7_gb300 import engine
    s = _water(n_mol, stretch, r_switch=switch)
    f_ref, _ = O.Oracle(s).forces(s.pos)
    with engine.Box(s, precision=engine.FE_PREC_MIXED) as b:
        b.nblist()
        b.forces()  # with an inner list: the pruning walk
        f1 = b.get_forces()
        b.forces()  # the walk of the inner rows
        f2 = b.get_forces()
    for f in (f1, f2):
        assert np.sqrt(((f - f_ref) ** 2).sum() / (f_ref ** 2).sum()) <= 1e-5


@pytest.mark.parametrize("n_mol", [500, 2731])
def test_mixed_nose_hoover_run_equals_its_steps(n_mol):
    """Steps of one run fold the scale that ends one into the next; runs of one
    step do not.  They differ by the rounding of one product per velocity; a
    coordinate that rounds to another of the 2^32 fractions changes a force by
    1e-5 kJ/mol/A and a velocity by 1e-7 of its rms: 1e-6 over seven steps."""
    from thecodecombo_7_gb300 import engine
    s = _water(n_mol)
    out = []
    for runs in ([7], [1] * 7):
        with engine.Box(s, precision=engine.FE_PREC_MIXED) as b:
            b.nblist()
            b.forces()
            rec, i = [], 1
            for k in runs:
                rec.append(b.run_md(k, nlist_freq=4, use_nhc=True, first_step=i))
                i += k
            out.append((b.get_positions(), b.get_velocities()[0], np.concatenate(rec)))
    (p1, v1, r1), (p2, v2, r2) = out
    vrms = np.sqrt((v1 ** 2).mean())
    assert np.abs(v1 - v2).max() <= 1e-6 * vrms
    assert np.abs(p1 - p2).max() <= 7 * s.dt * 1e-6 * vrms
    assert np.abs(r1 - r2).max() <= 1e-6 * np.abs(r1).max()


# clusters of 8, 8, 4 and 2 blocks per chain, one block per chain
@pytest.mark.parametrize("surrogate", [False, True])
def test_mc_chain_is_the_same_in_every_cluster(surrogate):
    from thecodecombo_7_gb300 import engine
    s = _water(1365, seed=31)
    rng = np.random.default_rng(2)
    first = None
    for nchains in (1, 9, 30, 60, 160):
        with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
            b.mc_chains_setup(nchains=nchains, seed=4, log_cap=40)
            if surrogate:
                net = engine.Mlp(seed=1)
                if first is None:
                    P = rng.normal(0, 0.15, net.n_params).astype(np.float32)
                net.set_params(P, np.zeros(M.N_IN), np.ones(M.N_IN))
                b.mc_chains_set_surrogate(net)
                b.mc_chains_set_mode(1)
                net.close()
            b.mc_chains_run(25)
            b.mc_chains_run(15)  # a second launch starts from the first's state
            rec, fx = b.mc_chains_log(40)
            xyz, moves, acc = b.mc_chains_state(0)
            got = (rec, fx, xyz, moves, acc, b.mc_chains_kspace_energy(0))
        if first is None:
            first = got
            assert moves == 40 and acc > 0
        for a, r in zip(got, first):
            assert np.array_equal(a, r, equal_nan=True), nchains


# one block's rows, a cluster's, several of each block
@pytest.mark.parametrize("B", [64, 192, 576, 1024])
def test_mlp_gradient_over_batch_sizes(B):
    from thecodecombo_7_gb300 import engine
    rng = np.random.default_rng(B)
    net = engine.Mlp(seed=5)
    try:
        P = rng.normal(0, 0.15, net.n_params).astype(np.float32)
        mean = rng.normal(0, 0.1, M.N_IN).astype(np.float32)
        istd = rng.uniform(0.8, 1.2, M.N_IN).astype(np.float32)
        net.set_params(P, mean, istd)
        data = rng.normal(0, 1, (B, 2 * M.N_IN)).astype(np.float32)
        y = rng.normal(0, 0.5, B).astype(np.float32)
        loss, G, out = net.grad(data, y)
    finally:
        net.close()
    l_ref, G_ref, out_ref = M.forward_backward(P, data, y, mean, istd)
    assert abs(loss - l_ref) <= 1e-4 * abs(l_ref)
    assert np.abs(out - out_ref).max() <= 1e-3 * (1 + np.abs(out_ref).max())
    for a, b in ((M.OFF_W1, M.OFF_B1), (M.OFF_B1, M.OFF_W2), (M.OFF_W2, M.OFF_B2),
                 (M.OFF_B2, M.OFF_W3), (M.OFF_W3, M.OFF_B3)):
        g, r = G[a:b].astype(np.float64), G_ref[a:b]
        assert np.linalg.norm(g - r) <= 2e-3 * max(np.linalg.norm(r), 1e-12)


def test_fp64_pairs_of_sites_past_2_to_the_25():
    """A dilute FP64 box of 2^25 + 64 sites on a lattice wider than the cutoff,
    the last 64 in 32 charged close pairs: the energies are those of a box that
    holds the 64 alone, and the forces on them too, but for the mean reciprocal
    force, which another number of sites shares."""
    from thecodecombo_7_gb300 import engine, systems
    n, h, m = (1 << 25) + 64, 8.0, 323
    i = np.arange(n)
    pos = np.stack([i // (m * m), i // m % m, i % m], 1) * h - 0.5 * h * (m - 1)
    rng = np.random.default_rng(3)
    d = rng.normal(size=(32, 3))
    d *= (rng.uniform(1.5, 2.0, 32) / np.linalg.norm(d, axis=1))[:, None]
    pos[n - 63::2] = pos[n - 64::2] + d
    q = np.zeros(n)
    q[n - 64::2], q[n - 63::2] = 0.4, -0.4
    none = np.zeros((0, 2), np.int32)
    s = systems.System(
        L=np.full(3, m * h), pos=pos, q=q, mass=np.full(n, 12.0), type=np.zeros(n, np.int32),
        vel=np.zeros((n, 3)), type_eps_kcal=np.array([-0.15]), type_rmin_half=np.array([0.9]),
        bonds=none, bond_req=np.zeros(0), bond_k=np.zeros(0), bends=np.zeros((0, 3), np.int32),
        bend_theta0=np.zeros(0), bend_k=np.zeros(0), excl=none, excl_flag=np.zeros(0, np.int32),
        rc=5.0, rclist=5.4, rclist_ew=5.4, rc_ew=5.0, kappa=0.6, grid=(64, 64, 64))
    with engine.Box(s, precision=engine.FE_PREC_FP64, max_neighbors=8) as b:
        b.nblist()
        assert b.list_stats() == (32, 1)
        en = b.forces()
        f = b.get_forces()[n - 64:]
    last = dataclasses.replace(s, pos=pos[n - 64:].copy(), q=q[n - 64:], mass=s.mass[n - 64:],
                               type=s.type[n - 64:], vel=s.vel[n - 64:])
    f_ref, en_ref = O.Oracle(last).forces(last.pos)
    f, f_ref = f - f.mean(0), f_ref - f_ref.mean(0)
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    for k in ("nbond", "nbonds", "rewald", "kewald"):
        assert abs(en[k] - en_ref[k]) <= 1e-10 * max(1.0, abs(en_ref[k])), (k, en[k], en_ref[k])


@pytest.mark.parametrize("charged", [False, True])
def test_fp64_sites_that_coincide_without_charge(charged):
    """Two hydrogens (no LJ) of different molecules at one place, one of them or
    both without charge: no real-space term, in the energy or the forces."""
    from thecodecombo_7_gb300 import engine, systems
    s = systems.water_box(200, L=25.0, seed=9, grid=(24, 24, 24))
    o = s.pos[0::3]
    d = o - o[0]
    d -= s.L * np.round(d / s.L)
    near = int(np.argsort((d ** 2).sum(1))[1])
    q = s.q.copy()
    q[:3] = 0.0
    if not charged:
        q[3 * near:3 * near + 3] = 0.0
    pos = s.pos.copy()
    pos[3 * near + 1] = pos[1]
    s = dataclasses.replace(s, q=q, pos=pos)
    f_ref, en_ref = O.Oracle(s).forces(s.pos)
    assert np.isfinite(f_ref).all()
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        b.nblist()
        en = b.forces()
        f = b.get_forces()
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    for k in ("nbond", "rewald", "kewald", "iewald"):
        assert abs(en[k] - en_ref[k]) <= 1e-10 * max(1.0, abs(en_ref[k])), (k, en[k], en_ref[k])


# a charged site with LJ, one without, and one in no excluded pair's reach
@pytest.mark.parametrize("site,axis,value", [(0, 0, np.nan), (4, 2, np.nan), (4, 1, -np.nan),
                                             (7, 0, np.inf)])
def test_fp64_energies_show_positions_that_are_not_finite(site, axis, value):
    """A list built from good positions, then one coordinate that is not a
    number: the energy terms that the reference's loop makes NaN are NaN.  An
    infinite one is beyond every cutoff in that loop."""
    from thecodecombo_7_gb300 import engine, systems
    s = systems.water_box(200, L=25.0, seed=9, grid=(24, 24, 24))
    orc = O.Oracle(s)
    nl = orc.nblist(s.pos)
    bad = s.pos.copy()
    bad[site, axis] = value
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        b.nblist()
        b.set_positions(bad)
        en = b.forces()
    _, e5 = orc.pair_forces(bad, nl)  # LJ, its shift, real space, its shift, excluded pairs
    assert np.isnan(e5[2]) == np.isnan(value)
    for k, want in (("rewald", e5[2]), ("iewald", e5[4])):
        if np.isnan(want):
            assert np.isnan(en[k]), k
        else:
            assert abs(en[k] - want) <= 1e-10 * max(1.0, abs(want)), (k, en[k], want)


def test_inner_list_stats_of_small_boxes():
    """Boxes that walk the outer list report an inner list of nothing, and the
    one that a batch of more sites keeps for them; radii without room for one
    are refused."""
    from thecodecombo_7_gb300 import engine
    ss = [_water(n, seed=70 + n) for n in (900, 950, 1000)]
    boxes = [engine.Box(s, precision=engine.FE_PREC_MIXED) for s in ss]
    try:
        for b in boxes:
            b.nblist()
            b.forces()
            assert b.inner_list_stats() == (0, 0, 0)
        batch = engine.Batch(boxes, seed=3)
        batch.set_fused(True)  # 8,550 sites in all
        batch.run(3, nlist_freq=10, swap_freq=0, first_step=1)
        for b, s in zip(boxes, ss):
            entries, row, prunes = b.inner_list_stats()
            assert prunes == 1 and 0 < row <= entries < b.list_stats()[0]
        batch.close()
    finally:
        for b in boxes:
            b.close()
    s = _water(500, rclist=10.5, rclist_ew=10.5)
    with engine.Box(s, precision=engine.FE_PREC_MIXED) as b:
        b.nblist()
        b.forces()
        with pytest.raises(engine.FeError) as ei:
            b.inner_list_stats()
    assert ei.value.code == engine.FE_ERR_STATE


def test_step_launches_are_those_of_an_ordinary_step():
    """Steps inside a mixed Nose-Hoover run take the launches of a plain run's
    steps: the thermostat rides on their last kernel."""
    from thecodecombo_7_gb300 import engine
    with engine.Box(_water(500), precision=engine.FE_PREC_MIXED) as b:
        b.nblist()
        b.forces()
        got = []
        for nhc in (False, True):
            b.run_md(3, nlist_freq=10, use_nhc=nhc, record=False)
            got.append(b.step_launches(nhc))
    assert got[0] == got[1] and got[0][0] < got[0][1]


# rows shared by warps and whole rows; 1-4 pairs and torsions
@pytest.mark.parametrize("which", ["water_200", "water_1365", "chains_150"])
def test_fp64_energies_repeat(which):
    """Energies at fixed positions are the same bits in every evaluation, with the
    same list, with one built again and in a box of its own: every sum has its
    order.  (Forces are summed by FP64 atomics and may differ in the last bit.)"""
    from thecodecombo_7_gb300 import engine, systems
    n = int(which.split("_")[1])
    s = systems.chain_box(n, seed=3) if which.startswith("chains") else _water(n)
    seen = set()
    for _ in range(3):
        with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
            for _ in range(4):
                b.nblist()
                for _ in range(3):
                    en = b.forces()
                    seen.add(tuple(en.values()))
    assert len(seen) == 1


# orders on four and on eight lanes a site; the project's transforms and (a factor of
# 7) the library's; many sites a grid point
@pytest.mark.parametrize("order,grid", [(4, (24, 24, 24)), (6, (25, 24, 27)), (4, (21, 24, 28)),
                                        (3, (8, 8, 8))])
def test_fp64_reciprocal_space_repeats(order, grid):
    """The charge grid, the reciprocal energy and its forces are the same bits in
    every evaluation of the same positions, and those of the oracle."""
    from thecodecombo_7_gb300 import engine
    s = _water(1365, order=order, grid=grid)
    orc = O.Oracle(s)
    seen = []
    for _ in range(2):
        with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
            for _ in range(4):
                g = b.charge_grid()
                b.zero_forces()
                e = b.pme_calc()
                seen.append((g, np.array(e), b.get_forces()))
    for got in seen[1:]:
        for a, r in zip(got, seen[0]):
            assert np.array_equal(a, r)
    g, e, f = seen[0]
    f_ref, e_ref = orc.pme(s.pos)
    np.testing.assert_allclose(g, orc.charge_grid(s.pos), rtol=0, atol=1e-13)
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    assert np.abs(e - e_ref).max() <= 1e-10 * np.abs(e_ref).max()


def test_fp64_reciprocal_space_shows_positions_that_are_not_finite():
    """As a sum of FP64 values would: the energy and every force are NaN, with the
    project's transforms and the library's, and no longer once the position is."""
    from thecodecombo_7_gb300 import engine
    for grid in ((24, 24, 24), (21, 24, 28)):
        s = _water(200, grid=grid)
        with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
            for value in (np.nan, np.inf):
                bad = s.pos.copy()
                bad[17, 1] = value
                b.set_positions(bad)
                b.zero_forces()
                assert np.isnan(b.pme_calc()[0])
                assert np.isnan(b.get_forces()).all()
                b.set_positions(s.pos)
                b.zero_forces()
                assert np.isfinite(b.pme_calc()).all() and np.isfinite(b.get_forces()).all()


def test_fp64_charge_grid_beyond_its_counts():
    """Lumps of 200 ions of each sign, 47 e at the grid point under them, where a
    point's count overflows at 16 e: the grid, the energy and the forces of the
    oracle.  The grid's sums of 200 values up to 50 e: 200 roundings of 4e-15."""
    from thecodecombo_7_gb300 import engine
    s = _water(200, seed=4)
    pos = s.pos.copy()
    pos[:200] = s.L * (np.array([8, 9, 10]) / np.array(s.grid) - 0.5)
    pos[200:400] = s.L * (np.array([17.5, 3.25, 12]) / np.array(s.grid) - 0.5)
    pos[:400] += np.random.default_rng(1).uniform(0, 1e-3, (400, 3))
    q = s.q.copy()
    q[:200], q[200:400], q[400:] = 0.8, -0.8, 0.0
    s = dataclasses.replace(s, pos=pos, q=q)
    orc = O.Oracle(s)
    g_ref = orc.charge_grid(s.pos)
    assert g_ref.max() > 40 and g_ref.min() < -16
    f_ref, e_ref = orc.pme(s.pos)
    seen = []
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        for _ in range(3):
            g = b.charge_grid()
            b.zero_forces()
            e = np.array(b.pme_calc())
            seen.append((g, e, b.get_forces()))
    for got in seen[1:]:
        for a, r in zip(got, seen[0]):
            assert np.array_equal(a, r)
    g, e, f = seen[0]
    assert np.abs(g - g_ref).max() <= 1e-12
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    assert np.abs(e - e_ref).max() <= 1e-10 * np.abs(e_ref).max()


# x lines in tiles of 16 (from 4,864 lines on) and of 8 on the same planes' border; the
# smallest axes the transform kernels take (4) and the next ragged ones
@pytest.mark.parametrize("grid,order", [((16, 100, 100), 4), ((20, 90, 100), 5), ((16, 96, 100), 4),
                                        ((4, 4, 4), 4), ((4, 6, 8), 3), ((5, 9, 24), 4),
                                        ((25, 4, 6), 4)])
def test_fp64_forces_over_line_tiles_and_short_axes(grid, order):
    from thecodecombo_7_gb300 import engine
    s = _water(200, (0, 1, 2), grid=grid, order=order)
    f_ref, en_ref = O.Oracle(s).forces(s.pos)
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        b.nblist()
        en = b.forces()
        f = b.get_forces()
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    for k in ("kewald", "rewald", "iewald"):
        assert abs(en[k] - en_ref[k]) <= 1e-10 * max(1.0, abs(en_ref[k])), (k, en[k], en_ref[k])


# the cutoff at half the box and beyond it
@pytest.mark.parametrize("rc", [10.0, 10.5])
def test_fp64_image_rule_at_half_the_box(rc):
    """Sites of a lattice, in any order, exactly half a box apart: the reference
    subtracts a box length beyond half a box, not at it."""
    from thecodecombo_7_gb300 import engine, systems
    rng = np.random.default_rng(12)
    i = rng.permutation(64)
    pos = np.stack([i // 16, i // 4 % 4, i % 4], 1) * 5.0 - 7.5
    q = rng.normal(0, 0.4, 64)
    q -= q.mean()
    none = np.zeros((0, 2), np.int32)
    s = systems.System(
        L=np.full(3, 20.0), pos=pos, q=q, mass=np.full(64, 12.0), type=np.zeros(64, np.int32),
        vel=np.zeros((64, 3)), type_eps_kcal=np.array([-0.15]), type_rmin_half=np.array([2.2]),
        bonds=none, bond_req=np.zeros(0), bond_k=np.zeros(0), bends=np.zeros((0, 3), np.int32),
        bend_theta0=np.zeros(0), bend_k=np.zeros(0), excl=none, excl_flag=np.zeros(0, np.int32),
        rc=rc, rclist=11.0, rclist_ew=11.0, rc_ew=rc, kappa=0.32, grid=(20, 20, 20))
    f_ref, en_ref = O.Oracle(s).forces(s.pos)
    with engine.Box(s, precision=engine.FE_PREC_FP64) as b:
        b.nblist()
        en = b.forces()
        f = b.get_forces()
    assert np.abs(f - f_ref).max() <= 1e-10 * np.abs(f_ref).max()
    for k in ("nbond", "nbonds", "rewald", "kewald"):
        assert abs(en[k] - en_ref[k]) <= 1e-10 * max(1.0, abs(en_ref[k])), (k, en[k], en_ref[k])


# a batch of fewer tiles than the cluster has blocks, of as many, of more
@pytest.mark.parametrize("B", [64, 192, 512, 576])
def test_mlp_training_step_is_adam_on_the_gradient(B):
    """One batch, one epoch: Adam's first step from the gradient call's gradient.
    The step is lr g / (|g| + 1e-8): where |g| is above 1e-4 of the largest, the
    order of its sums moves it by far less than 1e-4 lr."""
    from thecodecombo_7_gb300 import engine
    rng = np.random.default_rng(B)
    data = rng.normal(0, 1, (B, 2 * M.N_IN)).astype(np.float32)
    y = rng.normal(0, 0.5, B).astype(np.float32)
    lr = 1e-2
    net = engine.Mlp(seed=5)
    try:
        P0 = net.get_params()[0].copy()
        hist = net.train(data, y, epochs=1, batch=B, lr=lr, seed=3)
        P1, mean, istd = (x.copy() for x in net.get_params())
        net.set_params(P0, mean, istd)
        loss, G, _ = net.grad(data, y)
    finally:
        net.close()
    G = G.astype(float)
    on = np.abs(G) > 1e-4 * np.abs(G).max()
    assert on.mean() > 0.5
    want = P0 - lr * G / (np.abs(G) + 1e-8)
    assert np.abs(P1 - want)[on].max() <= 1e-4 * lr + 2.0 ** -23 * np.abs(P0).max()
    assert abs(hist[0] - loss) <= 1e-5 * abs(loss)
