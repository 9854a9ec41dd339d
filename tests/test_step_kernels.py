"""Edges of the step's kernels: sizes around the tiles and the rules by which
one kernel or another takes a step."""
import numpy as np
import pytest

import cellsim3d_b200 as cs
from cellsim3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _grid_state(n, spacing=2.4):
    k = int(np.ceil(n ** (1.0 / 3.0)))
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * spacing + 1.5
    return W.state(c.astype(np.float32)), float(k * spacing + 3.0)


def _sim(p, st, mesh, capacity=None):
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    sim = cs.Simulation(p, topo, capacity or st["n"])
    sim.load_state(st["X"], st["Y"], st["Z"], st.get("VX"), st.get("VY"), st.get("VZ"), n_cells=st["n"])
    return sim


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 700])
def test_com_correction_is_the_float_sum_in_cell_order(mesh, n):
    """The shift at set-up equals the float32 sum of the centres of mass in
    cell order over n, subtracted from every node (bit for bit)."""
    st, box = _grid_state(n)
    p = W.base_params(box_len=(box, box, box), growth_rate=0.0, correct_com=1, use_rigid_box=0)
    sim = _sim(p, st, mesh)
    got = sim.state()
    cm = sim.cells()["cm"]
    for q, k in enumerate("XYZ"):
        s = np.float32(0)
        for v in cm[:, q]:
            s = np.float32(s + v)
        want = st[k].reshape(n, 192) - np.float32(s / np.float32(n))
        assert np.array_equal(got[k].reshape(n, 192)[:, :180], want[:, :180])
    sim.close()


def _pairs_within(x, ra):
    """(cell, node, cell, node) of the nodes of different cells within ra, sorted keys."""
    from scipy.spatial import cKDTree
    n = x.shape[0]
    flat = x.reshape(n * 180, 3)
    pairs = cKDTree(flat).query_pairs(ra * 1.01, output_type="ndarray")
    pairs = pairs[pairs[:, 0] // 180 != pairs[:, 1] // 180]
    r = np.linalg.norm(flat[pairs[:, 0]] - flat[pairs[:, 1]], axis=1)
    assert len(r) == 0 or np.abs(r - ra).min() > 1e-7   # no pair that rounding decides
    pairs = pairs[r < ra]
    both = np.concatenate([pairs, pairs[:, ::-1]])
    return np.sort(both[:, 0].astype(np.int64) * (n * 180) + both[:, 1])


@pytest.mark.parametrize("small,scale", [(0, 1.0), (1, 1.0), (30, 8.0), (200, 8.0), (200, 14.0)])
def test_list_build_around_a_large_cell(mesh, small, scale):
    """Contact pairs against a search over all nodes where one cell's box
    reaches `small` others: below and above the 128 candidate slots, and with
    a cell so large that the table of the cells is left aside."""
    rng = np.random.default_rng(3)
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    turn = np.linalg.qr(rng.normal(size=(3, 3)))[0]
    k = int(np.ceil(max(small, 1) ** (1.0 / 3.0)))
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:small] * 1.15 - 0.575 * (k - 1)
    c = c + rng.uniform(-0.05, 0.05, c.shape)
    big = xyz @ turn * scale
    if small:   # one in contact with a node of the large cell
        c[small // 2] = big[7] * (1.0 - 0.6 / scale) if scale > 1 else [2.15, 0.0, 0.0]
    x = [big] + [xyz * (0.5 if scale > 1 else 1.0) + p for p in c]
    x = (np.stack(x) + 20.0).astype(np.float32)
    n = len(x)
    st = {"n": n}
    for q, key in enumerate("XYZ"):
        st[key] = np.zeros((n, 192), np.float32)
        st[key][:, :180] = x[..., q]
        st[key] = st[key].reshape(-1)
    p = W.base_params(box_len=(60.0, 60.0, 60.0), growth_rate=0.0, use_rigid_box=0)
    rest = np.zeros((192, 3), np.float32)
    rest[:180] = xyz
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])
    sim = cs.Simulation(p, topo, n)
    sim.set_option(cs.OPT_RECORD_PAIRS, 1)
    sim.set_option(cs.OPT_PAIR_CAPACITY, 1 << 20)
    sim.load_state(st["X"], st["Y"], st["Z"], n_cells=n)
    sim.forces()
    got = sim.pairs(0).astype(np.int64)
    got = np.sort((got[:, 0] * 180 + got[:, 1]) * (n * 180) + got[:, 2] * 180 + got[:, 3])
    want = _pairs_within(x.astype(np.float64), float(np.float32(p["attraction_range"])))
    assert np.array_equal(got, want)
    assert small == 0 or len(want) > 0
    sim.close()


def _growing(n, **over):
    """n cells close to each other; all of them divide in the first step (their volume is above the division volume)."""
    st, box = _grid_state(n, spacing=2.25)
    p = W.base_params(box_len=(box, box, box), div_time_steps=10 ** 9, rng_ij=11, rng_kl=1100)
    p.update(over)
    if p.get("correct_com"):
        p["use_rigid_box"] = 0
    return p, st


@pytest.mark.parametrize("n,steps,over", [(1, 40, {}), (8, 300, {}), (20, 60, {"correct_com": 1}),
                                          (20, 60, {"add_rands": 1, "rand_scale_factor": 0.1, "rand_seed": 5}),
                                          (60, 40, {"count_internal_radius": 0.5}), (74, 12, {}), (75, 12, {}),
                                          (148, 6, {"growth_rate": 0.0}), (149, 6, {"growth_rate": 0.0})])
def test_steps_in_one_kernel_equal_the_launch_sequence(mesh, n, steps, over):
    """A system small enough for the one-kernel path (alone) and the same
    system beside another instance that makes the context too large for it:
    states and events bit for bit, over sizes around the limit, divisions,
    the options of a step and several launches."""
    p, st = _growing(n, **over)
    q, big = _growing(200, growth_rate=0.0)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    got = []
    for others in (0, 1):
        ens = cs.Ensemble([p] + [q] * others, topo, [4 * n + 8] + [200] * others)
        ens.load_state(0, st["X"], st["Y"], st["Z"], n_cells=n)
        if others:
            ens.load_state(1, big["X"], big["Y"], big["Z"], n_cells=200)
        ens.step(steps - 1)
        ens.step(1)
        got.append((ens.state(0), ens.events(0), ens.forces(0), ens.cells(0), ens.far_counts(0)))
        ens.close()
    (a, ea, fa, ca, ra), (b, eb, fb, cb, rb) = got
    assert a["n"] == b["n"] and np.array_equal(ea, eb) and np.array_equal(ra, rb)
    for x, y in ((a, b), (fa, fb), (ca, cb)):
        for k in x:
            assert np.array_equal(x[k], y[k]), k


def _pack(x):
    st = {"n": len(x)}
    for q, key in enumerate("XYZ"):
        a = np.zeros((len(x), 192), np.float32)
        a[:, :180] = x[..., q]
        st[key] = a.reshape(-1)
    return st


def _distorted(mesh, noise):
    """The mesh at rest and three copies with random displacements of their nodes."""
    rng = np.random.default_rng(17)
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    x = np.stack([xyz] + [xyz + rng.normal(0, noise, xyz.shape) + [4.0 * (k + 1), 0, 0] for k in range(3)]) + 5.0
    return _pack(x.astype(np.float32))


def _crowded(mesh, flat):
    """The mesh at rest and a pair of flattened copies face to face."""
    rng = np.random.default_rng(19)
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    a = xyz * [1.0, 1.0, flat] + rng.normal(0, 1e-3, xyz.shape)
    b = a[:, [1, 0, 2]] + [0.03, 0.02, a[:, 2].max() - a[:, 2].min() + 0.15]
    return _pack((np.stack([xyz + [6.0, 0, 0], a, b]) + 3.0).astype(np.float32))


@pytest.mark.parametrize("make,arg", [(_distorted, 0.01), (_distorted, 0.06), (_distorted, 0.12),
                                      (_crowded, 1.0), (_crowded, 0.3), (_crowded, 0.1)])
def test_forces_of_bent_and_crowded_cells(mesh, make, arg):
    """Initial forces and contact pairs against the FP64 oracle, where bond
    angles lie on both sides of the polynomial's range (distorted cells) and
    where nodes have from none to several groups of eight entries (flattened
    cells face to face)."""
    from parity import TOL, force_errors, make_pair, sorted_pairs
    st = make(mesh, arg)
    p = W.base_params(box_len=(60.0, 60.0, 60.0), growth_rate=0.0, use_rigid_box=0)
    sim, orc = make_pair(p, st, mesh, capacity=st["n"])
    ec, ed = force_errors(sim, orc)
    assert ec[0] < TOL and ed[0] < TOL, (ec, ed)
    for kind in (0, 1):
        assert np.array_equal(sorted_pairs(sim.pairs(kind)), sorted_pairs(orc.recorded_pairs(kind)))
    sim.close()


@pytest.mark.parametrize("skin,over", [(0.25, {}), (0.35, {}), (0.2, {"correct_com": 1})])
def test_partial_builds_do_not_change_results(mesh, skin, over):
    """A growing colony with a wide list skin against the default one, bit for
    bit.  At 0.35 the radius of a partial build around a division gives some
    node more entries than it has room for (a whole build stays below): the
    cell takes the smaller radius and the instance is rebuilt in the next step.
    With the centre-of-mass correction the boxes that a division's neighbours are
    found by lie apart from the nodes."""
    p, st = _growing(64, **over)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    got = []
    for s in (0.1, skin):
        sim = cs.Simulation(p, topo, 512)
        sim.set_option(cs.OPT_SKIN, int(round(s * 1e6)))
        sim.load_state(st["X"], st["Y"], st["Z"], n_cells=64)
        sim.step(1200)
        got.append((sim.state(), sim.events()))
        sim.close()
    (a, ea), (b, eb) = got
    assert np.array_equal(ea, eb)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n", [8, 160])
@pytest.mark.parametrize("com", [0, 1])
def test_reloaded_context_repeats_the_run(mesh, n, com):
    """With noise, growth and divisions: a load into a context that has already
    run gives the states, forces and events of a fresh context, bit for bit
    (a daughter's slot keeps nothing of the cell it held before), with the steps
    in one kernel (8 cells) and as a launch sequence (160)."""
    p, st = _growing(n, add_rands=1, rand_scale_factor=0.5, rand_seed=5, correct_com=com)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    rng = cs.Ranmar(p["rng_ij"], p["rng_kl"])
    got = []
    for passes in (1, 2):
        sim = cs.Simulation(p, topo, 3 * n)
        for _ in range(passes):
            known = len(sim.events())
            sim.load_state(st["X"], st["Y"], st["Z"], n_cells=n)
            sim.set_rng(rng)
            sim.step(10)
        got.append((sim.state(), sim.forces(), sim.random_force(), sim.events()[known:]))
        sim.close()
    (a, fa, ra, ea), (b, fb, rb, eb) = got
    assert a["n"] == b["n"] > n and len(ea) == a["n"] - n and len(eb) == len(ea)
    for u, v in ((a, b), (fa, fb), (ra, rb)):
        for k in u:
            assert np.array_equal(u[k], v[k]), k


def _crowd_around(xyz, near, far):
    """A large flat cell, a cell inside it and others outside, each at a gap from
    a node of the large one: 115 at `near`, 35 at `far`."""
    from scipy.spatial import cKDTree
    axes = np.array([18.0, 18.0, 8.0])
    big = xyz * axes
    tree = cKDTree(big)
    cells = [big, xyz * 1.3]
    for q, i in enumerate(np.random.default_rng(1).permutation(180)[:150]):
        gap = near if q < 115 else far
        out = big[i] / axes ** 2
        out /= np.linalg.norm(out)
        lo, hi = 0.0, 3.0
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            if tree.query(xyz * 0.9 + big[i] + out * mid)[0].min() < gap:
                lo = mid
            else:
                hi = mid
        cells.append(xyz * 0.9 + big[i] + out * hi)
    return np.stack(cells)


def test_partial_build_with_more_candidates_than_slots(mesh):
    """A cell with 115 others within the list radius and 35 more within that of
    a partial build, which adds the distances from the anchors: 150 are more
    candidates than there are slots.  All cells drift at one velocity and the
    one inside divides in the first step.  The steps run, and their states are
    those with a skin so small that every build is a whole one."""
    from scipy.spatial import cKDTree
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    x = _crowd_around(xyz, 0.35, 0.45)
    # 0.3 and a skin of 0.1; two steps of 0.02 and less than half the skin
    gaps = np.array([cKDTree(x[0]).query(c)[0].min() for c in x[2:]])
    assert (gaps < 0.39).sum() == 115 and (gaps < 0.475).sum() == 150 and gaps.min() > 0.31
    n = len(x)
    st = _pack((x + 30.0).astype(np.float32))
    v = np.zeros(n * 192, np.float32)
    u = v.reshape(n, 192)
    u[:, :180] = 200.0
    p = W.base_params(box_len=(60.0, 60.0, 60.0), use_rigid_box=0, constrain_angles=0, youngs_mod=1e-3,
                      stiffness1=1e-6, internal_damping=0.0, viscotic_damping=0.0, gamma_visc=0.0, max_pressure=0.0,
                      min_pressure=0.0, growth_rate=1e-9, division_vol=6.0)
    rest = np.zeros((192, 3), np.float32)
    rest[:180] = xyz
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])
    got = []
    for skin in (0.1, 0.03):
        sim = cs.Simulation(p, topo, n + 8)
        sim.set_option(cs.OPT_SKIN, int(round(skin * 1e6)))
        sim.load_state(st["X"], st["Y"], st["Z"], v, v * 0, v * 0, n_cells=n)
        sim.step(4)
        got.append((sim.state(), sim.events(), sim.forces()))
        assert (sim.stats()["list_fallbacks"] > 0) == (skin == 0.1)
        sim.close()
    (a, ea, fa), (b, eb, fb) = got
    assert np.array_equal(ea, eb) and ea.tolist() == [[1, 1, n]]
    for s, t in ((a, b), (fa, fb)):
        for k in s:
            assert np.array_equal(s[k], t[k]), k


def _small_and_large(mesh, scales, small, deep):
    """Small cells on a lattice and large ones past one of its corners each, in contact with a few."""
    rng = np.random.default_rng(23)
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    k = int(np.ceil(small ** (1.0 / 3.0)))
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:small] * 1.15
    c = c + rng.uniform(-0.05, 0.05, c.shape)
    x = [xyz * 0.5 + p for p in c]
    for q, s in enumerate(scales):
        turn = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        out = np.array([1.0 if q >> b & 1 else -1.0 for b in range(3)])
        at = np.where(out > 0, c.max(0), 0.0) + out / np.sqrt(3.0) * (s - deep)
        x.insert(len(x) // (q + 2), xyz @ turn * s + at)
    return (np.stack(x) + 40.0).astype(np.float32)


def _check_pairs(mesh, x):
    """Contact pairs of the cells x against a search over all nodes; the context's counters."""
    n = len(x)
    st = _pack(x)
    p = W.base_params(box_len=(400.0, 400.0, 400.0), growth_rate=0.0, use_rigid_box=0)
    rest = np.zeros((192, 3), np.float32)
    rest[:180] = W.centred(W.scaled_xyz(mesh))
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])
    sim = cs.Simulation(p, topo, n)
    sim.set_option(cs.OPT_RECORD_PAIRS, 1)
    sim.set_option(cs.OPT_PAIR_CAPACITY, 1 << 21)
    sim.load_state(st["X"], st["Y"], st["Z"], n_cells=n)
    sim.forces()
    got = sim.pairs(0).astype(np.int64)
    got = np.sort((got[:, 0] * 180 + got[:, 1]) * (n * 180) + got[:, 2] * 180 + got[:, 3])
    want = _pairs_within(x.astype(np.float64), float(np.float32(p["attraction_range"])))
    assert np.array_equal(got, want)
    s = sim.stats()
    sim.close()
    return s


@pytest.mark.parametrize("scales,small,deep,searches", [((3.0, 3.2, 3.4, 3.6), 300, 0.8, 0), ((8.6,), 190, 2.5, 0),
                                                        ((14.0,), 400, 0.8, 1), ((4.0, 5.0, 14.0), 400, 0.8, 1),
                                                        ((12.0,) * 6, 729, 0.8, 6)])
def test_list_build_with_several_large_cells(mesh, scales, small, deep, searches):
    """Contact pairs against a search over all nodes, with cells on both sides
    of the largest that the table of the cells takes, and with 129 to 192 and
    more boxes in reach of one.  The small cells find theirs through the table all
    the same: only a large cell looks at all the others."""
    x = _small_and_large(mesh, scales, small, deep)
    s = _check_pairs(mesh, x)
    assert s["full_searches"] == searches and s["lists_built"] == len(x)
    lo, hi = x[:, :180].min(1) - 0.2, x[:, :180].max(1) + 0.2
    reach = [(np.all((lo <= hi[a]) & (hi >= lo[a]), axis=1)).sum() - 1 for a in range(len(x))]
    if small == 190:
        assert 128 < max(reach) <= 192


def test_list_build_with_cells_of_three_sizes(mesh):
    """Contact pairs against a search over all nodes where more cells than the
    list of large ones holds are 4 and 8 times the size of the others, lattice
    beside lattice: the size classes of the table."""
    rng = np.random.default_rng(31)
    xyz = W.centred(W.scaled_xyz(mesh)).astype(np.float64)
    x, right = [], 0.0
    for scale, m in ((0.9, (5, 10, 10)), (8.0, (4, 5, 5)), (3.8, (4, 5, 5)), (0.6, (3, 8, 8))):
        c = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3) * (2.0 * scale + 0.1)
        c = c + rng.uniform(-0.02, 0.02, c.shape) + [right + scale, 0.0, 0.0]
        x += [xyz * scale + p for p in c]
        right = c[:, 0].max() + scale + 0.1
    x = (np.stack(x)[rng.permutation(len(x))] + 10.0).astype(np.float32)
    assert _check_pairs(mesh, x)["full_searches"] == 0


SYNC = 0x400


@pytest.mark.parametrize("instances,com", [(1, 0), (1, 1), (2, 0)])
@pytest.mark.parametrize("done", [0, 3])
def test_steps_that_give_up_at_a_barrier(mesh, instances, com, done):
    """Blocks that look for the others 0 times give up at the first barrier of a
    launch: the step ends with SYNC, and further ones (also profiled, also with
    the limit back at its default) are refused until every instance is loaded
    again.  Then the run is that of a fresh context, bit for bit, divisions
    included."""
    p, st = _growing(8, correct_com=com)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])

    def load(ens, k):
        ens.load_state(k, st["X"], st["Y"], st["Z"], n_cells=8)
        ens.set_rng(k, cs.Ranmar(p["rng_ij"], p["rng_kl"]))

    got = []
    for give_up in (0, 1):
        ens = cs.Ensemble([p] * instances, topo, [40] * instances)
        for k in range(instances):
            load(ens, k)
        if give_up:
            ens.step(done)
            ens.set_option(cs.OPT_SYNC_POLLS, 0)
            assert ens.step(600, raise_on_error=False) == -7
            assert all(ens.last_error(k) & SYNC for k in range(instances))
            ens.set_option(cs.OPT_SYNC_POLLS, 1 << 22)
            for k in range(instances):
                assert ens.step(1, raise_on_error=False) == -7
                with pytest.raises(cs.CS3DError):
                    ens.profile_step(1)
                load(ens, k)
            assert ens.last_error(-1) == 0
        known = [len(ens.events(k)) for k in range(instances)]
        ens.step(20)
        assert ens.stats()["launches_per_step"] == 1
        got.append([(ens.state(k), ens.forces(k), len(ens.events(k)) - known[k]) for k in range(instances)])
        ens.close()
    for (a, fa, ea), (b, fb, eb) in zip(*got):
        assert a["n"] == b["n"] == 8 + ea == 8 + eb > 8
        for u, v in ((a, b), (fa, fb)):
            for k in u:
                assert np.array_equal(u[k], v[k]), k


def test_barrier_limit_option_is_checked(mesh):
    p, st = _growing(1)
    sim = _sim(p, st, mesh)
    for bad in (-1, 1 << 32):
        with pytest.raises(cs.CS3DError):
            sim.set_option(cs.OPT_SYNC_POLLS, bad)
    sim.close()


def _multiprocessors():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("over", [{}, {"correct_com": 1}, {"add_rands": 1, "rand_scale_factor": 0.1, "rand_seed": 5}])
@pytest.mark.parametrize("at", [1, 8, "limit", "limit + 1", 300])
def test_kernels_of_a_step(mesh, over, at):
    """Which path takes the steps, by the kernels that they launch: one launch
    for up to 256 steps of a context with at most a cell for each
    multiprocessor (the first half kick apart, of every launch with the
    centre-of-mass correction), the sequence of a step beyond; the same for two
    instances, whose cells add up."""
    cells = {"limit": _multiprocessors(), "limit + 1": _multiprocessors() + 1}.get(at, at)
    one = cells <= _multiprocessors()
    p, st = _growing(cells, growth_rate=0.0, **over)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    half = cells // 2
    for parts in ([cells], [half, cells - half]) if half else ([cells],):
        ens = cs.Ensemble([p] * len(parts), topo, parts)
        first = 0
        for k, n in enumerate(parts):
            ens.load_state(k, *[st[q][first * 192:(first + n) * 192] for q in "XYZ"], n_cells=n)
            first += n
        com = bool(over.get("correct_com"))
        ens.step(300)
        s = ens.stats()
        sequence = 5 + (3 if com else 0)   # half kick, centre and shift
        assert s["launches_per_step"] == (1 if one else sequence)
        want = 2 + (2 if com else 1) if one else 300 * sequence + (0 if com else 1)
        assert s["launches"] == want
        ens.step(2)
        assert ens.stats()["launches"] - want == (1 + com if one else 2 * sequence)
        ens.close()


def test_growth_out_of_the_one_kernel_path(mesh):
    """A context that outgrows the one-kernel steps goes on with the sequence, between two launches and between two calls."""
    n = _multiprocessors() // 2 + 1
    p, st = _growing(n)
    sim = _sim(p, st, mesh, capacity=4 * n)
    sim.step(2)
    assert sim.n_cells() > _multiprocessors()
    assert sim.stats()["launches_per_step"] == 1 and sim.stats()["launches"] == 2
    sim.step(1)
    assert sim.stats()["launches_per_step"] == 7 and sim.stats()["launches"] == 9
    sim.close()


@pytest.mark.parametrize("skin,some", [(0.1, False), (0.35, True)])
def test_wide_skin_takes_the_fallback(mesh, skin, some):
    """The colony of test_partial_builds_do_not_change_results: at a skin of 0.35 some lists are built with the smaller radius."""
    p, st = _growing(64)
    sim = _sim(p, st, mesh, capacity=512)
    sim.set_option(cs.OPT_SKIN, int(round(skin * 1e6)))
    sim.step(1200)
    assert (sim.stats()["list_fallbacks"] > 0) == some
    sim.close()
