"""A cell that is broken (NaN or infinite nodes) raises its error and leaves the
cells that do not touch it as they are without it."""
import numpy as np
import pytest

import cellsim3d_b200 as cs
from cellsim3d_b200 import workloads as W

pytestmark = pytest.mark.gpu

NAN = 0x001


def _cells(mesh, k=3, spacing=2.15):
    """k^3 cells in contact, [n, 192, 3] float32, and their box."""
    xyz = W.centred(W.scaled_xyz(mesh))
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * spacing + 2.0
    x = np.zeros((len(c), 192, 3), np.float32)
    x[:, :180] = xyz[None] + c[:, None].astype(np.float32)
    return x, float(k * spacing + 4.0)


def _run(mesh, x, box, steps=2, beside=None, **over):
    """Initial forces, then forces, state and cell data after some steps, and
    the error bits; beside: the cells of a second instance."""
    p = W.base_params(box_len=(box, box, box), growth_rate=0.0)
    p.update(over)
    rest = np.zeros((192, 3), np.float32)
    rest[:180] = W.centred(W.scaled_xyz(mesh))
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])
    xs = [x] if beside is None else [x, beside]
    sim = cs.Ensemble([p] * len(xs), topo, [len(y) for y in xs])
    for k, y in enumerate(xs):
        sim.load_state(k, *[np.ascontiguousarray(y[..., q].reshape(-1)) for q in range(3)], n_cells=len(y))
    out = [sim.forces()]
    sim.step(steps, raise_on_error=False)
    out += [sim.forces(), sim.state(), sim.cells()]
    err = sim.last_error()
    sim.close()
    return out, err


def _same(a, b, n, keep):
    """The per-node and per-cell arrays of the n cells `keep` picks from a, against all of b's."""
    for x, y in zip(a, b):
        for k in x:
            if k == "n":
                continue
            u = np.asarray(x[k]).reshape(n, -1)[keep]
            v = np.asarray(y[k]).reshape(len(u), -1)
            assert np.array_equal(u, v), k


@pytest.mark.parametrize("axes", [(0, 1, 2), (0,), (1,), (2,), (0, 2)])
@pytest.mark.parametrize("ensemble", [0, 1])
def test_cell_without_numbers_along_an_axis(mesh, axes, ensemble):
    """Forces, states and cell data of the others bit for bit, beside a cell
    whose nodes are all NaN along some axes (it has no box there), in the lists
    built at the load and in those of every step that follow from the NaN."""
    x, box = _cells(mesh)
    beside = x if ensemble else None
    want, err = _run(mesh, x, box, beside=beside)
    assert err == 0
    n = len(x) + 1
    broken = x[13:14].copy()
    broken[..., list(axes)] = np.nan
    y = np.concatenate([x[:13], broken, x[13:]])
    got, err = _run(mesh, y, box, beside=beside)
    assert err & NAN
    keep = np.arange(n) != 13
    _same(got, want, n, keep)


def test_nan_neighbour_leaves_the_conservative_force(mesh):
    """Two cells in contact, one of which has a NaN velocity at a node that
    touches nothing: in the first step the node and its three bond neighbours
    have NaN positions, listed as contacts of the other cell's nodes.  Their
    pairs take no part in the conservative force, which is that of the run
    without the NaN less the forces of those pairs, to the rounding of the two
    float results."""
    p = W.base_params(box_len=(20.0, 20.0, 20.0), growth_rate=0.0, use_rigid_box=0)
    st = W.state(np.array([[5.0, 5.0, 5.0], [7.1, 5.1, 5.05]], np.float32))
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), st["X"][:192], st["Y"][:192], st["Z"][:192])
    nn = np.asarray(mesh["nn"])[:, :180].T

    def run(node=None):
        sim = cs.Simulation(p, topo, 2)
        sim.set_option(cs.OPT_RECORD_PAIRS, 1)
        sim.set_option(cs.OPT_PAIR_CAPACITY, 1 << 16)
        v = [np.zeros(2 * 192, np.float32) for _ in range(3)]
        if node is not None:
            v[0][192 + node] = np.nan
        sim.load_state(st["X"], st["Y"], st["Z"], *v, n_cells=2)
        first = sim.pairs(0)
        sim.step(1, raise_on_error=False)
        f = sim.forces()
        s = sim.state()
        sim.close()
        return (first, np.stack([f["FC" + k] for k in "XYZ"], -1)[:180].astype(np.float64),
                np.stack([s[k] for k in "XYZ"], -1).astype(np.float64))

    pairs, want, x = run()
    touching = set(pairs[pairs[:, 0] == 1][:, 1].tolist())
    # a node next to a touching one that touches nothing itself
    node = next(m for m in range(180) if m not in touching and touching & set(nn[m].tolist()))
    gone = {node} | set(nn[node].tolist())
    _, got, y = run(node)
    assert np.isnan(y[192 + np.array(sorted(gone)), 0]).all() and np.isfinite(y[:180]).all()
    assert np.isfinite(got).all()
    lost = np.zeros((180, 3))
    for a, i, _, j in pairs:
        if a == 0 and j in gone:
            d = x[i] - x[192 + j]
            r = np.linalg.norm(d)
            assert r < p["attraction_range"] - 1e-4 and abs(r - p["repulsion_range"]) > 1e-4
            e = p["youngs_mod"]
            k = -p["attraction_strength"] * e * (p["attraction_range"] - r)
            if r < p["repulsion_range"]:
                k += p["repulsion_strength"] * e * (p["repulsion_range"] - r)
            lost[i] += k * d / r
    assert (np.abs(lost).max(1) > 0).any()
    tol = 2.0 ** -23 * (np.abs(want).max(1) + np.abs(got).max(1) + np.abs(lost).max(1))[:, None]
    assert (np.abs(want - lost - got) <= tol).all()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("far", [-9.0e4, -1.0e5, -4.0e5])
def test_contacts_of_a_wide_system(mesh, axis, far):
    """The cells of a cluster bit for bit with a lone cell so far below them
    that their grid bins number more than 16 bits hold (32767 bins of 2.9)."""
    x, box = _cells(mesh)
    want, err = _run(mesh, x, box, use_rigid_box=0)
    assert err == 0
    n = len(x) + 1
    lone = x[:1].copy()
    lone[:, :180, axis] += np.float32(far)
    got, err = _run(mesh, np.concatenate([x[:13], lone, x[13:]]), box, use_rigid_box=0)
    assert err == 0
    _same(got, want, n, np.arange(n) != 13)


@pytest.mark.parametrize("ensemble", [0, 1])
def test_cell_at_infinity(mesh, ensemble):
    """A cell at +inf in x: its box and centre of mass are there, and the
    others' forces, states and cell data are those without it, bit for bit."""
    x, box = _cells(mesh)
    beside = x if ensemble else None
    want, _ = _run(mesh, x, box, beside=beside, use_rigid_box=0)
    n = len(x) + 1
    far = x[13:14].copy()
    far[:, :180, 0] = np.inf
    got, err = _run(mesh, np.concatenate([x[:13], far, x[13:]]), box, beside=beside, use_rigid_box=0)
    assert err & NAN   # its forces are no numbers, and so its positions after a step
    _same(got, want, n, np.arange(n) != 13)


def test_centre_of_mass_of_an_infinite_node(mesh):
    """Centres of mass and boxes as float64 sums give them, with one node of one cell at -inf, at the load."""
    x, box = _cells(mesh, k=2)
    x[5, 17, 1] = -np.inf
    out, _ = _run(mesh, x, box, steps=0, use_rigid_box=0)
    cells = out[-1]
    cm = (x[:, :180].astype(np.float64).sum(1) / 180.0).astype(np.float32)
    assert np.isneginf(cells["cm"][5, 1]) and np.isneginf(cm[5, 1])
    # the float64 sums differ by their order, so that the floats may differ by one
    ok = np.isfinite(cm)
    assert ok.sum() == cm.size - 1
    assert np.allclose(cells["cm"][ok], cm[ok], rtol=2.0 ** -23, atol=0)
    assert np.array_equal(cells["aabb"][:, 0::2], x[:, :180].min(1))
    assert np.array_equal(cells["aabb"][:, 1::2], x[:, :180].max(1))


def test_grid_of_a_system_that_reaches_minus_infinity(mesh):
    """With a cell at -inf along an axis every node's bin is the last one and
    every box's range begins past it (float to int conversion saturates, as in
    the reference's grid), so that no pair counts."""
    x, box = _cells(mesh, k=2)
    rest = np.zeros((192, 3), np.float32)
    rest[:180] = W.centred(W.scaled_xyz(mesh))
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])
    far = x[:1].copy()
    far[:, :180, 2] = -np.inf
    counts = []
    for y in (x, np.concatenate([x, far])):
        sim = cs.Simulation(W.base_params(box_len=(box, box, box), growth_rate=0.0), topo, len(y))
        sim.set_option(cs.OPT_RECORD_PAIRS, 1)
        sim.set_option(cs.OPT_PAIR_CAPACITY, 1 << 16)
        sim.load_state(*[np.ascontiguousarray(y[..., q].reshape(-1)) for q in range(3)], n_cells=len(y))
        counts.append(len(sim.pairs(1)))
        sim.close()
    assert counts[0] > 0 and counts[1] == 0


def test_area_and_volume_of_a_broken_cell(mesh):
    """The division test of a cell with a NaN node stores a volume and an area
    that are no numbers and raises its bit; those of a cell that does not touch it are
    those of the run without the NaN."""
    x, box = _cells(mesh, k=2)
    got = []
    for node in (None, 17):
        y = x.copy()
        if node is not None:
            y[5, node] = np.nan
        out, err = _run(mesh, y, box, steps=1, growth_rate=0.002, division_vol=1e3)
        got.append(out[-1])
    assert err & NAN and err & 0x010
    for k in ("volume", "area"):
        assert np.isnan(got[1][k][5]) and np.isfinite(got[0][k]).all() and (got[0][k] > 0).all()
    far = (np.abs(x[:, 0] - x[5, 0]) > 1.0).sum(1) == 3   # the one that does not touch it
    assert far.sum() == 1
    for k in ("volume", "area"):
        assert np.array_equal(got[0][k][far], got[1][k][far])
