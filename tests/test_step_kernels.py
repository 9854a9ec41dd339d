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
