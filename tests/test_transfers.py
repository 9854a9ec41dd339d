"""Loads and read-backs on both sides of the size that takes one copy through
the context's buffer (256 KB), and requests of some of the arrays only."""
import ctypes as C

import numpy as np
import pytest

import cellsim3d_b200 as cs
from cellsim3d_b200 import _lib
from cellsim3d_b200 import workloads as W

pytestmark = pytest.mark.gpu

NODE = ("X", "Y", "Z", "VX", "VY", "VZ")
CELL = ("pressure", "youngs")


def _arrays(n, seed):
    """n cells of the mesh on a line, with velocities, pressures and stiffnesses of their own; padding zero."""
    rng = np.random.default_rng(seed)
    c = np.zeros((n, 3), np.float32)
    c[:, 0] = 2.6 * np.arange(n) + 2.0
    c[:, 1:] = 2.0
    st = W.state(c)
    a = {k: st[k] for k in "XYZ"}
    for k in ("VX", "VY", "VZ"):
        v = rng.normal(0, 0.01, (n, 192)).astype(np.float32)
        v[:, 180:] = 0
        a[k] = v.reshape(-1)
    a["pressure"] = rng.uniform(50, 60, n).astype(np.float32)
    a["youngs"] = rng.uniform(900, 1100, n).astype(np.float32)
    return a


def _ensemble(mesh, n):
    """A context whose second instance has room for n cells and does not begin at cell 0."""
    p = W.base_params(box_len=(5000.0, 10.0, 10.0), growth_rate=0.0, use_rigid_box=0)
    a = _arrays(3, 1)
    topo = cs.build_topology(cs.mesh_from_arrays(mesh), a["X"][:192], a["Y"][:192], a["Z"][:192])
    ens = cs.Ensemble([p, p], topo, [3, n + 2])
    ens.load_state(0, **{k: a[k] for k in ("X", "Y", "Z")}, n_cells=3)
    return ens, p


def _get(ens, wanted, n, fn="cs3d_get_state"):
    """The wanted arrays alone, from the C call; what is not asked for is NULL."""
    keys = NODE + CELL if fn == "cs3d_get_state" else ("FCX", "FCY", "FCZ", "FDX", "FDY", "FDZ")
    out = {k: np.full(n if k in CELL else n * 192, np.nan, np.float32) for k in wanted}
    ptr = [out[k].ctypes.data_as(C.POINTER(C.c_float)) if k in wanted else None for k in keys]
    nn = C.c_int32()
    lead = [C.byref(nn)] if fn == "cs3d_get_state" else []
    _lib.check(getattr(_lib.lib(), fn)(ens.h, 1, *lead, *ptr), fn)
    assert not lead or nn.value == n
    return out


# 4616 bytes a cell with velocities and both cell arrays, 2304 with positions alone
@pytest.mark.parametrize("n", [1, 56, 57, 58, 113, 114, 150])
@pytest.mark.parametrize("with_v", [0, 1])
@pytest.mark.parametrize("with_cells", [(), ("pressure",), ("youngs",), CELL])
def test_load_and_read_back(mesh, n, with_v, with_cells):
    a = _arrays(n, n)
    ens, p = _ensemble(mesh, n)
    given = {k: a[k] for k in NODE[:6 if with_v else 3] + tuple(with_cells)}
    held = {k: v.copy() for k, v in given.items()}
    ens.load_state(1, **held, n_cells=n)
    for v in held.values():   # the caller's arrays are free once the call returns
        v[:] = np.nan
    want = dict(given)
    for k in NODE[3:]:
        want.setdefault(k, np.zeros(n * 192, np.float32))
    want.setdefault("pressure", np.full(n, p["min_pressure"], np.float32))
    want.setdefault("youngs", np.full(n, p["stiffness1"], np.float32))
    full = ens.state(1)
    for k in NODE + CELL:
        assert np.array_equal(full[k], want[k]), k
    for wanted in (("X",), ("Z",), ("VY",), ("Y", "VZ"), NODE[:3], NODE[3:], ("pressure",), ("youngs",), CELL,
                   ("X", "youngs"), ("VX", "pressure"), NODE, ()):
        got = _get(ens, wanted, n)
        for k in wanted:
            assert np.array_equal(got[k], want[k]), (wanted, k)
    ens.close()


@pytest.mark.parametrize("n", [56, 57, 114, 150])
def test_partial_read_back_of_forces_and_after_steps(mesh, n):
    a = _arrays(n, n)
    ens, _ = _ensemble(mesh, n)
    ens.load_state(1, **a, n_cells=n)
    ens.step(2)
    f = ens.forces(1)
    assert all(np.abs(v).max() > 0 for v in f.values())
    for wanted in (("FCY",), ("FDZ",), ("FCX", "FDX"), ("FDX", "FDY", "FDZ"), ()):
        got = _get(ens, wanted, n, "cs3d_get_forces")
        for k in wanted:
            assert np.array_equal(got[k], f[k]), (wanted, k)
    full = ens.state(1)
    for wanted in (("Y",), ("VX", "VZ"), ("Z", "pressure"), CELL):
        got = _get(ens, wanted, n)
        for k in wanted:
            assert np.array_equal(got[k], full[k]), (wanted, k)
    other = ens.state(0)
    assert other["n"] == 3 and len(other["X"]) == 3 * 192
    ens.close()
