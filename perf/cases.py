"""The work that users of cellsim3d_b200 have it do, as timed cases.

A pass is what a program does between two points at which it looks at the
cells: it loads a state (a start, a restart, a checkpoint), takes steps and
reads the state back into page-locked memory; or it asks for the forces of a
state.  Every pass starts from the same loaded state and the same RANMAR
streams, so all passes on one state are the same work.

The cells of dividing systems are daughters of a division at all stages of
their growth, turned at random and in contact with their neighbours, and some
of them divide within a pass.  Cells of systems without growth are the unit
cells of the packed workloads.

Kinds of cases:
  forces  load a state and read the conservative and dissipative forces of its
          nodes (analysis of a stored frame; the start of every run)
  static  the same through the entry point without allocation, on device
          buffers the caller owns, 1 to 64 cells
  run     load, take `steps` steps, read the state back
  frames  load, take steps and read every `every` steps through the
          asynchronous read-back with its two slots (a trajectory writer)
  ensemble  many independent simulations of different sizes and parameters
          stepped together (parameter sweeps, seeds)
"""
import ctypes
import math

import numpy as np
import torch

import cellsim3d_b200 as cs
from cellsim3d_b200 import _lib
from cellsim3d_b200 import workloads as W

SLOTS, NODES = cs.SLOTS, cs.NODES
DIV_VOLUME = 2.9
COMPONENTS = ("X", "Y", "Z", "VX", "VY", "VZ")
FORCES = ("FCX", "FCY", "FCZ", "FDX", "FDY", "FDZ")


# ------------------------------------------------------------------- cases

def listed():
    return [
        # smallest call: the forces of a handful of cells
        dict(name="forces_8", kind="forces", cells=8, growing=True),
        # a plug-in host's force call on its own device buffers
        dict(name="static_27", kind="static", cells=27, growing=False),
        # analysis of a stored frame of a packed tissue
        dict(name="forces_3001", kind="forces", cells=3001, growing=False),
        # the first configuration of the benchmark: a few cells in a box
        dict(name="run_small8", kind="run", cells=8, growing=True, steps=300, noise=False, stiff=False),
        # a young colony between two trajectory frames
        dict(name="run_colony301", kind="run", cells=301, growing=True, steps=150, noise=False, stiff=False),
        # a grown colony, the decade in which most steps' time goes
        dict(name="run_colony2500", kind="run", cells=2500, growing=True, steps=100, noise=False, stiff=False),
        # Langevin force, centre-of-mass correction and softer cells switched on
        dict(name="run_noise1023", kind="run", cells=1023, growing=True, steps=60, noise=True, stiff=True),
        # a packed tissue without growth, one rank's worth of an ordinary study
        dict(name="run_packed10007", kind="run", cells=10007, growing=False, steps=60, noise=False, stiff=False),
        # the headline workload: 100k packed cells, state in and out over PCIe
        dict(name="run_packed100k", kind="run", cells=100000, growing=False, steps=40, noise=False, stiff=False),
        # trajectory output every 20 steps while the steps go on
        dict(name="frames_4100", kind="frames", cells=4100, growing=True, steps=80, every=20),
        # a parameter sweep of small colonies of very different sizes
        dict(name="ensemble_sweep", kind="ensemble", instances=48, least=1, most=512, steps=60, own_stiffness=False),
        # few large heterogeneous tissues with their own bond stiffness
        dict(name="ensemble_het", kind="ensemble", instances=8, least=256, most=8192, steps=30, own_stiffness=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("forces", "static", "run", "run", "run", "frames", "ensemble"))
    if kind == "forces":
        return dict(kind=kind, cells=_log(rng, 2, 6000), growing=rng.random() < 0.5)
    if kind == "static":
        return dict(kind=kind, cells=rng.randint(1, 64), growing=rng.random() < 0.5)
    if kind == "run":
        growing = rng.random() < 0.6
        cells = _log(rng, 1, 6000 if growing else 60000)
        odd = rng.random() < 0.25
        return dict(kind=kind, cells=cells, growing=growing, steps=rng.randint(20, 150 if cells < 4000 else 50),
                    noise=odd, stiff=odd and growing)
    if kind == "frames":
        return dict(kind=kind, cells=_log(rng, 4, 5000), growing=rng.random() < 0.7, steps=rng.randint(40, 100),
                    every=rng.randint(5, 25))
    if rng.random() < 0.5:
        return dict(kind=kind, instances=rng.randint(2, 64), least=1, most=_log(rng, 16, 512),
                    steps=rng.randint(20, 80), own_stiffness=rng.random() < 0.3)
    return dict(kind=kind, instances=rng.randint(2, 8), least=128, most=_log(rng, 512, 8192),
                steps=rng.randint(10, 30), own_stiffness=True)


# ------------------------------------------------------------------- inputs

def _rest_mesh():
    return W.centred(W.scaled_xyz(W.load_mesh()))


def _unit(v):
    return v / (np.linalg.norm(v, axis=-1, keepdims=True) if isinstance(v, np.ndarray) else v.norm(dim=-1, keepdim=True))


def _volume_area(x, faces):
    """Volume and area of meshes (k, 180, 3) about their centres, each face cut at its vertex mean."""
    x = x - x.mean(1, keepdims=True)
    vol = area = 0.0
    for f in range(92):
        p = x[:, faces[f, : 5 if f < 12 else 6]]
        m, q = p.mean(1, keepdims=True), np.roll(p, -1, 1)
        vol = vol + np.abs((np.cross(p, q) * m).sum(-1)).sum(-1) / 6
        area = area + np.linalg.norm(np.cross(p - m, q - m), axis=-1).sum(-1) / 2
    return vol, area


def _life(x, mesh, rest, most):
    """The free motion of cells without contacts (springs, pressure, bond
    angles, damping, drag; the step of the framework in 64 bits) until all of
    them would divide: positions and velocities every ten steps."""
    nn = mesh["nn"][:, :NODES].astype(int)
    arm0 = [rest[nn[k]] - rest for k in range(3)]
    r0 = [np.linalg.norm(a, axis=-1) for a in arm0]
    angles = ((0, 1), (1, 2), (0, 2))
    th0 = [np.arccos((_unit(arm0[a]) * _unit(arm0[b])).sum(-1)) for a, b in angles]
    # the arm of each neighbour that ends at a node, in the stacked arms
    back = np.array([[int(np.nonzero(nn[:, nn[q, i]] == i)[0][0]) * NODES + nn[q, i] for i in range(NODES)]
                     for q in range(3)])

    def conservative(x, press):
        arm = [x[:, nn[k]] - x for k in range(3)]
        R = [np.sqrt((a * a).sum(-1)) for a in arm]
        F = 3 * press * _unit(x - x.mean(1, keepdims=True))
        ends = [0.0, 0.0, 0.0]
        for k in range(3):
            F += (1000 * (1 / r0[k] - 1 / R[k]))[..., None] * arm[k]
        for (a, b), t in zip(angles, th0):
            P, Q, dot = arm[a], arm[b], (arm[a] * arm[b]).sum(-1)
            p2, q2 = R[a] ** 2, R[b] ** 2
            g = (1000 * (np.arccos(dot / (R[a] * R[b] + 1e-3)) - t) / np.sqrt(p2 * q2 - dot * dot + 1e-3))[..., None]
            ends[a] = ends[a] + g * (Q - (dot / p2)[..., None] * P)
            ends[b] = ends[b] + g * (P - (dot / q2)[..., None] * Q)
        all_ = np.concatenate(ends, 1)
        return F + all_[:, back[0]] + all_[:, back[1]] + all_[:, back[2]] - (ends[0] + ends[1] + ends[2])

    damping = lambda v: -100 * (3 * v - v[:, nn[0]] - v[:, nn[1]] - v[:, nn[2]]) - v
    v, press, half = np.zeros_like(x), 50.0, 0.5 * 1e-4 / 0.04
    fc, fd, got = conservative(x, press), damping(v), []
    for s in range(most):
        if s % 10 == 0:
            got.append((x, v))
            vol, area = _volume_area(x, mesh["faces"])
            round_ = np.abs(1 - 4.835975862049408 * np.cbrt(vol) ** 2 / area) <= 0.05
            if s and ((vol > DIV_VOLUME) & round_).all():
                break
        v = v + half * (fc + fd)
        x = x + v * 1e-4
        press += 0.002
        fc = conservative(x, press)
        v = v + half * (fc + damping(v))
        fd = damping(v)
    return got


_shapes = []


def _cell_shapes():
    """Shapes and node velocities of cells between their birth as one half of a
    divided cell and the end of their growth: (count, 180, 3) each."""
    if not _shapes:
        mesh, rest = W.load_mesh(), _rest_mesh().astype(np.float64)
        parent = _life(0.8 * rest[None], mesh, rest, 600)[-1][0]
        normal = _unit(np.random.default_rng(5).normal(size=(4, 1, 3)))
        y = parent - parent.mean(1, keepdims=True) - 0.1 * normal
        d = (y * normal).sum(-1, keepdims=True)
        lives = _life(y - np.where(d <= 0, d, 0) * normal, mesh, rest, 1000)
        lives = lives[: int(0.9 * len(lives))]
        x = np.concatenate([a - a.mean(1, keepdims=True) for a, _ in lives])
        _shapes.append((x, np.concatenate([v for _, v in lives])))
    return _shapes[0]


def _centres(cells, spacing, jitter, gen):
    """Cell centres (float64, on the GPU) on a jittered face-centred lattice
    with the given nearest distance, `cells` of its sites inside a cube, and
    the side of the cube."""
    k = max(1, int(math.ceil((cells / 4.0) ** (1.0 / 3.0))))
    a = spacing * math.sqrt(2.0)
    r = torch.arange(k, dtype=torch.float64, device="cuda")
    g = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 1, 3)
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], dtype=torch.float64, device="cuda")
    sites = ((g + basis).reshape(-1, 3) + 0.25) * a
    keep = torch.randperm(len(sites), generator=gen, device="cuda")[:cells].sort().values
    c = sites[keep]
    return c + (torch.rand(c.shape, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1) * jitter, k * a


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


class _System:
    """One system's parameters and state, arrays on the GPU."""

    def __init__(self, cells, growing, seed, noise=False, stiff=False, bond=1000.0, spread=1.0):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed) % (1 << 62))
        if growing:
            shapes, moves = (torch.from_numpy(t).cuda() for t in _cell_shapes())
            which = torch.randint(len(shapes), (cells,), generator=gen, device="cuda")
            q = torch.randn(cells, 3, 3, generator=gen, device="cuda", dtype=torch.float64)
            e1 = _unit(q[:, 0])
            e2 = _unit(q[:, 1] - (q[:, 1] * e1).sum(-1, keepdim=True) * e1)
            turn = torch.stack([e1, e2, torch.linalg.cross(e1, e2)], 1)
            c, side = _centres(cells, 2.2 * spread, 0.05, gen)
            x0, v0 = shapes[which] @ turn, (moves[which] @ turn).float()
        else:
            # fcc at volume fraction 0.5 of unit cells, the packed workloads' density
            c, side = _centres(cells, (4 * (4.0 / 3.0) * math.pi / 0.5) ** (1.0 / 3.0) / math.sqrt(2.0), 0.1, gen)
            x0 = torch.from_numpy(_rest_mesh().astype(np.float64)).cuda()[None]
            v0 = torch.randn(cells, NODES, 3, generator=gen, device="cuda") * 0.01
        margin = 1.05
        c = c + margin
        box = side + 2 * margin
        x = torch.zeros(cells, SLOTS, 3, dtype=torch.float32, device="cuda")
        x[:, :NODES] = (x0 + c[:, None, :]).float()
        v = torch.zeros(cells, SLOTS, 3, dtype=torch.float32, device="cuda")
        v[:, :NODES] = v0
        self.cells = cells
        self.nodes = {k: x[..., q].reshape(-1).contiguous() for q, k in enumerate("XYZ")}
        self.nodes.update({"V" + k: v[..., q].reshape(-1).contiguous() for q, k in enumerate("XYZ")})
        press = torch.rand(cells, generator=gen, device="cuda") + 50 if growing else torch.full((cells,), 200.0, device="cuda")
        self.pressure = press.float().cpu().numpy()
        ij, kl = W.seed_pair(int(seed) % 301)
        p = W.base_params(box_len=(box, box, box), div_time_steps=10 ** 9, rng_ij=ij, rng_kl=kl, stiffness1=bond,
                          division_vol=DIV_VOLUME)
        if not growing:
            p.update(growth_rate=0.0, min_pressure=200.0, max_pressure=200.0, div_time_steps=5000)
        if noise:
            # a free cluster: the correction moves it out of any box
            p.update(add_rands=1, rand_scale_factor=0.1, rand_seed=int(seed) % 100000, correct_com=1, use_rigid_box=0)
        self.youngs = np.full(cells, bond, np.float32)
        if stiff:
            p = W.soft_params(p, 0.8, phase_count=2000000000)
            soft = torch.rand(cells, generator=gen, device="cuda") < 0.25
            self.youngs[soft.cpu().numpy()] = np.float32(p["stiffness2"])
        self.params = p
        # room for the divisions of a pass
        self.capacity = 2 * cells + 8 if growing else cells

    def host(self):
        return {k: _pinned(a) for k, a in self.nodes.items()}


def _systems(case, seed):
    if case["kind"] != "ensemble":
        return [_System(case["cells"], case["growing"], seed, noise=bool(case.get("noise")), stiff=bool(case.get("stiff")))]
    # the sizes and stiffnesses are the study's design: they belong to the case
    sm = W.SplitMix(2024 + case["instances"] + case["most"])
    out = []
    for k in range(case["instances"]):
        n = int(round(case["least"] * math.exp(sm.uniform() * math.log(case["most"] / case["least"]))))
        bond = 500 + 1500 * sm.uniform() if case["own_stiffness"] else 1000.0
        growth = 0.001 + 0.003 * sm.uniform()
        s = _System(max(1, n), True, seed * 1009 + k, bond=float(np.float32(bond)), spread=1.0 + 0.1 * sm.uniform())
        s.params["growth_rate"] = growth
        out.append(s)
    return out


def _topology():
    rest = np.zeros((SLOTS, 3), np.float32)
    rest[:NODES] = _rest_mesh()
    return cs.build_topology(cs.mesh_from_arrays(W.load_mesh()), *[np.ascontiguousarray(rest[:, q]) for q in range(3)])


def _buffers(capacities):
    """Page-locked room for every instance's state, back to back: the whole
    arrays, and each instance's part of them."""
    total = sum(capacities)
    whole = {k: torch.zeros(total * SLOTS, dtype=torch.float32, pin_memory=True).numpy() for k in COMPONENTS}
    whole.update({k: torch.zeros(total, dtype=torch.float32, pin_memory=True).numpy() for k in ("pressure", "youngs")})
    parts, at = [], 0
    for c in capacities:
        parts.append({k: a[at * SLOTS:(at + c) * SLOTS] if k in COMPONENTS else a[at:at + c] for k, a in whole.items()})
        at += c
    return whole, parts


def prepare(case, seed):
    sys_ = _systems(case, seed)
    st = {"case": case, "topo": _topology()}
    if case["kind"] == "static":
        s = sys_[0]
        st.update(params=cs.make_params(s.params), nodes=s.nodes, cells=s.cells,
                  out={k: torch.zeros(s.cells * SLOTS, dtype=torch.float32, device="cuda") for k in FORCES})
        torch.cuda.synchronize()
        return st
    st["ens"] = cs.Ensemble([s.params for s in sys_], st["topo"], [s.capacity for s in sys_])
    st["in"] = [dict(s.host(), pressure=s.pressure, youngs=s.youngs, n_cells=s.cells) for s in sys_]
    st["rng"] = [cs.Ranmar(s.params["rng_ij"], s.params["rng_kl"]) for s in sys_]
    if case["kind"] != "forces":
        # a frame writer has two buffers, one for each slot of the read-back
        st["out"] = [_buffers([s.capacity for s in sys_]) for _ in range(2 if case["kind"] == "frames" else 1)]
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- pass

def run(st):
    case = st["case"]
    if case["kind"] == "static":
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        _lib.check(_lib.lib().cs3d_forces_static(
            ctypes.byref(st["params"]), ctypes.byref(st["topo"]), st["cells"], *[ptr(st["nodes"][k]) for k in COMPONENTS],
            None, None, *[ptr(st["out"][k]) for k in FORCES], None), "cs3d_forces_static")
        return st["out"]
    ens = st["ens"]
    for k, a in enumerate(st["in"]):
        ens.load_state(k, **a)
        ens.set_rng(k, st["rng"][k])
    if case["kind"] == "forces":
        return ens.forces()
    if case["kind"] == "frames":
        counts, done = [], 0
        while done < case["steps"]:
            k = min(case["every"], case["steps"] - done)
            ens.step(k)
            done += k
            slot = len(counts) & 1
            ens.wait_state(slot)
            counts.append(ens.state_async(0, slot, st["out"][slot][1][0]))
        ens.wait_state(0)
        ens.wait_state(1)
        # the last two frames, in the buffers, and the cell counts of all
        return {"counts": np.array(counts, np.int64), "slot0": st["out"][0][0], "slot1": st["out"][1][0]}
    ens.step(case["steps"])
    whole, parts = st["out"][0]
    counts = [ens.state(k, out=o)["n"] for k, o in enumerate(parts)]
    return {"counts": np.array(counts, np.int64), "state": whole}


def _sizes(case):
    if case["kind"] != "ensemble":
        return [case["cells"]]
    sm = W.SplitMix(2024 + case["instances"] + case["most"])
    out = []
    for _ in range(case["instances"]):
        out.append(max(1, int(round(case["least"] * math.exp(sm.uniform() * math.log(case["most"] / case["least"]))))))
        for _ in range(3 if case["own_stiffness"] else 2):
            sm.uniform()
    return out


def work(case):
    """Bytes: the state in (24 B a node) and out (24 B), and for each step the
    positions and velocities read and written once (48 B a node), as the
    benchmark counts them.  Operations of a step, a node: three springs, the
    pressure, three bond angles, about two contacts, two dissipative forces,
    three kicks and its share of the cell's centre and volume."""
    nodes = sum(_sizes(case)) * NODES
    steps = case.get("steps", 1)
    return {"bytes": nodes * 48.0 * (steps + 1), "flops": nodes * 700.0 * steps}


# ------------------------------------------------- the forces in 64 bits

def _contact_pairs(x, ra):
    """Nodes (cell, node) of different cells within ra of each other: indices
    (i, j) into the flattened (cells * 180) nodes, both orders."""
    n = x.shape[0]
    lo, hi = x.min(1).values, x.max(1).values
    near = ((lo[:, None] - ra <= hi[None]) & (hi[:, None] + ra >= lo[None])).all(-1)
    near.fill_diagonal_(False)
    a, b = near.nonzero(as_tuple=True)
    got = [], []
    for k in range(0, len(a), 2048):
        p, q = a[k:k + 2048], b[k:k + 2048]
        d = x[p][:, :, None, :] - x[q][:, None, :, :]
        m, i, j = ((d * d).sum(-1) <= ra * ra).nonzero(as_tuple=True)
        got[0].append(p[m] * NODES + i)
        got[1].append(q[m] * NODES + j)
    if not got[0]:
        z = torch.zeros(0, dtype=torch.int64, device=x.device)
        return z, z
    return torch.cat(got[0]), torch.cat(got[1])


def exact(case, seed):
    """The initial forces in FP64 (springs, pressure, bond angles, contacts,
    walls; bond damping, friction, drag).  Runs of many steps have none."""
    if case["kind"] not in ("forces", "static"):
        return None
    s = _systems(case, seed)[0]
    p, n = s.params, s.cells
    f = {k: float(np.float32(v)) for k, v in p.items() if isinstance(v, (int, float))}
    prod = lambda a, b: float(np.float32(a) * np.float32(b))
    x32 = torch.stack([s.nodes[k].view(n, SLOTS)[:, :NODES] for k in "XYZ"], -1)
    x = x32.double()
    v = torch.stack([s.nodes["V" + k].view(n, SLOTS)[:, :NODES] for k in "XYZ"], -1).double()
    mesh = W.load_mesh()
    nn = torch.from_numpy(np.ascontiguousarray(mesh["nn"][:, :NODES]).astype(np.int64)).cuda()
    sign = torch.from_numpy(np.asarray(mesh["sign"][:NODES]).astype(np.float64)).cuda()
    # rest lengths and angles, held in 32 bits as the mesh tables are
    rest = torch.from_numpy(_rest_mesh()).cuda().double()
    arm0 = [rest[nn[k]] - rest for k in range(3)]
    ang = lambda a, b: torch.acos((_unit(a) * _unit(b)).sum(-1))
    t = _topology()
    r0 = torch.from_numpy(np.array(t.r0, np.float64).reshape(3, SLOTS)[:, :NODES].copy()).cuda()
    th0 = torch.from_numpy(np.array(t.theta0, np.float64)[: 3 * NODES].reshape(NODES, 3).copy()).cuda()
    for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2))):
        assert float((ang(arm0[a], arm0[b]) - th0[:, k]).abs().max()) < 1e-3
        assert float((arm0[k].norm(dim=-1) - r0[k]).abs().max()) < 1e-5

    FC = torch.zeros_like(x)
    arm = [x[:, nn[k]] - x for k in range(3)]
    bond = torch.from_numpy(s.youngs).cuda().double() if case["kind"] == "forces" else torch.full((n,), f["stiffness1"], device="cuda", dtype=torch.float64)
    for k in range(3):
        FC += (bond[:, None] * (1 / r0[k] - 1 / arm[k].norm(dim=-1)))[..., None] * arm[k]
    press = torch.from_numpy(s.pressure).cuda().double() if case["kind"] == "forces" else torch.full((n,), f["min_pressure"], device="cuda", dtype=torch.float64)
    cm = x.mean(1).float().double()  # the centre of mass is a 32-bit state
    FC += 3 * press[:, None, None] * _unit(x - cm[:, None])
    for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2))):
        P, Q = arm[a], arm[b]
        dot, p2, q2 = (P * Q).sum(-1), (P * P).sum(-1), (Q * Q).sum(-1)
        dth = torch.acos(dot / (p2.sqrt() * q2.sqrt() + 1e-3)) - th0[:, k]
        g = (1000 * dth / (p2 * q2 - dot * dot + 1e-3).sqrt())[..., None]
        Fp, Fq = g * (Q - (dot / p2)[..., None] * P), g * (P - (dot / q2)[..., None] * Q)
        FC.index_add_(1, nn[a], Fp)
        FC.index_add_(1, nn[b], Fq)
        FC -= Fp + Fq
    ra, rr = f["attraction_range"], f["repulsion_range"]
    asE, rsE = prod(f["attraction_strength"], f["youngs_mod"]), prod(f["repulsion_strength"], f["youngs_mod"])
    i, j = _contact_pairs(x, ra)
    xf, vf = x.reshape(-1, 3), v.reshape(-1, 3)
    e = xf[i] - xf[j]
    R = e.norm(dim=-1)
    mag = torch.where(R < ra, -asE * (ra - R) / R, 0.0) + torch.where(R <= rr, rsE * (rr - R) / R, 0.0)
    FC.view(-1, 3).index_add_(0, i, mag[:, None] * e)
    wall, th = 100.0 * f["youngs_mod"], f["thresh_dist"]
    for q in range(3):
        box = torch.tensor(p["box_len"][q], dtype=torch.float32, device="cuda")
        g1, g2 = x32[..., q], box - x32[..., q]
        FC[..., q] += torch.where(g1 < np.float32(th), -wall * (g1.double() - th), 0.0)
        FC[..., q] += torch.where(g2 < np.float32(th), wall * (g2.double() - th), 0.0)

    S = torch.zeros_like(v)
    S.view(-1, 3).index_add_(0, i, vf[i] - vf[j])
    normal = _unit(torch.linalg.cross(x[:, nn[1]] - x[:, nn[0]], x[:, nn[2]] - x[:, nn[0]])) * sign[None, :, None]
    S = S - (S * normal).sum(-1, keepdim=True) * normal
    damp = sum(v - v[:, nn[k]] for k in range(3))
    FD = -f["internal_damping"] * damp - f["viscotic_damping"] * S - f["gamma_visc"] * v
    out = {}
    for name, F in (("FC", FC), ("FD", FD)):
        full = torch.zeros(n, SLOTS, 3, dtype=torch.float64, device="cuda")
        full[:, :NODES] = F
        for q, c in enumerate("XYZ"):
            a = full[..., q].reshape(-1).contiguous()
            out[name + c] = a if case["kind"] == "static" else a.cpu().numpy()
    return out
