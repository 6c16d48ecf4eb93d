"""The workloads the speed of this framework is judged by.

Every case is one thing a program does with the public interface
(``iwf_mfree_gpu_3d_b200.api`` / ``serve``): step a cutting scene (one call of
the reference's ``leap_frog::step``, or a few replays of the captured step),
step a batch of uneven scenes, serve one request from creation to read-back,
or build a cell list in place.  Sizes, materials and tools are those of the
scene generators, the tests and the benchmark: 1,600 to 4.1 million particles,
lattices with odd edges, one to five tools, meshes of 12 and 1,280 triangles,
hashed and exhaustive contact, the three conduction options, CSPM on and off,
plain and compensated positions, locked and unlocked grids.  Scenes start
either at rest (the first cut) or from a developed state: smooth stress,
velocity, density, temperature and plastic-strain fields, as after some
thousand steps.

``run`` returns the state arrays of the scene in its current (cell-sorted)
order as views of the device memory, without a copy.  The low parts of the
compensated form are left out of them: they are the rounding remainders of the
high parts, and what they do shows in the served request's read-back and in
the rates of the following step.

``exact`` restates one step of the method in FP64 with plain torch.  It covers
scenes of any size cut by wedges.  It is None for the icosphere tools, whose
inside test depends on last bits of a hit on a cell border of the triangle
grid, and for particles that belong to a tool.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from iwf_mfree_gpu_3d_b200 import api, scenes, serve

# ---------------------------------------------------------------- the cases --


def listed():
    return [
        # the smallest scene (the smoke test's): one call per step and the tool
        # force read after it, as a driver that logs forces does; latency and
        # launches
        _step("first_cut_1600", 20, 10, 8, call="step", forces=True),
        # the small benchmark configuration, 8,000 particles from rest, in the
        # chunks of graph replays a program steps it with
        _step("small_8k", 40, 20, 10, steps=5),
        # five meshed tools in one contact pass (the five-grain arrangement):
        # contact work on a small scene
        _step("five_grains_10k", 24, 44, 10, tool="five_grains", v_tool=3.0e-3),
        # odd lattice, every correction on, developed state with a temperature
        # field: no stencil or conduction work can be left out
        _step("odd_30k_cspm_pse", 47, 31, 21, cspm=1, conduction=2, loaded=1),
        # the unlocked grid (the box is taken from the particles before every
        # step) with two wedges and exhaustive contact, no conduction
        _step("unlocked_58k", 61, 33, 29, tool="two_wedges", algorithm=1, conduction=0, unlocked=1, loaded=1),
        # an ordinary scene: a quarter million particles, heat by Brookshaw,
        # compensated positions, developed
        _step("ordinary_250k", 125, 63, 32, conduction=1, precision=1, loaded=1),
        # the million-particle benchmark configuration from rest
        _step("million_rest", 200, 100, 50, steps=2, cspm=1, conduction=2),
        # the same with compensated positions, well into the cut: every
        # temperature differs, so every conduction term counts
        _step("million_developed", 200, 100, 50, cspm=1, conduction=2, precision=1, loaded=1),
        # the largest configuration: a 1,280-triangle grain with its volume
        # sampled into heat-conducting tool particles
        _step("grain_4m", 400, 160, 64, tool="grain", v_tool=3.0e-3, precision=1),
        # a batch of uneven scenes, one graph replay for all of them
        dict(name="batch_32_mixed", kind="batch", count=32, n_lo=5000, n_hi=200000, specs=1, steps=2),
        # a served request from its host arrays to the fields read back: set-up,
        # admission, steps and read-back with a new context every time
        dict(name="served_request_33k", kind="served", nz=16, v_tool=2.0e-3, depth=5.0, steps=8),
        # the allocation-free cell list, near its particle limit
        dict(name="cell_list_250k", kind="cells", n=249999, nx=81, ny=63, nz=41),
    ]


def _step(name, nx, ny, nz, steps=1, call="advance", forces=False, tool="wedge", algorithm=0, cspm=0, conduction=1,
          precision=0, unlocked=0, loaded=0, v_tool=1.0e-3):
    return dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, steps=steps, call=call, forces=forces, tool=tool,
                algorithm=algorithm, cspm=cspm, conduction=conduction, precision=precision, unlocked=unlocked,
                loaded=loaded, v_tool=v_tool)


def draw(rng):
    """A further case of the same ranges; the lattices keep the generators' proportions within a factor of two."""
    kind = rng.choices(("step", "batch", "served", "cells"), (14, 3, 2, 1))[0]
    if kind == "batch":
        lo = int(10 ** rng.uniform(3.3, 4.3))
        return dict(kind="batch", count=rng.randint(2, 40), n_lo=lo, n_hi=int(lo * 10 ** rng.uniform(0.3, 1.0)),
                    specs=rng.randint(2, 10000), steps=rng.randint(2, 3))
    if kind == "served":
        return dict(kind="served", nz=rng.randint(8, 30), v_tool=rng.uniform(1e-4, 5e-3), depth=rng.uniform(2.0, 6.0),
                    steps=rng.randint(2, 20))
    if kind == "cells":
        n3 = [rng.randint(5, 80) for _ in range(3)]
        return dict(kind="cells", n=int(10 ** rng.uniform(3.0, math.log10(262144))), nx=n3[0], ny=n3[1], nz=n3[2])
    n = 10 ** rng.uniform(3.2, 6.1)
    nz = max(6, round((n / 8.0) ** (1.0 / 3.0) * rng.uniform(0.7, 1.4)))
    ny = max(6, round((n / nz / 2.0) ** 0.5 * rng.uniform(0.7, 1.4)))
    nx = max(12, round(n / nz / ny))
    tool = rng.choices(("wedge", "two_wedges", "five_grains"), (6, 3, 2))[0]
    if tool == "five_grains":  # the grains stand beside one another: a block at least as wide as the leading row
        nx, ny, nz = max(nx, 24), max(ny, 44), max(nz, 8)
    small = nx * ny * nz < 20000
    call = "step" if rng.random() < 0.3 else "advance"
    return dict(kind="step", nx=nx, ny=ny, nz=nz, steps=1 if call == "step" or not small else rng.randint(1, 5),
                call=call, forces=call == "step" and rng.random() < 0.5, tool=tool,
                algorithm=int(rng.random() < 0.25), cspm=rng.randint(0, 1), conduction=rng.choice((0, 1, 1, 2, 2)),
                precision=rng.randint(0, 1), unlocked=int(rng.random() < 0.15), loaded=rng.randint(0, 1),
                v_tool=rng.choice((5e-4, 1e-3, 3e-3)))


# ---------------------------------------------------------- inputs and passes --

# the compact state arrays that run() returns, in the library's order
ARRAYS = ("POS_H", "VEL_RHO", "S_A", "S_B", "POS_T", "VEL_T", "S_T_A", "S_T_B", "FC", "FT")
SERVED_FIELDS = ("POS", "VEL", "S", "T", "EPS_PL", "RHO")


@functools.lru_cache(maxsize=2)
def _geometry(nx, ny, nz, tool, algorithm, cspm, conduction, precision, v_tool):
    """The scene of a case with its lattice as generated; positions are drawn anew per seed."""
    if tool == "grain":
        sc = scenes.single_grain(nx, ny, nz, v_tool=v_tool, precision=precision)
        sc.options.update(cspm=int(cspm), conduction=int(conduction))
    elif tool == "five_grains":
        sc = scenes.five_grain_scene(nx, ny, nz, v_tool=v_tool, precision=precision)
        sc.options.update(cspm=int(cspm), conduction=int(conduction))
        for t in sc.tools:
            t.algorithm = algorithm
    else:
        make = scenes.two_tool_scene if tool == "two_wedges" else scenes.orthogonal_cutting
        sc = make(nx, ny, nz, v_tool=v_tool, cspm=bool(cspm), conduction=conduction, precision=precision,
                  algorithm=algorithm)
    return sc


def _scene(case, seed):
    """The case's scene for one seed: its own lattice jitter and, for a developed state, its own fields."""
    sc = _geometry(*(case[k] for k in ("nx", "ny", "nz", "tool", "algorithm", "cspm", "conduction", "precision",
                                       "v_tool")))
    rng = np.random.default_rng(seed)
    dx, n = 1.0e-3, sc.n
    out = scenes.dataclasses.replace(sc, pos=sc.pos.copy())
    free = sc.tool_p == 0.0
    out.pos[:, :3] += (0.005 * dx) * (rng.random((n, 3), dtype=np.float32) * 2.0 - 1.0) * free[:, None]
    if case["unlocked"]:
        # max_cell bounds the unlocked grid: room for the box to grow
        out.grid_max_cell = int(4 * n + 4096)
    state = None
    if case["loaded"]:
        p = out.pos[:, :3].astype(np.float32)

        def field(amp):  # two plane waves of wavelength ~15-40 dx, random direction and phase
            f = np.zeros(n, np.float32)
            for _ in range(2):
                k = rng.normal(size=3)
                k *= 2.0 * math.pi / (rng.uniform(15.0, 40.0) * dx) / np.linalg.norm(k)
                f += np.sin(p @ k.astype(np.float32) + np.float32(rng.uniform(0.0, 2.0 * math.pi)))
            return (0.5 * amp) * f

        # stresses up to about the yield stress (A = 7.9e-3 Mbar), a few m/s,
        # 300 to 500 K, densities +-0.05 %, plastic strains up to 0.05
        xx, yy, xy, xz, yz = (field(3.0e-3) for _ in range(5))
        out.vel = sc.vel.copy()
        for d in range(3):
            out.vel[:, d] = field(3.0e-4)
        out.rho = (sc.rho * (1.0 + field(5.0e-4))).astype(np.float32)
        out.T = (400.0 + field(100.0)).astype(np.float32)
        eps = np.abs(field(0.05))
        state = dict(S_A=np.stack([xx, yy, -xx - yy, xy], 1).astype(np.float32),
                     S_B=np.stack([xz, yz, out.T, eps], 1).astype(np.float32))
    return out, state


@functools.lru_cache(maxsize=1)
def _stream():
    """One stream for all scenes, so that passes follow one another as the steps of one program do."""
    return torch.cuda.Stream()


class _Device:
    """A float4 array of the library as torch sees foreign device memory; keeps its owner alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n, 4), typestr="<f4", data=(ptr, False), version=2)


def _views(sim, kept, owner):
    """The current state arrays; a program keeps the views of the two copies the steps alternate between."""
    ptr = sim.array_device_ptr("POS_H")
    if ptr not in kept:
        kept[ptr] = {a: torch.as_tensor(_Device(sim.array_device_ptr(a), sim.n_init, owner), device="cuda")
                     for a in ARRAYS}
    return kept[ptr]


def prepare(case, seed):
    if case["kind"] == "step":
        sc, state = _scene(case, seed)
        sim = api.Simulation.from_scene(sc, stream=_stream().cuda_stream)
        for name, values in (state or {}).items():
            sim.set_array(name, values)
        return dict(case=case, sim=sim, kept={})
    if case["kind"] == "batch":
        batch, sims, kept = api.Batch(stream=_stream().cuda_stream), [], []
        for k, spec in enumerate(_specs(case)):
            spec.seed = seed * 1009 + k
            sims.append(api.Simulation.from_scene(scenes.mixed_scene(spec)))
            kept.append({})
            batch.admit(sims[-1])
        return dict(case=case, batch=batch, sims=sims, kept=kept)
    if case["kind"] == "served":
        return dict(case=case, scene=scenes.mixed_scene(_request(case, seed)), batch=api.Batch())
    pos, _ = _points(case, seed)
    cells = case["nx"] * case["ny"] * case["nz"]
    return dict(case=case, pos=torch.from_numpy(pos).cuda(), lo=(ctypes.c_float * 3)(0.0, 0.0, 0.0),
                perm=torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                first=torch.empty(cells + 1, dtype=torch.int32, device="cuda"))


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        sim = state["sim"]
        if case["call"] == "step":
            for _ in range(case["steps"]):
                sim.step(record_forces=case["forces"])
        else:
            sim.advance(case["steps"])
        out = dict(_views(sim, state["kept"], sim))
        if case["forces"]:
            out["forces"] = sim.tool_forces()
        return out
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        # 60 outputs at most are compared: four arrays of every fourth scene
        # (every scene when there are fewer), and all of them have stepped
        views = [_views(s, k, (s, state["batch"])) for s, k in zip(state["sims"], state["kept"])]
        every = max(1, len(views) // 12)
        return [[v[a] for a in ("POS_H", "VEL_RHO", "S_A", "S_T_A")] for v in views[::every][:15]]
    if case["kind"] == "served":
        sim = api.Simulation.from_scene(state["scene"])
        batch = state["batch"]
        slot = batch.admit(sim, case["steps"])
        batch.step(case["steps"])
        out = serve.scene_state(sim, SERVED_FIELDS)
        batch.retire(slot)
        return out
    L, pos, perm, first = api.lib(), state["pos"], state["perm"], state["first"]
    fp = ctypes.POINTER(ctypes.c_float)
    st = L.mfree_cell_list_static(ctypes.cast(pos.data_ptr(), fp), case["n"], state["lo"], 1.0e-3, case["nx"],
                                  case["ny"], case["nz"], perm.data_ptr(), first.data_ptr(),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st != 0:
        raise api.MfreeError(st, L.mfree_last_error().decode())
    return perm, first


def _specs(case):
    return scenes.mixed_specs(case["count"], seed=case["specs"], n_lo=case["n_lo"], n_hi=case["n_hi"])


def _request(case, seed):
    return scenes.MixedSpec(nz=case["nz"], v_tool=case["v_tool"], depth=case["depth"], rake_deg=-5.0,
                            jc_scale=(1.0, 1.05, 0.95), seed=seed)


def _points(case, seed):
    """Particles of a moving cloud in a slightly smaller grid: about one in fifty lies outside."""
    rng = np.random.default_rng(seed)
    n3 = np.array([case["nx"], case["ny"], case["nz"]], np.float32)
    pos = np.zeros((case["n"], 4), np.float32)
    pos[:, :3] = (rng.random((case["n"], 3), dtype=np.float32) * 1.007 * n3) * np.float32(1e-3)
    # a program's particles come roughly in last step's cell order
    c = np.minimum((pos[:, :3] / np.float32(1e-3)).astype(np.int64), n3.astype(np.int64) - 1)
    order = np.argsort((c[:, 0] * case["ny"] + c[:, 1]) * case["nz"] + c[:, 2], kind="stable")
    swap = rng.integers(0, case["n"], size=case["n"] // 10)
    order[swap] = order[swap[::-1]]
    pos = np.ascontiguousarray(pos[order])
    return pos, n3


# ------------------------------------------------------ work and tolerances --

def _particles(case):
    if case["kind"] == "batch":
        return sum(s.n for s in _specs(case))
    if case["kind"] == "served":
        return 8 * case["nz"] ** 3
    n = case["nx"] * case["ny"] * case["nz"]
    return n + 26190 if case["tool"] == "grain" else n  # with the grain's tool particles


def work(case):
    if case["kind"] == "cells":
        cells = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=20.0 * case["n"] + 4.0 * cells, flops=6.0 * case["n"])
    n = _particles(case)
    precision = case.get("precision", 1)
    cspm, conduction = case.get("cspm", 0), case.get("conduction", 1)
    # per particle and step: the state read and written once (the creation
    # index, flags and tool forces move with the sort); per candidate of the
    # 5x5x5 cells (247 on this lattice) the support test and the PSE term, per
    # neighbour in support (77) the pair terms, and the per-particle rest
    per = 352.0 if precision else 304.0
    flops = 247.0 * (14.0 if conduction == 2 else 8.0) + 77.3 * (107.0 + 59.0 * cspm + 10.0 * (conduction == 1)) + 150.0
    extra = n * (52.0 + 4.0 * 18.0) if case["kind"] == "served" else 0.0  # host arrays in, fields out
    return dict(bytes=n * per * case["steps"] + extra, flops=n * flops * case["steps"])


def tolerance(case):
    if case["kind"] == "cells":
        return "exact"
    # Sums taken in another order (8, 16 and 32 lanes a particle) part by up to
    # 3e-7 (largest entry 1e-5) in one step and, where contact feeds them back,
    # by 2e-6 (9e-5) over ten.  A contact force is a gap of about 5e-5 cm
    # between coordinates rounded to 1e-8 cm: one last bit of a position is
    # 2e-4 of its particle's force, and the forces are up to 1e-4 (friction
    # 3e-4, largest entry 8e-3) from exact().
    one = case["kind"] == "step" and case["steps"] == 1
    return dict(rel=4e-5, max=4e-3) if one else dict(rel=1e-4, max=1e-2)


# ------------------------------------------------------------- FP64 restatement --

F64 = torch.float64


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "cells":
        pos, n3 = _points(case, seed)
        c = (torch.from_numpy(pos).to(dev)[:, :3] / torch.tensor(1e-3, dtype=torch.float32, device=dev)).to(torch.int64)
        top = torch.tensor([case["nx"], case["ny"], case["nz"]], device=dev)
        key = (c[:, 0] * top[1] + c[:, 1]) * top[2] + c[:, 2]
        cells = int(top.prod())
        key = torch.where((c < top).all(1), key, cells)
        perm = torch.argsort(key, stable=True)
        first = torch.zeros(cells + 2, dtype=torch.int64, device=dev)
        first[1:] = torch.cumsum(torch.bincount(key, minlength=cells + 1), 0)
        return perm.to(torch.int32), first[: cells + 1].to(torch.int32)
    if case["kind"] == "batch":
        specs = _specs(case)
        if sum(s.n for s in specs) * case["steps"] > 4_000_000:
            return None
        every = max(1, len(specs) // 12)
        out = []
        for k, spec in list(enumerate(specs))[::every][:15]:
            spec.seed = seed * 1009 + k
            m = _Step64(scenes.mixed_scene(spec), None, dev)
            for _ in range(case["steps"]):
                m.step()
            a = m.arrays()
            out.append([a[x] for x in ("POS_H", "VEL_RHO", "S_A", "S_T_A")])
        return out
    if case["kind"] == "served":
        m = _Step64(scenes.mixed_scene(_request(case, seed)), None, dev)
        for _ in range(case["steps"]):
            m.step()
        return m.fields_by_id()
    if case["tool"] in ("grain", "five_grains") or _particles(case) * case["steps"] > 2_500_000:
        return None
    sc, state = _scene(case, seed)
    m = _Step64(sc, state, dev)
    for _ in range(case["steps"]):
        m.step()
    out = dict(m.arrays())
    if case["forces"]:
        out["forces"] = m.forces.cpu().numpy()
    return out


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _Tool64:
    """A closed convex triangle tool: features with inward normals, closest point and inside test."""

    def __init__(self, t, dev):
        v = torch.from_numpy(np.asarray(t.verts, np.float32)).to(dev, F64)
        tri = torch.from_numpy(np.asarray(t.tris, np.int64)).to(dev)
        self.tri, self.v = tri, v
        p = v[tri]
        n = _unit(torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]))
        # inward: the mesh is convex, its centroid lies on the inner side of every face
        if float(_dot(n, v.mean(0) - p[:, 0]).sum()) < 0.0:
            n = -n
        edges, verts = {}, {}
        T = tri.tolist()
        for i, f in enumerate(T):
            for a, b in ((0, 1), (1, 2), (2, 0)):
                edges.setdefault(frozenset((f[a], f[b])), []).append(i)
            for q in range(3):
                a, b = (v[f[k]] - v[f[q]] for k in range(3) if k != q)
                ang = torch.acos((_dot(a, b) / (a.norm() * b.norm())).abs())
                verts[f[q]] = verts.get(f[q], 0.0) + ang * n[i]
        # feature normals per triangle: face, three vertices, three edges 12, 23, 31
        self.normals = torch.stack([torch.stack(
            [n[i]] + [_unit(verts[q]) for q in f] +
            [_unit(sum(n[j] for j in edges[frozenset((f[a], f[b]))])) for a, b in ((0, 1), (1, 2), (2, 0))])
            for i, f in enumerate(T)])
        self.vel = torch.from_numpy(np.asarray(t.vel, np.float32)).to(dev, F64)
        self.alpha, self.mu = float(np.float32(t.contact_alpha)), float(np.float32(t.mu))
        self.hashed = t.algorithm == 0
        self.lo, self.hi = v.min(0).values - 1e-4, v.max(0).values + 1e-4

    def contact(self, q, time, moved):
        """Of points q: which are in contact, their closest surface points and those features' normals."""
        in_box = ((q > self.lo + moved * self.vel) & (q < self.hi + moved * self.vel)).all(1)
        p = (self.v + self.vel * time)[self.tri]
        v1, v2, v3 = (p[None, :, k] for k in range(3))
        qq = q[:, None]
        ea, eb, w = v2 - v1, v3 - v1, v1 - qq
        ab, aa, bb = _dot(ea, eb), _dot(ea, ea), _dot(eb, eb)
        den = ab * ab - aa * bb
        sa = (_dot(ea, w) * bb - _dot(eb, w) * ab) / den
        sb = (_dot(eb, w) * aa - _dot(ea, w) * ab) / den

        def segment(a, b, ia, ib, ie):
            s = (_dot(b - a, qq - a) / _dot(b - a, b - a)).clamp(0.0, 1.0)
            f = torch.where(s <= 0.0, ia, torch.where(s >= 1.0, ib, ie))
            return a + s[..., None] * (b - a), f

        cp = v1 + sa[..., None] * ea + sb[..., None] * eb
        feat = torch.zeros(cp.shape[:2], dtype=torch.int64, device=q.device)
        for cond, (c, f) in ((sa + sb > 1.0, segment(v2, v3, 2, 3, 5)), (sb < 0.0, segment(v1, v2, 1, 2, 4)),
                             (sa < 0.0, segment(v1, v3, 1, 3, 6))):  # the last one that holds decides
            cp = torch.where(cond[..., None], c, cp)
            feat = torch.where(cond, f, feat)
        k = ((cp - qq) ** 2).sum(-1).argmin(1)
        r = torch.arange(len(q), device=q.device)
        cp, n = cp[r, k], self.normals[k, feat[r, k]]
        if self.hashed:  # inside by the parity of the hits of a +z ray
            h = torch.stack([-eb[..., 1], eb[..., 0], torch.zeros_like(eb[..., 0])], -1)
            a = _dot(ea, h)
            s = qq - v1
            u = _dot(s, h) / a
            c = torch.linalg.cross(s, ea.expand_as(s))
            vv = c[..., 2] / a
            hit = (a.abs() > 1e-30) & (u >= 0.0) & (u <= 1.0) & (vv >= 0.0) & (u + vv <= 1.0) & (_dot(eb, c) / a > 1e-7)
            return in_box & (hit.sum(1) % 2 == 1), cp, n
        return in_box & (_dot(cp - q, n) <= 0.0), cp, n


class _Step64:
    """One cutting scene stepped in FP64: cell sort, predictor, pair sums, rates, corrector, plasticity, contact."""

    def __init__(self, sc, state, dev):
        f = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(dev, F64)  # noqa: E731
        g = lambda d: {k: float(np.float32(v)) for k, v in d.items()}  # noqa: E731
        n = sc.n
        self.sc, self.dev, self.n = sc, dev, n
        z3, z6 = torch.zeros(n, 3, dtype=F64, device=dev), torch.zeros(n, 6, dtype=F64, device=dev)
        s6, eps = z6, z6[:, 0]
        if state is not None:
            a, b = f(state["S_A"]), f(state["S_B"])
            s6, eps = torch.cat([a, b[:, :2]], 1), b[:, 3]
        self.s = dict(x=f(sc.pos)[:, :3], h=f(sc.h), v=f(sc.vel)[:, :3], rho=f(sc.rho), S=s6, T=f(sc.T), eps=eps,
                      xd=z3, rd=z6[:, 0], vd=z3, Td=z6[:, 0], Sd=z6, epsd=z6[:, 0], fixed=f(sc.fixed), fc=z3, ft=z3,
                      id=torch.arange(n, device=dev))
        self.ph, self.co, self.jc = g(sc.phys), g(sc.corr), g(sc.joco) if sc.joco else None
        self.wp = g(sc.trml_wp)
        self.cond, self.cspm = int(sc.options["conduction"]), bool(sc.options["cspm"])
        self.dt = float(np.float32(sc.dt))
        self.t = np.float32(0) + np.float32(sc.dt)
        self.moved = 0.0
        self.tools = [_Tool64(t, dev) for t in sc.tools]
        self.forces = torch.zeros(len(self.tools), 3, dtype=F64, device=dev)

    def sort(self):
        s, sc = self.s, self.sc
        x = s["x"].to(torch.float32)
        f32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.float32, device=self.dev)  # noqa: E731
        if sc.grid_max_cell > 0:
            lo, hi, dx = x.min(0).values.cpu().numpy(), x.max(0).values.cpu().numpy(), np.float32(s["h"].max().item())
        else:
            lo, hi, dx = np.float32(sc.grid_bbmin), np.float32(sc.grid_bbmax), np.float32(sc.grid_h)
        lo, hi = (np.float32(np.float64(a) + e) for a, e in ((lo, -1e-6), (hi, 1e-6)))
        n3 = [int(math.ceil(np.float32(hi[d] - lo[d]) / dx)) for d in range(3)]
        c = ((x - f32(lo)) / f32(dx)).to(torch.int64)
        key = (c[:, 0] * n3[1] + c[:, 1]) * n3[2] + c[:, 2]
        order = torch.argsort(key, stable=True)
        self.s = {k: v[order] for k, v in s.items()}
        first = torch.zeros(n3[0] * n3[1] * n3[2] + 1, dtype=torch.int64, device=self.dev)
        first[1:] = torch.cumsum(torch.bincount(key, minlength=len(first) - 1), 0)
        return c[order], n3, first

    def candidates(self, c, n3, first, i0, i1):
        """Pairs (i, j) of particles i in [i0, i1) with everything in their 5 x 5 x 5 cells."""
        ci = c[i0:i1]
        off = torch.arange(25, device=self.dev)
        cx, cy = ci[:, :1] + off[None] // 5 - 2, ci[:, 1:2] + off[None] % 5 - 2
        ok = (cx >= 0) & (cx < n3[0]) & (cy >= 0) & (cy < n3[1])
        base = (cx.clamp(0, n3[0] - 1) * n3[1] + cy.clamp(0, n3[1] - 1)) * n3[2]
        a = first[base + (ci[:, 2:] - 2).clamp(min=0)]
        b = first[base + (ci[:, 2:] + 2).clamp(max=n3[2] - 1) + 1]
        ln = torch.where(ok, b - a, 0).reshape(-1)
        row = torch.repeat_interleave(torch.arange(len(ln), device=self.dev), ln)
        start = torch.cumsum(ln, 0) - ln
        j = a.reshape(-1)[row] + torch.arange(len(row), device=self.dev) - start[row]
        return i0 + row // 25, j

    def step(self):
        c, n3, first = self.sort()
        s, ph, co, dt = self.s, self.ph, self.co, self.dt
        n, dev = self.n, self.dev
        hd = 0.5 * dt
        x, v, rho, T = s["x"] + hd * s["xd"], s["v"] + hd * s["vd"], s["rho"] + hd * s["rd"], s["T"] + hd * s["Td"]
        S = s["S"] + hd * s["Sd"]
        p = (ph["K"] / ph["rho0"]) * (rho - ph["rho0"])
        R = _artificial_stress(S, p, rho, co["stresseps"])
        diag = torch.tensor([1.0, 1.0, 1.0, 0.0, 0.0, 0.0], dtype=F64, device=dev)
        sig = (S - p[:, None] * diag) / (rho * rho)[:, None]
        snd, vol, h = torch.sqrt(ph["K"] / rho), ph["mass"] / rho, s["h"]
        L = torch.zeros(n, 9, dtype=F64, device=dev)
        acc = torch.zeros(n, 9, dtype=F64, device=dev)  # stress divergence, viscosity, XSPH
        heat = torch.zeros(n, dtype=F64, device=dev)
        full = lambda m: m[:, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(-1, 3, 3)  # noqa: E731
        chunk = 65536 if dev == "cuda" else 4096
        for i0 in range(0, n, chunk):
            i1 = min(n, i0 + chunk)
            i, j = self.candidates(c, n3, first, i0, i1)
            d = x[i] - x[j]
            r2 = (d * d).sum(1)
            m = i1 - i0
            if self.cond == 2:
                heat[i0:i1].index_add_(0, i - i0, (T[j] - T[i]) * vol[j] * torch.exp(-r2 / (h[i] * h[i])))
            keep = (r2 < 4.0 * h[i] * h[i]) & (r2 >= 1e-8)
            i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
            r = torch.sqrt(r2)
            q = r / h[i]
            fac = 1.0 / (math.pi * h[i] ** 3)
            far = q > 1.0
            w = fac * torch.where(far, 0.25 * (2.0 - q) ** 3, 1.0 - 1.5 * q * q * (1.0 - 0.5 * q))
            dw = fac * torch.where(far, -0.75 * (2.0 - q) ** 2, -3.0 * q * (1.0 - 0.75 * q)) / (h[i] * r)
            g = dw[:, None] * d
            at = i - i0
            if self.cspm:
                B = torch.zeros(m, 9, dtype=F64, device=dev)
                B.index_add_(0, at, -((vol[j] * dw)[:, None, None] * d[:, :, None] * d[:, None, :]).reshape(-1, 9))
                B = B.reshape(-1, 3, 3)
                good = torch.linalg.det(B) > 1e-8
                eye = torch.eye(3, dtype=F64, device=dev)
                inv = torch.where(good[:, None, None], torch.linalg.inv(torch.where(good[:, None, None], B, eye)), eye)
                g = (inv[at] @ g[:, :, None])[:, :, 0]
            dv = v[j] - v[i]
            L[i0:i1].index_add_(0, at, ((vol[j][:, None] * dv)[:, :, None] * g[:, None, :]).reshape(-1, 9))
            t6 = sig[i] + sig[j]
            if co["wdeltap"] > 0.0:
                t6 = t6 + ((w / co["wdeltap"]) ** 4)[:, None] * (R[i] + R[j])
            div = (full(t6) @ g[:, :, None])[:, :, 0]
            vr = -_dot(dv, d)
            rij, cij, hij = 0.5 * (rho[i] + rho[j]), 0.5 * (snd[i] + snd[j]), 0.5 * (h[i] + h[j])
            mu = torch.where(vr < 0.0, hij * vr / (r2 + co["eta"] ** 2 * hij * hij), 0.0)
            pij = (-co["alpha"] * cij * mu + co["beta"] * mu * mu) / rij
            acc[i0:i1].index_add_(0, at, torch.cat([div, -pij[:, None] * g, -(w / rij)[:, None] * dv], 1))
            if self.cond == 1:
                heat[i0:i1].index_add_(0, at, vol[j] * (T[i] - T[j]) * _dot(d, g) / r2)
        # rates
        G, mass = ph["G"], ph["mass"]
        Lm = L.reshape(-1, 3, 3)
        e, w = 0.5 * (Lm + Lm.transpose(1, 2)), 0.5 * (Lm - Lm.transpose(1, 2))
        tr = torch.diagonal(e, dim1=1, dim2=2).sum(1)
        Sm = full(S)
        rate = 2.0 * G * (e - (tr / 3.0)[:, None, None] * torch.eye(3, dtype=F64, device=dev)) + w @ Sm + Sm @ w.transpose(1, 2)
        Sd = rate.reshape(-1, 9)[:, [0, 4, 8, 1, 2, 5]]
        rd = -rho * tr
        vd = mass * (acc[:, 3:6] + acc[:, :3]) + (s["fc"] + s["ft"]) / mass
        xd = v - co["xspheps"] * mass * acc[:, 6:9]
        Td = s["Td"]
        if self.cond == 1:
            Td = self.wp["alpha"] * 2.0 * heat
        elif self.cond == 2:
            Td = self.wp["alpha"] * 4.0 / (h ** 5 * math.pi ** 1.5) * heat
        # corrector
        x1, v1, S1 = s["x"] + dt * xd, s["v"] + dt * vd, s["S"] + dt * Sd
        rho1, T1, eps, epsd = s["rho"] + dt * rd, s["T"] + dt * Td, s["eps"], s["epsd"]
        if self.jc:
            S1, T1, eps, epsd = self.plasticity(S1, T1, rho1, eps, epsd)
        # contact at the new positions, friction heat, boundary conditions
        fc, ft = torch.zeros_like(x1), torch.zeros_like(x1)
        nl = torch.zeros_like(x1)
        self.moved += dt
        cand = torch.zeros(n, dtype=torch.bool, device=dev)
        for k, tool in enumerate(self.tools):
            lo, hi = tool.lo + self.moved * tool.vel, tool.hi + self.moved * tool.vel
            idx = ((x1 > lo) & (x1 < hi)).all(1).nonzero()[:, 0]
            self.forces[k] = 0.0
            if not len(idx):
                continue
            cand[idx] = True
            hit, cp, nr = tool.contact(x1[idx], float(self.t), self.moved)
            idx, cp, nr = idx[hit], cp[hit], nr[hit]
            gn = _dot(x1[idx] - cp, nr)
            fn = (-mass * gn / (dt * dt) * tool.alpha)[:, None] * nr
            fr = torch.zeros_like(fn)
            if tool.mu != 0.0:
                vr = v1[idx] * (1.0 - nr)
                fs = ft[idx] - (tool.alpha * mass / dt) * vr
                fy, lf = tool.mu * fn.norm(dim=1), fs.norm(dim=1)
                fr = torch.where((lf > fy)[:, None], (fy / lf.clamp(min=1e-300))[:, None] * fs, fs)
            fc[idx], ft[idx], nl[idx] = fn, fr, nr
            self.forces[k] = (fn + fr).sum(0)
        if self.wp["eta"] != 0.0 and self.tools:
            dvt = v1 - self.tools[0].vel
            rv = dvt - _dot(dvt, nl)[:, None]
            T1 = T1 + torch.where(cand, self.wp["eta"] * dt * ft.norm(dim=1) * rv.norm(dim=1) / (self.wp["cp"] * mass), 0.0)
        fx = (s["fixed"] != 0.0)
        z = torch.zeros((), dtype=F64, device=dev)
        v1, xd, vd, fc = (torch.where(fx[:, None], z, a) for a in (v1, xd, vd, fc))
        if self.wp["alpha"] != 0.0:
            T1 = torch.where(s["fixed"] == 1.0, torch.full_like(T1, self.wp["T_init"]), T1)
        s.update(x=x1, v=v1, S=S1, rho=rho1, T=T1, eps=eps, epsd=epsd, xd=xd, vd=vd, Sd=Sd, rd=rd, Td=Td, fc=fc, ft=ft)
        self.t = self.t + np.float32(self.sc.dt)

    def plasticity(self, S, T, rho, eps, epsd):
        """Johnson-Cook radial return: the secant iteration on the plastic multiplier, for the yielding particles."""
        j, dt, G = self.jc, self.dt, self.ph["G"]
        Tc = torch.where(T > j["Tmelt"], j["Tmelt"] - 1.0, T) if j["clamp_temp"] else T
        norm = torch.sqrt((S[:, :3] ** 2).sum(1) + 2.0 * (S[:, 3:] ** 2).sum(1))

        def flow(e, ed, T):
            ed = ed / j["eps_dot_ref"]
            b = torch.where(ed > 1.0, 1.0 + j["C"] * torch.log(ed.clamp(min=1.0)), (1.0 + ed) ** j["C"])
            return (j["A"] + j["B"] * e ** j["n"]) * b * (1.0 - ((T - j["Tref"]) / (j["Tmelt"] - j["Tref"])) ** j["m"])

        s23 = math.sqrt(2.0 / 3.0)
        idx = (math.sqrt(1.5) * norm >= flow(eps, epsd, Tc)).nonzero()[:, 0]
        new = torch.zeros_like(epsd)
        if not len(idx):
            return S, T, eps, new
        nS, e0, Ti = norm[idx], eps[idx], Tc[idx]
        opt = lambda dl: nS - 2.0 * G * dl - s23 * flow(e0 + s23 * dl.clamp(min=0.0), s23 * dl.clamp(min=0.0) / dt, Ti)  # noqa: E731
        dl = (epsd[idx] * dt * s23).clamp(min=1e-8)
        live = torch.ones_like(dl, dtype=torch.bool)
        for _ in range(102):
            g, g1 = opt(dl), opt(dl * 1.01)
            nx = dl - g / ((g - g1) / (dl - dl * 1.01))
            nx = torch.where(nx < 0.0, -0.1 * nx, nx)
            stop = (nx - dl).abs() < 1e-6
            dl = torch.where(live, nx, dl)
            live = live & ~stop
            if not bool(live.any()):
                break
        pl = dl.clamp(min=0.0)
        e1, ed1 = e0 + s23 * pl, s23 * pl / dt
        S, T, eps = S.clone(), T.clone(), eps.clone()
        S[idx] = S[idx] - S[idx] / nS[:, None] * dl[:, None] * 2.0 * G
        T[idx] = T[idx] + self.wp["tq"] / (self.wp["cp"] * rho[idx]) * (e1 - e0) * flow(e1, ed1, Ti)
        eps[idx] = e1
        new[idx] = ed1
        return S, T, eps, new

    def arrays(self):
        s = self.s
        col = lambda *a: torch.cat([b if b.dim() == 2 else b[:, None] for b in a], 1)  # noqa: E731
        z = torch.zeros(self.n, dtype=F64, device=self.dev)
        return dict(POS_H=col(s["x"], s["h"]), VEL_RHO=col(s["v"], s["rho"]), S_A=s["S"][:, :4].contiguous(),
                    S_B=col(s["S"][:, 4:], s["T"], s["eps"]), POS_T=col(s["xd"], s["rd"]),
                    VEL_T=col(s["vd"], s["Td"]), S_T_A=s["Sd"][:, :4].contiguous(),
                    S_T_B=col(s["Sd"][:, 4:], s["epsd"], s["fixed"]), FC=col(s["fc"], z), FT=col(s["ft"], z))

    def fields_by_id(self):
        s, back = self.s, torch.argsort(self.s["id"])
        z = torch.zeros(self.n, 1, dtype=F64, device=self.dev)
        out = dict(POS=torch.cat([s["x"], z], 1), VEL=torch.cat([s["v"], z], 1),
                   S=s["S"][:, [0, 3, 4, 3, 1, 5, 4, 5, 2]], T=s["T"], EPS_PL=s["eps"], RHO=s["rho"])
        return {k: v[back].cpu().numpy() for k, v in out.items()}


def _artificial_stress(S, p, rho, eps):
    """Monaghan's artificial stress from the principal stresses.

    The method rotates with the eigenvectors as rows, so the result depends on
    how the eigenvectors are oriented: they are built here by the same closed
    form (Eberly's robust 3 x 3 solver), eigenvalues ascending."""
    a00, a11, a22 = S[:, 0] - p, S[:, 1] - p, S[:, 2] - p
    a01, a02, a12 = S[:, 3], S[:, 4], S[:, 5]
    big = torch.stack([a00, a01, a02, a11, a12, a22], 1).abs().max(1).values
    tiny = big < 1e-8
    k = 1.0 / torch.where(tiny, torch.ones_like(big), big)
    a00, a01, a02, a11, a12, a22 = (a * k for a in (a00, a01, a02, a11, a12, a22))
    off = a01 * a01 + a02 * a02 + a12 * a12
    q = (a00 + a11 + a22) / 3.0
    b00, b11, b22 = a00 - q, a11 - q, a22 - q
    pp = torch.sqrt((b00 ** 2 + b11 ** 2 + b22 ** 2 + 2.0 * off) / 6.0)
    det = (b00 * (b11 * b22 - a12 * a12) - a01 * (a01 * b22 - a12 * a02) + a02 * (a01 * a12 - b11 * a02)) / pp.clamp(min=1e-300) ** 3
    half = (0.5 * det).clamp(-1.0, 1.0)
    ang = torch.acos(half) / 3.0
    e2, e0 = 2.0 * torch.cos(ang), 2.0 * torch.cos(ang + 2.0 * math.pi / 3.0)
    l0, l1, l2 = q + pp * e0, q - pp * (e0 + e2), q + pp * e2
    up = half >= 0.0
    ev = torch.where(up, l2, l0)
    r = [torch.stack(t, 1) for t in ((a00 - ev, a01, a02), (a01, a11 - ev, a12), (a02, a12, a22 - ev))]
    cr = torch.stack([torch.linalg.cross(r[0], r[1]), torch.linalg.cross(r[0], r[2]), torch.linalg.cross(r[1], r[2])], 1)
    d = (cr * cr).sum(2)
    w = cr[torch.arange(len(d), device=d.device), d.argmax(1)] / torch.sqrt(d.max(1).values.clamp(min=1e-300))[:, None]
    zero = torch.zeros_like(w[:, 0])
    wide = w[:, 0].abs() > w[:, 1].abs()
    U = torch.where(wide[:, None], torch.stack([-w[:, 2], zero, w[:, 0]], 1), torch.stack([zero, w[:, 2], -w[:, 1]], 1))
    U = U / U.norm(dim=1, keepdim=True).clamp(min=1e-300)
    V = torch.linalg.cross(w, U)
    mul = lambda y: torch.stack([a00 * y[:, 0] + a01 * y[:, 1] + a02 * y[:, 2],  # noqa: E731
                                 a01 * y[:, 0] + a11 * y[:, 1] + a12 * y[:, 2],
                                 a02 * y[:, 0] + a12 * y[:, 1] + a22 * y[:, 2]], 1)
    AU, AV = mul(U), mul(V)
    m00, m01, m11 = _dot(U, AU) - l1, _dot(U, AV), _dot(V, AV) - l1

    def pair(m, o):  # (larger entry normalised): coefficients of the two basis vectors
        small = m.abs() >= o.abs()
        t1 = o / torch.where(m == 0.0, torch.ones_like(m), m)
        c1 = 1.0 / torch.sqrt(1.0 + t1 * t1)
        t2 = m / torch.where(o == 0.0, torch.ones_like(o), o)
        c2 = 1.0 / torch.sqrt(1.0 + t2 * t2)
        return torch.where(small, c1, t2 * c2), torch.where(small, t1 * c1, c2)

    mm, mo = pair(m00, m01)
    first = mo[:, None] * U - mm[:, None] * V
    first = torch.where((torch.maximum(m00.abs(), m01.abs()) > 0.0)[:, None], first, U)
    nm, no = pair(m11, m01)
    second = nm[:, None] * U - no[:, None] * V
    second = torch.where((torch.maximum(m11.abs(), m01.abs()) > 0.0)[:, None], second, U)
    mid = torch.where((m00.abs() >= m11.abs())[:, None], first, second)
    third = torch.where(up[:, None], torch.linalg.cross(mid, w), torch.linalg.cross(w, mid))
    E = torch.stack([torch.where(up[:, None], third, w), mid, torch.where(up[:, None], w, third)], 1)
    lam = torch.stack([l0, l1, l2], 1)
    plain = off <= 0.0
    lam = torch.where(plain[:, None], torch.stack([a00, a11, a22], 1), lam)
    E = torch.where(plain[:, None, None], torch.eye(3, dtype=F64, device=S.device), E)
    lam = torch.where(tiny[:, None], torch.zeros_like(lam), lam * big[:, None])
    lam = torch.where(lam > 0.0, -eps * lam / (rho * rho)[:, None], torch.zeros_like(lam))
    M = E @ torch.diag_embed(lam) @ E.transpose(1, 2)
    return M.reshape(-1, 9)[:, [0, 4, 8, 1, 2, 5]]
