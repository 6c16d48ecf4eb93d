"""The contact kernel's groups of lanes and its bitmap of contact particles.

A particle in a tool box is served by 2, 8 or 32 lanes, chosen by how many of
them a block holds and by the triangles of the tools; the closest triangle must
be the one a serial search keeps.  Scenes with few and with many particles in
contact, tools on both sides of the triangle limit, both algorithms and particle
counts that do not fill the bitmap's last word are stepped beside the FP32
oracle, which takes the same inside decisions: the first contact forces of
every tool agree to FP32 rounding of the gaps they come from (a last bit of a
coordinate of 0.04 cm, 4e-9, in a gap of 5e-5 cm: 1e-4 of a force).  The same
kernel moves the tool particles of the blanked tail with their tool."""
import numpy as np
import pytest

import oracle
from iwf_mfree_gpu_3d_b200 import api, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "few_in_contact": lambda: scenes.orthogonal_cutting(9, 5, 7, depth=2.0),          # 315 particles, n % 32 != 0
    "block_full_of_contact": lambda: scenes.orthogonal_cutting(21, 17, 11, depth=8.0, engage=0.9),
    "two_tools_exhaustive": lambda: scenes.two_tool_scene(21, 16, 9, engage=(0.6, 0.9), algorithm=1),
    "grain_mesh": lambda: scenes.single_grain(22, 18, 9, depth=4.0, radius=6.0, precision=0, engage=0.8),
    "grain_mesh_exhaustive": lambda: _exhaustive(scenes.single_grain(22, 18, 9, depth=4.0, radius=6.0, precision=0)),
}


def _exhaustive(sc):
    for t in sc.tools:
        t.algorithm = 1
    return sc


@pytest.mark.parametrize("name", sorted(SCENES))
def test_first_contact_forces_match_the_oracle(name):
    sc = SCENES[name]()
    sim = api.Simulation.from_scene(sc)
    orc = oracle.Oracle(sc, prec=32)
    sim.step(record_forces=True)
    orc.step(True)
    ids, io = sim.get("ID"), orc.field("ID").astype(int)
    for f, tol in (("FC", 2e-4), ("FT", 2e-3)):
        g, o = np.empty((sc.n, 3)), np.empty((sc.n, 3))
        g[ids], o[io] = sim.get(f), orc.field(f)
        assert ((g != 0).any(1) == (o != 0).any(1)).all(), f  # the same particles
        assert np.linalg.norm(g - o) <= tol * np.linalg.norm(o), f
    fg, fo = sim.tool_forces(), np.asarray(orc.tool_forces()).reshape(-1, 3)
    # the same contributions in another order: n additions of FP32
    assert np.abs(fg - fo).max() <= 2e-4 * np.abs(fo).max()
    assert np.abs(fo).max() > 0.0
    sim.close()


def test_contact_marks_do_not_outlive_their_step():
    # the tool is taken away (its life ends): particles marked while it was there must not be taken again
    sc = scenes.orthogonal_cutting(21, 17, 11, depth=8.0, engage=0.9)
    sim = api.Simulation.from_scene(sc)
    sim.advance(3, record_every=1)
    assert np.abs(sim.get("FC")).max() > 0.0
    sim.L.mfree_tool_set_birth_death(sim.h, 0, -1.0, -0.5)
    sim.advance(2, record_every=1)
    assert np.abs(sim.get("FC")).max() == 0.0 and np.abs(sim.tool_forces()).max() == 0.0
    sim.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_blanked_tool_particles_move_with_the_tool(precision):
    sc = scenes.single_grain(22, 18, 9, depth=4.0, radius=6.0, precision=precision, engage=0.8)
    tool = sc.tool_p == 1
    x = sc.pos[:, 0]
    sc.blank_bbmax = sc.blank_bbmax.copy()
    sc.blank_bbmax[0] = np.median(x[tool])  # half of them are blanked
    sim = api.Simulation.from_scene(sc)
    sim.advance(4)
    ids = sim.get("ID")
    moved, blanked = np.empty((sc.n, 3)), np.empty(sc.n)
    moved[ids] = (sim.get64("POS") if precision else sim.get("POS"))[:, :3]
    blanked[ids] = sim.get("BLANKED")
    sim.close()
    tail = tool & (blanked == 1)
    assert tail.sum() > 300 and (tool & (blanked == 0)).sum() > 300
    p, v = sc.pos[tail, :3], np.float32(sc.tools[0].vel)
    if precision:
        want = p.astype(np.float64) + 4.0 * v.astype(np.float64) * float(np.float32(sc.dt))
        # high and low parts hold 48 bits; a step moves a particle by 1e-6
        np.testing.assert_allclose(moved[tail], want, rtol=0.0, atol=1e-12)
    else:
        for _ in range(4):  # fmaf(v, dt, p)
            p = (p.astype(np.float64) + v.astype(np.float64) * float(np.float32(sc.dt))).astype(np.float32)
        np.testing.assert_array_equal(moved[tail].astype(np.float32), p)
