"""The pair kernel's tiles: where the grid is cut must not show in the results.

A target's candidates are shared between its two lanes by the parity of their
sorted index, and its sums are joined in a fixed order, so they are the same
bits for every tile depth, for tiles that hold more targets than a block
serves at once, for halos read from global memory instead of shared memory and
for neighbour queues that overflow -- and the same in a batch, whose tiles are
sized by the particles of all its scenes.
"""
import numpy as np
import pytest

import oracle
from iwf_mfree_gpu_3d_b200 import api, scenes

from helpers import compare, gpu_state, loaded, oracle_state

pytestmark = pytest.mark.gpu

NAMES = ("POS", "VEL", "S", "T", "EPS_PL", "RHO", "POS_T", "VEL_T", "S_T", "T_T", "FC", "NUM_NBH", "ID")


def _state(sc, steps, **opt):
    sim = api.Simulation.from_scene(sc, diagnostics=1, **opt)
    if hasattr(sc, "S0"):
        sim.set("S", sc.S0)
    sim.advance(steps, record_every=1)
    out = {n: sim.get(n) for n in NAMES}
    out["forces"] = sim.tool_forces()
    c = sim.counters()
    assert c["staging_timeouts"] == 0 and c["bounds_errors"] == 0
    sim.close()
    return out


def _same(a, b, what):
    for n in a:
        np.testing.assert_array_equal(a[n], b[n], err_msg=f"{what}: {n}")


def _dense(sc, f):
    """The scene's particles drawn together by f in y: more neighbours than a
    queue holds and, at the smaller f, halos beyond the staging area."""
    sc.pos[:, 1] *= np.float32(f)
    return sc


CASES = {
    # one cell column and ragged edges: tiles of a few targets
    "ragged": lambda: scenes.orthogonal_cutting(29, 7, 5, conduction=0),
    "cspm_pse": lambda: loaded(scenes.orthogonal_cutting(23, 17, 13, cspm=True, conduction=2)),
    "cspm_brookshaw": lambda: loaded(scenes.orthogonal_cutting(23, 17, 13, cspm=True, conduction=1, precision=1)),
    "overflow": lambda: _dense(scenes.orthogonal_cutting(26, 20, 12, conduction=1), 0.6),
    "from_global": lambda: _dense(scenes.orthogonal_cutting(26, 40, 12, cspm=True, conduction=2), 0.2),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_results_do_not_depend_on_the_tiles(case):
    ref = _state(CASES[case](), 3)
    if case in ("overflow", "from_global"):
        assert ref["NUM_NBH"].max() > 96  # beyond a queue's capacity
    for depth in (1, 2, 5, 7):
        _same(ref, _state(CASES[case](), 3, tile_depth=depth), f"{case}, depth {depth}")


def test_tall_grids_against_the_oracle():
    # bundles of more levels than one warp cuts: every level must be in a tile
    for dims in ((4, 5, 400), (9, 3, 170)):
        sc = loaded(scenes.orthogonal_cutting(*dims, cspm=True, conduction=1))
        sim = api.Simulation.from_scene(sc, diagnostics=1)
        assert sim.grid()[0][2] > 128
        orc = oracle.Oracle(sc, prec=32)
        sim.step()
        orc.step()
        assert sim.get("NUM_NBH").min() > 0
        err = compare(gpu_state(sim), oracle_state(orc), sc)
        sim.close()
        assert err["blank_mismatch"] == 0
        for k in ("POS", "VEL", "RHO", "VEL_T", "POS_T", "RHO_T", "S_T"):
            assert err[k] < 2e-5, (dims, k, err)


def test_tall_and_long_blocks_take_about_as_long():
    # the same block lying and standing (it stood 2.2 times as long while one
    # warp cut all the tiles above one another)
    def ms(*dims):
        sim = api.Simulation.from_scene(scenes.orthogonal_cutting(*dims))
        sim.advance(3)
        sim.sync()
        t = []
        for _ in range(3):
            sim.timer_start()
            sim.advance(20)
            t.append(sim.timer_stop() / 20)
        sim.close()
        return min(t)

    tall, long = ms(4, 4, 2000), ms(2000, 4, 4)
    assert tall < 1.7 * long, (tall, long)


def test_results_do_not_depend_on_the_batch_around_a_scene():
    # alone its tiles hold 32 targets at most; beside the larger scene they are fuller
    small = lambda: scenes.orthogonal_cutting(18, 9, 7, precision=1)  # noqa: E731
    big = scenes.orthogonal_cutting(80, 40, 20, precision=1)
    b = api.Batch()
    sims = [api.Simulation.from_scene(sc) for sc in (small(), big)]
    for s in sims:
        b.admit(s)
    b.step(4, record_every=1)
    ref = api.Simulation.from_scene(small())
    ref.advance(4, record_every=1)
    for n in ("POS", "VEL", "S", "T", "VEL_T", "ID"):
        np.testing.assert_array_equal(sims[0].get(n), ref.get(n), err_msg=n)
    ref.close()
    b.close()


def test_batch_of_dense_scenes_in_tight_boxes():
    # h = 1.7 dx and boxes half a spacing around the particles: 84 particles a
    # level of a bundle, where the halo cuts tiles to one level each -- 1,142
    # tiles, of which the depth limit and the target count alone would explain
    # 1,034 at most.  The batch's list must hold them all.
    def scene(*dims):
        sc = scenes.orthogonal_cutting(*dims, hdx=1.7)
        p, m = sc.pos[:, :3], np.float32(0.5e-3)
        sc.grid_bbmin, sc.grid_bbmax = p.min(0) - m, p.max(0) + m
        return sc

    dims = ((40, 20, 80), (26, 13, 100))
    b = api.Batch()
    sims = [api.Simulation.from_scene(scene(*d)) for d in dims]
    for s in sims:
        b.admit(s)
    b.step(3, record_every=1)
    b.sync()
    for s, d in zip(sims, dims):
        ref = api.Simulation.from_scene(scene(*d))
        ref.advance(3, record_every=1)
        for n in ("POS", "VEL", "S", "T", "VEL_T", "ID"):
            np.testing.assert_array_equal(s.get(n), ref.get(n), err_msg=f"{d}: {n}")
        assert ref.counts()[0] == ref.counts()[1]
        ref.close()
    b.close()
