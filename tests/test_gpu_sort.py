"""The cell sort's four kernels beside the oracle's integer pipeline, bit for bit.

Particles in no order (no stretches of equal cells to count together, tiles of
the scan far from a block's own), blanked particles spread over more than one
group of hash blocks, cells with many entries, and particle counts at the edges
of warps, blocks and groups; two steps and more, since each step clears the
counters of the next."""
import numpy as np
import pytest

import oracle
from iwf_mfree_gpu_3d_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _take(sc, idx):
    for f in ("pos", "vel", "rho", "T", "h", "fixed", "tool_p"):
        setattr(sc, f, np.ascontiguousarray(getattr(sc, f)[idx]))
    return sc


def _scene(n, shuffled, blanked, dense):
    nz = max(4, round((n / 8.0) ** (1.0 / 3.0)) + 1)
    sc = scenes.orthogonal_cutting(4 * nz, 2 * nz, nz, conduction=0)
    rng = np.random.default_rng(n)
    idx = rng.permutation(sc.n)[:n]
    sc = _take(sc, idx if shuffled else np.sort(idx))
    if dense:
        sc.pos[:, :3] *= np.float32(0.3)
    if blanked:  # the blanking box cuts through the block: about a third of it lies outside
        lo, hi = sc.pos[:, :3].min(0), sc.pos[:, :3].max(0)
        sc.blank_bbmax = sc.blank_bbmax.copy()
        sc.blank_bbmax[1] = lo[1] + 0.66 * (hi[1] - lo[1])
    return sc


@pytest.mark.parametrize("n,shuffled,blanked,dense", [
    (31, True, False, False), (256, True, True, False), (257, False, True, False), (2049, True, False, True),
    (32768, False, True, False), (40001, True, True, False), (70000, True, True, True)])
def test_sort_matches_the_oracle(n, shuffled, blanked, dense):
    sc = _scene(n, shuffled, blanked, dense)
    sim = api.Simulation.from_scene(sc)
    (nx, ny, nz), lo, dx = sim.grid()
    for _ in range(3):
        before = sim.get("POS")
        sim.step()
        idx, keys, flag = sim.get("IDX"), sim.get("HASH"), sim.get("BLANKED")
        was = np.empty_like(flag)
        was[idx] = flag
        n_act, _ = sim.counts()
        ref = oracle.hash_fp32(before, was, np.array(lo, np.float32), dx, (nx, ny, nz))
        assert n_act == int((ref != np.iinfo(np.int32).max).sum()) and (n_act < n) == blanked
        for got, want in zip((idx, keys, *sim.cells()), oracle.sort_cells(ref, n_act, nx * ny * nz)):
            np.testing.assert_array_equal(got, want)
    sim.close()
