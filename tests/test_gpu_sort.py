"""The cell sort's kernels beside the oracle's integer pipeline, bit for bit.

Particles in no order (no stretches of equal cells to count together, tiles of
the scan far from a block's own), blanked particles spread over more than one
group of hash blocks, cells with many entries, and particle counts at the edges
of warps, blocks and groups, and sparse grids whose tile sums have a scan of
their own; two steps and more, since each step clears the
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


def _sparse(cells):
    """3,000 particles spread over a box of the given numbers of cells"""
    sc = scenes.orthogonal_cutting(20, 15, 10, conduction=0)
    rng = np.random.default_rng(cells[0])
    lo, h = sc.grid_bbmin, np.float32(sc.grid_h)
    size = (np.array(cells, np.float32) - np.float32(0.5)) * h
    sc.pos[:, :3] = lo + size * rng.random((sc.n, 3), dtype=np.float32)
    sc.grid_bbmax = sc.blank_bbmax = (lo + size).astype(np.float32)
    return sc


# 8,160 and 8,225 scan tiles (beyond 8,192 the tile sums have a scan of their own, 8,192 a round)
@pytest.mark.parametrize("cells", [(255, 257, 255), (256, 256, 257), (330, 320, 310)])
def test_sort_of_sparse_grids_matches_the_oracle(cells):
    sim = api.Simulation.from_scene(_sparse(cells))
    (nx, ny, nz), lo, dx = sim.grid()
    assert (nx, ny, nz) == cells
    for _ in range(2):
        before = sim.get("POS")
        sim.step()
        idx, keys, flag = sim.get("IDX"), sim.get("HASH"), sim.get("BLANKED")
        was = np.empty_like(flag)
        was[idx] = flag
        ref = oracle.hash_fp32(before, was, np.array(lo, np.float32), dx, cells)
        n_act, _ = sim.counts()
        for got, want in zip((idx, keys, *sim.cells()), oracle.sort_cells(ref, n_act, nx * ny * nz)):
            np.testing.assert_array_equal(got, want)
    sim.close()


def test_sparse_grid_in_a_batch():
    # one scene's tile sums are scanned in a kernel of their own, the other's are not
    make = (lambda: _sparse((256, 256, 257)), lambda: scenes.orthogonal_cutting(20, 15, 10, conduction=0))
    b = api.Batch()
    sims = [api.Simulation.from_scene(m()) for m in make]
    for s in sims:
        b.admit(s)
    b.step(3)
    for s, m in zip(sims, make):
        ref = api.Simulation.from_scene(m())
        ref.advance(3)
        for f in ("POS", "VEL", "ID"):
            np.testing.assert_array_equal(s.get(f), ref.get(f), err_msg=f)
        ref.close()
    b.close()


def test_scan_time_is_linear_in_the_cells():
    # eight times the cells took 6.6 times as long, and 21 times while each of
    # the scan's blocks added up all the tiles before it (0.43 and 1.43 ms)
    def ms(cells):
        sim = api.Simulation.from_scene(_sparse(cells))
        sim.step()
        sim.set_kernel_timing(True)
        best = np.inf
        for _ in range(5):
            sim.kernel_times()
            sim.step()
            t = sim.kernel_times()
            best = min(best, sum(t[k][0] for k in ("scan_reduce", "scan_top", "scan_down")))
        sim.close()
        return best

    small, large = ms((320, 320, 320)), ms((640, 640, 640))
    assert large < 12.0 * small, (small, large)
