"""The partition sort where its paths meet: particle counts on and beside a
scan tile (4,096) and a shared-memory unit (8,192), boxes whose units are too
large for one block (a share of the particles in one cell or one row), chain
meshes of many shapes up to 260 cells a side, far fewer particles than cells,
sets large enough for the gather's records, and a captured batch step
replayed.  Positions, velocities and rungs in the
oracle's order, bit for bit."""
import numpy as np
import pytest

import oracle as O
from helpers import oracle_particles, with_random_motion
from tigerpm_b200 import workloads as W
from tigerpm_b200.api import Batch, TigerPM, make_options

pytestmark = pytest.mark.gpu


def check(ps, C, t):
    x, y, z, vx, vy, vz, r = t.get_particles()
    offs = t.chainmesh_offsets()
    p = oracle_particles(O, ps)
    pb, pe = O.chainmesh_sort(C, p)
    assert np.array_equal(offs[:-1], pb) and np.array_equal(offs[1:], pe)
    for a, b in ((x, p.x), (y, p.y), (z, p.z), (r, p.rung)):
        assert np.array_equal(a, b)
    for a, b in ((vx, p.vx), (vy, p.vy), (vz, p.vz)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def sort_and_check(ps, C, times=1):
    with TigerPM(make_options(max(2, round(ps.n ** (1 / 3))), 16, chain=C), max(ps.n, 1)) as t:
        for _ in range(times):
            t.set_particles(ps)
            t.chainmesh_create()
        check(ps, C, t)


def crowded(n, share, where, C, seed):
    """share of n particles inside one chain cell ("cell"), one x row ("row") or one z plane ("plane")."""
    ps = W.uniform(n, seed)
    g = W.rng(seed + 1)
    k = int(share * n)
    pick = g.choice(n, k, replace=False)
    width = (1 << 32) // C
    for axis, a in zip("xyz", (ps.x, ps.y, ps.z)):
        if axis in {"cell": "xyz", "row": "yz", "plane": "z"}[where]:
            a[pick] = (C // 2 * width + g.integers(width // 8, width * 7 // 8, k)).astype(np.uint32)
    return ps


@pytest.mark.parametrize("C", [3, 5, 16])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4095, 4096, 4097, 8191, 8192, 8193, 12289, 65537])
def test_counts_beside_tiles_and_units(n, C):
    sort_and_check(with_random_motion(W.uniform(n, n), n), C, times=2)


@pytest.mark.parametrize("where", ["cell", "row", "plane"])
@pytest.mark.parametrize("n,C", [(30000, 6), (300000, 17), (300000, 33)])
def test_units_too_large_for_a_block(n, C, where):
    sort_and_check(with_random_motion(crowded(n, 0.4, where, C, 3), 3), C)


@pytest.mark.parametrize("C", [4, 6, 7, 9, 12, 15, 31, 32, 47, 64])
def test_chain_mesh_shapes(C):
    sort_and_check(with_random_motion(W.uniform(150001, C), C), C)


def test_large_chain_mesh():
    sort_and_check(with_random_motion(crowded(200003, 0.1, "row", 260, 5), 5), 260)


def test_no_unit_fits_a_block():
    """Thousands of particles in every chain cell (the reference's default options): the level kernels alone."""
    sort_and_check(with_random_motion(W.uniform(200003, 8), 8), 3)


def test_gather_of_many_particles_in_no_order():
    """Above 4,194,304 particles the gather reads records where most sources lie apart, as in a random set; the set
    sorted once more is in order, and is gathered from the arrays."""
    ps = with_random_motion(W.uniform(4300003, 9), 9)
    with TigerPM(make_options(163, 16, chain=37), ps.n) as t:
        t.set_particles(ps)
        for _ in range(2):
            t.chainmesh_create()
            check(ps, 37, t)


@pytest.mark.parametrize("n,C", [(1000, 160), (3000, 160), (200003, 160), (200003, 200), (200003, 260), (2200000, 160)])
def test_chain_mesh_finer_than_the_particles(n, C):
    """Units of a few particles in a thousand cells each: sorted by the level kernels alone once there are many."""
    ps = with_random_motion(W.uniform(n, C), C)
    with TigerPM(make_options(max(2, round(n ** (1 / 3))), 16, chain=C), n) as t:
        t.set_particles(ps)
        before = t.launch_count()
        t.chainmesh_create()
        launches = t.launch_count() - before
        check(ps, C, t)
    levels = 3 * int(np.ceil(np.log2(C)))
    many = n in (3000, 200003)
    if many:  # keys, three of the cell counts' scan, cells of positions, two per level, gather
        assert launches == 6 + 2 * levels


def test_replayed_capture_sorts_new_input():
    """A captured batch step replayed on other particles: nothing of the first sort is left behind."""
    n, C = 20000, 5
    b = Batch([make_options(27, 16, chain=C)], [n])
    for seed in (1, 2, 3):
        ps = with_random_motion(W.uniform(n, seed) if seed != 2 else crowded(n, 0.6, "cell", C, seed), seed, max_rung=0)
        b.set_input(0, ps)
        b.step(restore=True, graph=True, t0=1e-9)
        b.synchronize()
        x, y, z, _, _, _, _ = b.box(0).get_particles()
        p = oracle_particles(O, ps)
        O.chainmesh_sort(C, p)
        assert np.array_equal(x, p.x) and np.array_equal(y, p.y) and np.array_equal(z, p.z)
    b.close()
