"""The long-range interpolation over the forms its kernels take: meshes whose
rows are not whole quads, runs at every place of a quad and across the
boundary, scalar tiles, sparse cells, cells split over many blocks, some sinks
only, a kick box inside the mesh, the per-cell launch without the work queue, and
a batch of boxes of all kinds.  Forces against the oracle's FP64 kick on the same
potential; with and without the queue on the same bits of it."""
import numpy as np
import pytest

import oracle as O
from helpers import kick_params, particle_set, rel_rms, with_random_motion
from tigerpm_b200.api import GRAVITY_LONG_PME, Batch, Range, TigerPM, make_options

pytestmark = pytest.mark.gpu


def oracle_forces(opts, sorted_ps, phi, offs, min_rung):
    p = O.Particles(*(a.copy() for a in sorted_ps))
    kp = kick_params(O, opts, min_rung=min_rung, first_call=False, t0=0.01, precision=1)
    ogx, ogy, ogz, opot, _, _ = O.kick_pme(kp, p, offs[:-1].copy(), offs[1:].copy(), phi)
    return np.stack([ogx, ogy, ogz, opot], 1)


@pytest.mark.parametrize("min_rung", [0, 2])
@pytest.mark.parametrize("kind,n_side,grid,C", [
    ("uniform", 24, 30, 5), ("uniform", 24, 32, 5), ("uniform", 24, 44, 7), ("uniform", 24, 45, 7), ("uniform", 20, 64, 6),
    ("uniform", 24, 16, 3), ("uniform", 12, 96, 8), ("uniform", 30, 100, 11), ("halos", 32, 48, 6), ("halos", 32, 64, 12)])
def test_forces(kind, n_side, grid, C, min_rung):
    ps = with_random_motion(particle_set(kind, n_side, 3), 3)
    opts = make_options(n_side, grid, chain=C, rs_cells=grid / C / 4.5, rcut_over_rs=4.5)
    with TigerPM(opts, ps.n) as t:
        t.set_particles(ps)
        t.chainmesh_create()
        before = t.get_particles()
        offs = t.chainmesh_offsets()
        t.gravity_long_compute(GRAVITY_LONG_PME)
        phi = t.gravity_long_get_phi(Range((0, 0, 0), (grid,) * 3))
        t.kick_pme_begin(min_rung, 1.0, 0.01, False)
        t.kick_pme_end()
        G = np.stack(t.get_forces(), 1)
        # the same through a box of cells
        t.set_particles(ps)
        t.chainmesh_create()
        t.gravity_long_compute(GRAVITY_LONG_PME)
        t.kick_pme(Range((1, 0, 1), (C, C - 1, 2)), min_rung, 1.0, 0.01, False)
        B = np.stack(t.get_forces(), 1)
    due = before[6] >= min_rung
    OG = oracle_forces(opts, before, phi, offs, min_rung)
    # FP32 weights and sums against FP64 (the tolerance of the whole-box kick tests)
    assert rel_rms(G[due, :3], OG[due, :3]) < 1e-5
    assert rel_rms(G[due, 3], OG[due, 3]) < 1e-5
    key = np.repeat(np.arange(C ** 3), np.diff(offs))
    x, y, z = key % C, key // C % C, key // (C * C)
    inside = due & (x >= 1) & (y < C - 1) & (z == 1)
    assert rel_rms(B[inside], OG[inside]) < 2e-5 and not np.any(B[~inside])


@pytest.mark.parametrize("kind,n_side,grid,C", [
    ("uniform", 24, 30, 5), ("uniform", 24, 45, 7), ("uniform", 20, 64, 6), ("uniform", 24, 16, 3), ("uniform", 30, 100, 11),
    ("halos", 32, 48, 6), ("halos", 32, 64, 12)])
def test_without_the_queue(kind, n_side, grid, C):
    """kick_grid = 1: no queue, whole cells in the staged tile, the direct form and the scalar one.  The split cells'
    sinks take another form in the queue's run, so forces agree to the rounding of the interpolation's sums."""
    ps = with_random_motion(particle_set(kind, n_side, 3), 3)
    opts = make_options(n_side, grid, chain=C, rs_cells=grid / C / 4.5, rcut_over_rs=4.5, deterministic_deposit=1)
    G = []
    for kick_grid in (0, 1):
        opts.kick_grid = kick_grid
        with TigerPM(opts, ps.n) as t:
            t.set_particles(ps)
            t.chainmesh_create()
            before = t.get_particles()
            offs = t.chainmesh_offsets()
            t.gravity_long_compute(GRAVITY_LONG_PME)
            phi = t.gravity_long_get_phi(Range((0, 0, 0), (grid,) * 3))
            t.kick_pme_begin(0, 1.0, 0.01, False)
            t.kick_pme_end()
            G.append(np.stack(t.get_forces(), 1))
    OG = oracle_forces(opts, before, phi, offs, 0)
    assert rel_rms(G[1][:, :3], OG[:, :3]) < 1e-5 and rel_rms(G[1][:, 3], OG[:, 3]) < 1e-5
    if kind == "uniform":  # no cell is split: the same kernels
        assert np.array_equal(G[0].view(np.uint32), G[1].view(np.uint32))
    else:
        assert rel_rms(G[0], G[1]) < 1e-6


def test_batch_of_all_kinds():
    forms = [(24, 48, 6), (16, 30, 5), (10, 96, 8)]
    opts = [make_options(n, g, chain=c, rs_cells=g / c / 4.5, rcut_over_rs=4.5) for n, g, c in forms]
    sets = [with_random_motion(particle_set("halos" if n == 24 else "uniform", n, n), n, max_rung=0) for n, _, _ in forms]
    b = Batch(opts, [s.n for s in sets])
    for i, s in enumerate(sets):
        b.set_input(i, s)
    for graph in (False, True):
        b.step(restore=True, graph=graph, t0=0.01)
        b.synchronize()
        for i, s in enumerate(sets):
            with TigerPM(opts[i], s.n) as t:
                t.set_particles(s)
                t.pme_step(0, 1.0, 0.01, True)
                one = np.stack(t.get_forces(), 1)
            many = np.stack(b.box(i).get_forces(), 1)
            # FP32 deposit order differs between the two runs
            assert rel_rms(many[:, :3], one[:, :3]) < 1e-5 and rel_rms(many[:, 3], one[:, 3]) < 1e-5
    b.close()
