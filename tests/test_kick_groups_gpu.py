"""The kick's sink groups and source steps at their edges: chain cells whose
counts sit on and beside the group (8), pass (64 .. 256) and source-step
sizes, with and without a cutoff, under the minimum image (chain_dim = 3),
and with only some sinks due; and the forms that take a cell's passes as items
of a queue (cells of more than four passes of 64 to 256 sinks): without a cutoff,
under the minimum image, where every cell is split, with passes that have no due
sink, and in a batch whose boxes differ in their cutoffs.  Against the oracle's
FP64 pair sum."""
import numpy as np
import pytest

import oracle as O
from helpers import kick_params, rel_rms
from tigerpm_b200 import workloads as W
from tigerpm_b200.api import GRAVITY_LONG_PME, Batch, Range, TigerPM, make_options

pytestmark = pytest.mark.gpu


def cells_with(counts, C, seed):
    """A particle set whose chain cells hold the given counts, taken in turn."""
    g = W.rng(seed)
    per = np.resize(np.array(counts), C ** 3)
    cell = np.repeat(np.arange(C ** 3), per)
    pos = np.stack([cell % C, cell // C % C, cell // (C * C)]) + g.uniform(0.001, 0.999, (3, cell.size))
    raw = np.minimum(np.floor(pos / C * W.TWO32), W.TWO32 - 1).astype(np.uint32)
    n = cell.size
    v = g.normal(0, 1e-3, (3, n)).astype(np.float32)
    return W.ParticleSet(raw[0].copy(), raw[1].copy(), raw[2].copy(), v[0].copy(), v[1].copy(), v[2].copy(),
                         g.integers(0, 4, n).astype(np.int8))


@pytest.mark.parametrize("min_rung", [0, 2])
@pytest.mark.parametrize("C,rcut", [(3, 0.0), (3, 4.5), (4, 0.0), (5, 4.5)])
@pytest.mark.parametrize("counts", [(1, 0, 7, 8, 9), (15, 16, 17, 33), (63, 64, 65, 2), (127, 0, 129), (255, 3, 257, 0, 9)])
def test_group_edges(counts, C, rcut, min_rung):
    grid = 32
    ps = cells_with(counts, C, 7 + C)
    rs = grid / C / 4.5 if rcut > 0 else 1.0
    opts = make_options(max(2, round(ps.n ** (1 / 3))), grid, chain=C, rs_cells=rs, rcut_over_rs=rcut)
    with TigerPM(opts, ps.n) as t:
        t.set_particles(ps)
        t.chainmesh_create()
        x, y, z, vx, vy, vz, r = t.get_particles()
        t.gravity_long_compute(GRAVITY_LONG_PME)
        phi = t.gravity_long_get_phi(Range((0, 0, 0), (grid, grid, grid)))
        t.kick_pme_begin(min_rung, 1.0, 0.01, False)
        t.kick_pme_end()
        after = t.get_particles()
        G = np.stack(t.get_forces(), 1)
        offs = t.chainmesh_offsets()
    p = O.Particles(x.copy(), y.copy(), z.copy(), vx.copy(), vy.copy(), vz.copy(), r.copy())
    kp = kick_params(O, opts, min_rung=min_rung, first_call=False, t0=0.01, precision=1)
    ogx, ogy, ogz, opot, _, _ = O.kick_pme(kp, p, offs[:-1].copy(), offs[1:].copy(), phi)
    due = r >= min_rung
    # FP32 pair terms and sums against FP64 (the tolerance of the whole-box kick tests)
    assert rel_rms(G[due, :3], np.stack([ogx, ogy, ogz], 1)[due]) < 1e-5
    assert rel_rms(G[due, 3], opot[due]) < 1e-5
    assert not np.any(G[~due])
    assert np.array_equal(after[6][~due], r[~due]) and np.mean(after[6] != p.rung) < 1e-3 + 1.5 / ps.n


def sampled_error(opts, sorted_ps, phi, offs, G, cells, min_rung, first=False):
    """Relative rms error of forces and potentials at the due sinks of the given cells."""
    p = O.Particles(*(a.copy() for a in sorted_ps))
    kp = kick_params(O, opts, min_rung=min_rung, first_call=first, t0=0.01, precision=1)
    ogx, ogy, ogz, opot, _, _ = O.kick_pme(kp, p, offs[:-1].copy(), offs[1:].copy(), phi,
                                           sink_cells=np.array(cells, np.int32))
    idx = np.concatenate([np.arange(offs[c], offs[c + 1]) for c in cells])
    idx = idx[sorted_ps[6][idx] >= min_rung]
    OG = np.stack([ogx, ogy, ogz, opot], 1)
    return rel_rms(G[idx, :3], OG[idx, :3]), rel_rms(G[idx, 3], OG[idx, 3])


HEAVY = [20] * 21 + [3000] + [20] * 42  # chain_dim = 4: one cell of 24 passes of 128 sinks, its neighbours light


@pytest.mark.parametrize("min_rung,due", [(0, 1.0), (2, 0.5), (2, 0.002)])
@pytest.mark.parametrize("counts,C,rcut,cells", [
    (HEAVY, 4, 0.0, [21, 22, 5, 63]), (HEAVY, 4, 4.5, [21, 22, 5, 63]),
    ([1100, 1500, 1300], 3, 0.0, [0, 13]), ([1100, 1500, 1300], 3, 4.5, [0, 13])])
def test_split_cells(counts, C, rcut, cells, min_rung, due):
    grid = 32
    ps = cells_with(counts, C, 11)
    g = W.rng(12)
    ps.rung[:] = np.where(g.random(ps.n) < due, 3, 0)  # due = 0.002: most passes have no due sink
    opts = make_options(max(2, round(ps.n ** (1 / 3))), grid, chain=C, rs_cells=grid / C / 4.5 if rcut > 0 else 1.0,
                        rcut_over_rs=rcut)
    with TigerPM(opts, ps.n) as t:
        t.set_particles(ps)
        t.chainmesh_create()
        before = t.get_particles()
        t.gravity_long_compute(GRAVITY_LONG_PME)
        phi = t.gravity_long_get_phi(Range((0, 0, 0), (grid, grid, grid)))
        t.kick_pme_begin(min_rung, 1.0, 0.01, False)
        t.kick_pme_end()
        G = np.stack(t.get_forces(), 1)
        offs = t.chainmesh_offsets()
    assert np.diff(offs).max() > 4 * 256
    # the tolerance of the whole-box kick tests
    assert max(sampled_error(opts, before, phi, offs, G, cells, min_rung)) < 1e-5
    assert not np.any(G[before[6] < min_rung])


def test_batch_of_cut_and_uncut_boxes():
    """One launch for boxes with and without a cutoff, each with a cell of several pass items."""
    grid, C = 32, 4
    sets = [cells_with(HEAVY, C, 21), cells_with(HEAVY[::-1], C, 22), cells_with([40, 0, 90], C, 23)]
    opts = [make_options(max(2, round(s.n ** (1 / 3))), grid, chain=C, rs_cells=grid / C / 4.5, rcut_over_rs=r,
                         deterministic_deposit=1) for s, r in zip(sets, (0.0, 4.5, 0.0))]
    b = Batch(opts, [s.n for s in sets])
    for i, s in enumerate(sets):
        s.rung[:] = 0
        b.set_input(i, s)
    for graph in (False, True):
        b.step(restore=True, graph=graph, t0=0.01)
        b.synchronize()
        for i, (o, s) in enumerate(zip(opts, sets)):
            with TigerPM(o, s.n) as t:  # the same box and potential alone, for the oracle
                t.set_particles(s)
                t.chainmesh_create()
                before = t.get_particles()
                offs = t.chainmesh_offsets()
                t.gravity_long_compute(GRAVITY_LONG_PME)
                phi = t.gravity_long_get_phi(Range((0, 0, 0), (grid, grid, grid)))
            G = np.stack(b.box(i).get_forces(), 1)
            cells = [21, 22, 42, 5]
            assert max(sampled_error(o, before, phi, offs, G, cells, 0, first=True)) < 1e-5
    b.close()
