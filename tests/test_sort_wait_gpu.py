"""A look-back wait of the sort that gives up: the sort ends, every particle is
still there exactly once, the timeout is reported, and the context sorts
correctly afterwards; and every call that reports device errors reports it.  The limit is set to zero polls, so that waits run out at
once on sets that need them (more than one scan tile of 4,096)."""
import numpy as np
import pytest

import oracle as O
from helpers import oracle_particles, with_random_motion
from tigerpm_b200 import _lib
from tigerpm_b200 import workloads as W
from tigerpm_b200.api import GRAVITY_LONG_PME, Server, TigerPM, TPMError, make_options

pytestmark = pytest.mark.gpu


def rows(arrays):
    x, y, z, vx, vy, vz, r = arrays
    a = np.stack([x, y, z, vx.view(np.uint32), vy.view(np.uint32), vz.view(np.uint32), r.astype(np.uint32)])
    return a[:, np.lexsort(a)]


@pytest.mark.parametrize("n,C", [(9000, 3), (50000, 16), (300000, 17), (300000, 64), (4300000, 20)])
def test_sort_that_gave_up_keeps_every_particle(n, C):
    ps = with_random_motion(W.uniform(n, n), n)
    with TigerPM(make_options(max(2, round(n ** (1 / 3))), 16, chain=C), n) as t:
        t.set_wait_limit(0)
        t.set_particles(ps)
        t.chainmesh_create()
        assert np.array_equal(rows(t.get_particles()), rows(ps.arrays()))
        with pytest.raises(TPMError) as e:
            t.check_errors()
        assert e.value.status == _lib.TPM_ERR_TIMEOUT
        t.check_errors()  # reported once
        t.set_wait_limit(1 << 22)
        t.set_particles(ps)
        t.chainmesh_create()
        t.check_errors()
        x, y, z, *_ = t.get_particles()
        p = oracle_particles(O, ps)
        O.chainmesh_sort(C, p)
        assert np.array_equal(x, p.x) and np.array_equal(y, p.y) and np.array_equal(z, p.z)


def test_every_reporting_call_reports_the_timeout():
    ps = with_random_motion(W.uniform(20000, 2), 2)
    opts = make_options(27, 32, chain=6, rs_cells=1.0, rcut_over_rs=4.5)
    with TigerPM(opts, ps.n) as t:
        t.set_wait_limit(0)

        def step(last):
            t.set_particles(ps)
            t.chainmesh_create()
            t.gravity_long_compute(GRAVITY_LONG_PME)
            with pytest.raises(TPMError) as e:
                last()
            assert e.value.status == _lib.TPM_ERR_TIMEOUT
            t.check_errors()

        step(lambda: t.kick_pme_begin(0, 1.0, 0.01, False))
        step(lambda: t.drift(0.01))
        step(lambda: t.integrate(0.01))
    with Server(max_slots=1) as s:
        b = s.add_box(opts, ps)
        s.box(b).set_wait_limit(0)
        with pytest.raises(TPMError) as e:
            s.wait(s.submit(b, 0.01, t0=0.01, first_call=False))
        assert e.value.status == _lib.TPM_ERR_TIMEOUT
