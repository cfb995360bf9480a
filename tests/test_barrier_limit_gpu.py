"""A grid-wide barrier of the many-step launches that gives up (a limit of no looks at its counter: every
block returns at its first barrier): each call that waits for the lattice or goes on with it returns
CLB_TIMEOUT, until the lattice is initialised again; then the handle answers as a new one does."""
import numpy as np
import pytest

from helpers import mixed_geometry

pytestmark = pytest.mark.gpu

SHAPE, TIMEOUT, DEFAULT = (19, 12, 23), 6, 1 << 24
SP = [dict(omega_pore=1 / 0.9, omega_biofilm=1 / 0.7, left_type=0, right_type=1, left_bc=1.0, c0=0.1)]


def domain(clb):
    mat = mixed_geometry(*SHAPE, seed=4)
    D = clb.Domain(mat, *SHAPE, 0.8, flow_precision=clb.F32, ade_precision=clb.F32, bio_codes=(3, 4),
                   perm_ratio=(0.3, 0.0))
    D.flow_init(2e-4)
    transport(clb, D)
    return D


def transport(clb, D):
    D.ade_init(SP)
    D.set_kinetics(clb.LAW_DECAY, [1e-3], 1.0)


def times_out(clb, call, *args, **kw):
    with pytest.raises(clb.ClbError) as e:
        call(*args, **kw)
    assert e.value.status == TIMEOUT


def test_flow_solve_reports_a_barrier_that_gave_up(clb, tmp_path):
    D, E = domain(clb), domain(clb)
    D.tune("barrier_polls", 0)
    times_out(clb, D.flow_solve, 3000, 1e-9)
    D.tune("barrier_polls", DEFAULT)
    for call, args in ((D.flow_solve, (3000, 1e-9)), (D.flow_step, (1,)), (D.velocity, ()), (D.flow_populations, ()),
                       (D.flow_stats, ()), (D.autotune, (8,)), (D.couple_velocity, ()), (D.checkpoint_save, (str(tmp_path / "c"),)), (D.sync, ())):
        times_out(clb, call, *args)
    D.ade_step(4)  # the species lattices are not concerned
    D.concentration(0)
    D.flow_init(2e-4)
    for X in (D, E):
        X.flow_solve(40, 1e-12, allow_unconverged=True)
        X.sync()
    np.testing.assert_array_equal(D.flow_populations(), E.flow_populations())
    assert D.flow_stats()["iterations"] == 40


def test_run_reports_a_barrier_that_gave_up(clb):
    D = domain(clb)
    D.tune("barrier_polls", 0)
    times_out(clb, D.run, 3, resolve_every=2, flow_max_iterations=600, flow_eps=1e-9)
    times_out(clb, D.run, 3, resolve_every=2, flow_max_iterations=600, flow_eps=1e-9)


def test_transport_reports_a_barrier_that_gave_up(clb, tmp_path):
    D, E = domain(clb), domain(clb)
    D.tune("barrier_polls", 0)
    D.ade_step(2500)  # enqueued; the launches after the first that gave up do nothing
    times_out(clb, D.concentration, 0)
    D.tune("barrier_polls", DEFAULT)
    batch = clb.Batch([D])
    for call, args in ((D.ade_step, (1,)), (D.ade_populations, (0,)), (D.reduce, ()), (D.reduce_noalloc, ()), (D.run, (2,)),
                       (batch.step, (2,)), (D.checkpoint_save, (str(tmp_path / "c"),)), (D.sync, ())):
        times_out(clb, call, *args)
    batch.close()
    D.flow_step(4)  # the flow lattice is not concerned
    D.velocity()
    transport(clb, D)
    for X in (D, E):
        X.ade_step(9)
        X.sync()
    np.testing.assert_array_equal(D.concentration(0), E.concentration(0))


def test_a_limit_below_zero_is_refused(clb):
    D = domain(clb)
    with pytest.raises(clb.ClbError):
        D.tune("barrier_polls", -1)
    D.ade_step(9)
    D.sync()
