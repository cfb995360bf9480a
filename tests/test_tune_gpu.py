"""Tuning keys and the route of the flow step. The route shows in a solve of a small lattice whose grid-wide
barrier may not wait: many steps to a launch (the default) meet the barrier and time out, the per-step kernels a
key chooses have none."""
import numpy as np
import pytest

from helpers import mixed_geometry

pytestmark = pytest.mark.gpu

SHAPE, TIMEOUT = (19, 12, 23), 6


def domain(clb, prec="F32"):
    D = clb.Domain(mixed_geometry(*SHAPE, seed=4), *SHAPE, 0.8, flow_precision=getattr(clb, prec), bio_codes=(3, 4),
                   perm_ratio=(0.3, 0.0))
    D.flow_init(2e-4)
    return D


def many_steps_per_launch(clb, D):
    D.tune("barrier_polls", 0)
    try:
        D.flow_solve(8, 1e-12, allow_unconverged=True)
    except clb.ClbError as e:
        if e.status == TIMEOUT:
            return True
        raise
    finally:
        D.close()
    return False


@pytest.mark.parametrize("prec,key,value", [("F16S", "flow_odd_pipe", 1), ("F32", "flow_min_blocks", 5),
                                            ("F64", "flow_x", 1), ("F32", "flow_", 0)])
def test_a_refused_key_leaves_the_route(clb, prec, key, value):
    D = domain(clb, prec)
    with pytest.raises(clb.ClbError):
        D.tune(key, value)
    assert many_steps_per_launch(clb, D)


@pytest.mark.parametrize("key,value", [("flow_even_tma", 1), ("flow_odd_pipe", 0), ("flow_min_blocks", 2), ("flow_streamed", 0)])
def test_an_accepted_key_changes_the_route_and_one_restores_it(clb, key, value):
    A, B = domain(clb), domain(clb)
    for D in (A, B):
        D.tune(key, value)
        D.flow_step(3)
    B.tune("flow_streamed", 1)
    for D in (A, B):
        D.flow_step(4)
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())
    assert not many_steps_per_launch(clb, A)
    assert many_steps_per_launch(clb, B)


@pytest.mark.parametrize("key", [None, "flow_even_tma"])
def test_autotune_leaves_the_solve_to_its_default(clb, key):
    """The autotuner times steps without the tracer, so whatever it chooses for them a solve goes many steps to
    a launch; the lattice is as it was."""
    A, B = domain(clb), domain(clb)
    for D in (A, B):
        D.flow_step(3)
    if key:
        A.tune(key, 1)
    assert "stream:" in A.autotune(8)
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())
    for D in (A, B):
        D.flow_step(5)
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())
    assert many_steps_per_launch(clb, A)
