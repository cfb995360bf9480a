"""Flow steps launched in a chain, and many traced steps in one launch (small lattices), against the
kernels a tuning key selects, one launch per step: the same populations bit for bit, and the solve's
tracer stopping at the same iteration."""
import numpy as np
import pytest

from helpers import mixed_geometry

pytestmark = pytest.mark.gpu


def domain(clb, shape, prec, per_step):
    mat = clb.sphere_pack(*shape, 0.5, 2.0, 4.0, 7) if min(shape) > 40 else mixed_geometry(*shape, seed=4)
    D = clb.Domain(mat, *shape, 0.8, flow_precision=getattr(clb, prec), bio_codes=(3, 4), perm_ratio=(0.3, 0.0))
    D.flow_init(2e-4)
    if per_step:
        D.tune("flow_min_blocks", 3)
    return D


# a few nodes; a ragged last block; the last size of one traced node per thread and the first of a walk
# (148 x 2 x 256 threads); several nodes per thread
SHAPES = [(4, 3, 3), (19, 12, 23), (66, 50, 50), (70, 54, 54), (80, 90, 70)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
def test_chained_steps_match_single_steps(clb, shape, prec):
    A, B = (domain(clb, shape, prec, per_step) for per_step in (False, True))
    for n in (3, 8, 1, 4):  # either parity at the start of a chain, single steps in between
        A.flow_step(n)
        B.flow_step(n)
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())
    a, b = A.flow_stats(), B.flow_stats()
    assert a["iterations"] == b["iterations"] == 16
    # the same squares added up in another order: N roundings at most
    np.testing.assert_allclose(a["energy"], b["energy"], rtol=A.N * 2.0 ** -53)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
def test_traced_steps_per_launch_match_single_steps(clb, shape, prec):
    A, B = (domain(clb, shape, prec, per_step) for per_step in (False, True))

    def solve(D, n):  # a map without an open path ends at the cap with an error, on both alike
        try:
            return D.flow_solve(n, 1e-12, allow_unconverged=True)
        except clb.ClbError as e:
            return str(e)

    for n in (31, 8):  # either parity, fewer steps than the tracer's window
        assert solve(A, n) == solve(B, n)
    a, b = A.flow_stats(), B.flow_stats()
    assert a["iterations"] == b["iterations"] == 39
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())


@pytest.mark.parametrize("prec", ["F64", "F32"])
def test_traced_solve_stops_at_the_same_iteration(clb, prec):
    A, B = (domain(clb, (19, 12, 23), prec, per_step) for per_step in (False, True))
    ia, ib = A.flow_solve(5000, 1e-3), B.flow_solve(5000, 1e-3)
    assert ia == ib and ia[1] and ia[0] > 500
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())
    # a cap inside a launch, and a second solve that starts from the settled state
    assert A.flow_solve(7, 1e-12, allow_unconverged=True) == B.flow_solve(7, 1e-12, allow_unconverged=True) == (7, False)
    assert A.flow_solve(5000, 1e-3) == B.flow_solve(5000, 1e-3)
    np.testing.assert_array_equal(A.flow_populations(), B.flow_populations())


@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
def test_streamed_step_matches_the_tiled_step(clb, prec):
    """A lattice past the many-step limit (the streamed step, plain and traced; a ragged last block)
    against the tiled and pipelined kernels a tuning key selects: the same bits and iterations."""
    shape = (90, 101, 110)
    mat = clb.sphere_pack(*shape, 0.55, 3.0, 6.0, 3)
    out = []
    for tuned in (False, True):
        D = clb.Domain(mat, *shape, 0.8, flow_precision=getattr(clb, prec))
        D.flow_init(2e-4)
        if tuned:
            D.tune("flow_even_tma", 1)
        D.flow_step(1)
        D.flow_step(6)
        stats = D.flow_stats()
        solved = D.flow_solve(700, 0.2, allow_unconverged=True)
        out.append((D.flow_populations(), stats, solved, D.flow_stats()["iterations"]))
        D.close()
    (fa, sa, va, ia), (fb, sb, vb, ib) = out
    assert sa["active_nodes"] > 400000 and sa["iterations"] == sb["iterations"] == 7
    np.testing.assert_allclose(sa["energy"], sb["energy"], rtol=sa["active_nodes"] * 2.0 ** -53)
    assert va == vb and ia == ib and va[0] >= 500
    np.testing.assert_array_equal(fa, fb)
