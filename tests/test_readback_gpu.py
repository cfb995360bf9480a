"""Fields read back a run of rows at a time against the populations they are sums of, on a box larger
than the staging buffer with rows that are not a multiple of a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C19 = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1),
       (0, -1, 1)]
C19 = np.array(C19 + [tuple(-v for v in c) for c in C19[1:]], dtype=np.float64)


@pytest.mark.parametrize("steps", [4, 5])
@pytest.mark.parametrize("prec", ["F64", "F32"])
def test_fields_equal_the_sums_of_their_populations(clb, prec, steps):
    shape = (47, 173, 201)  # 1.6 M voxels: 39 MB of FP64 velocity, 13 MB of one FP64 concentration
    mat = clb.sphere_pack(*shape, 0.45, 3.0, 6.0, 9)
    p = getattr(clb, prec)
    D = clb.Domain(mat, *shape, 0.8, flow_precision=p, ade_precision=p)
    D.flow_init(1e-4)
    D.flow_step(steps)
    D.ade_init([dict(omega_pore=1.1, left_type=2, right_type=2, c0=0.3),
                dict(omega_pore=0.9, left_type=0, right_type=1, left_bc=1.0, c0=0.1)])
    D.couple_velocity()
    D.ade_step(steps)
    # sums of 19 (7) stored values in another order: a rounding of the arithmetic type per term
    eps = 2.0 ** (-53 if prec == "F64" else -24)
    f = D.flow_populations()
    u = C19.T @ f
    open_ = (mat == 2).reshape(shape)
    inner = open_.copy()
    inner[0] = inner[-1] = False
    scale = np.abs(f).max() * 19
    v = D.velocity()
    assert np.abs(v - u)[:, inner.ravel()].max() <= 19 * eps * scale
    assert not v[:, ~open_.ravel()].any()
    np.testing.assert_array_equal(D.velocity(dtype=np.float32), v.astype(np.float32))
    for s, closed in ((0, True), (1, False)):
        c = D.concentration(s)
        total = 1.0 + D.ade_populations(s).sum(axis=0)
        sel = np.ones(shape, bool) if closed else ~open_ | inner
        assert np.abs(c - total)[sel.ravel()].max() <= 14 * eps * 7
    D.close()
