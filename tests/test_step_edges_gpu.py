"""The step kernels at the ends of their ranges, on open boxes (every voxel a fluid node): the smallest
lattices, and the last and first sizes on either side of the limit up to which transport steps go many to a
launch (60,000 nodes x mobile species)."""
import numpy as np
import pytest

from test_ade_stream_gpu import CASES, STEPS, TOL

pytestmark = pytest.mark.gpu

TIMEOUT = 6


def domain(clb, shape, prec, law, mobile, immobile, microbes, staged=False, seed=3):
    rng = np.random.default_rng(seed)
    N = int(np.prod(shape))
    mat = np.where(rng.random(N) < 0.2, np.where(rng.random(N) < 0.5, 3, 4), 2).astype(np.int8)  # pore and two biofilms
    D = clb.Domain(mat, *shape, 0.8, ade_precision=getattr(clb, prec), bio_codes=(3, 4), perm_ratio=(0.3, 0.3))
    sp = [dict(omega_pore=float(rng.uniform(0.6, 1.6)), omega_biofilm=float(rng.uniform(0.6, 1.6)), mobile=int(s < mobile),
               left_type=s % 3, right_type=(s + 1) % 3, left_bc=0.8, right_bc=0.3, c0=float(rng.uniform(0.05, 0.5)))
          for s in range(mobile + immobile)]
    if immobile and mobile > 1:
        sp = sp[-1:] + sp[:-1]  # the dual-Monod donor is an immobile one
    D.ade_init(sp)
    D.set_velocity(rng.uniform(-0.02, 0.02, (3, N)))
    if microbes:
        D.set_biomass(np.where(rng.random((microbes, N)) < 0.3, rng.uniform(0.0, 60.0, (microbes, N)), 0.0))
    n = mobile + immobile
    D.set_kinetics(law, {0: [], 1: [2e-2] * n, 2: [3e-2] * n + [0.2] * n, 3: [2e-3, 0.1, 0.4, 1e-4]}[law], 1.0)
    if staged:
        D.set_abiotic_kinetics(clb.LAW_PRECIP, [0.0, 0, min(1, n - 1), 0])
    return D


def fields(D, species, microbes):
    return [D.concentration(s) for s in range(species)] + [D.biomass(m) for m in range(microbes)]


@pytest.mark.parametrize("shape", [(3, 2, 2), (4, 3, 3)])
@pytest.mark.parametrize("prec,law,mobile,immobile,microbes", CASES)
def test_smallest_boxes_match_the_staged_step(clb, shape, prec, law, mobile, immobile, microbes):
    out = []
    for staged in (False, True):
        D = domain(clb, shape, prec, law, mobile, immobile, microbes, staged)
        start = fields(D, mobile + immobile, microbes)
        D.ade_step(STEPS)
        out.append(fields(D, mobile + immobile, microbes))
        assert not np.array_equal(start[0], out[-1][0]) or (immobile and law == 0)
        D.close()
    for a, b in zip(*out):
        np.testing.assert_allclose(a, b, rtol=TOL[prec], atol=TOL[prec])


# every form the law enters the step in: none, species by species, dual Monod with mobile and with immobile partners
FORMS = [(0, 1, 0, 0), (2, 1, 1, 0), (3, 1, 1, 1), (0, 2, 0, 0), (1, 2, 0, 0), (3, 2, 0, 1), (3, 2, 1, 2)]


@pytest.mark.parametrize("size", ["smallest", "last", "first past"])
@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
@pytest.mark.parametrize("law,mobile,immobile,microbes", FORMS)
def test_many_steps_per_launch_up_to_their_limit(clb, prec, law, mobile, immobile, microbes, size):
    shape = {"smallest": (4, 3, 3), "last": (40, 50, 30 // mobile), "first past": (41, 50, 30 // mobile)}[size]
    args = (clb, shape, prec, law, mobile, immobile, microbes)
    A, B = domain(*args), domain(*args)
    for n in (4, 3, 7):
        A.ade_step(n)
        for _ in range(n):
            B.ade_step(1)
    for a, b in zip(fields(A, mobile + immobile, microbes), fields(B, mobile + immobile, microbes)):
        np.testing.assert_array_equal(a, b)
    # a barrier that may not wait tells which launch took the steps
    A.tune("barrier_polls", 0)
    A.ade_step(3)
    if size == "first past":
        A.sync()
    else:
        with pytest.raises(clb.ClbError) as e:
            A.sync()
        assert e.value.status == TIMEOUT
    A.close()
    B.close()


@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
def test_flow_of_the_smallest_box(clb, prec):
    out = []
    for keyed in (False, True):
        D = clb.Domain(np.full(36, 2, np.int8), 4, 3, 3, 0.8, flow_precision=getattr(clb, prec))
        D.flow_init(2e-4)
        if keyed:
            D.tune("flow_min_blocks", 3)
        for n in (3, 8, 1):
            D.flow_step(n)
        D.flow_solve(31, 1e-12, allow_unconverged=True)
        stats = D.flow_stats()
        assert stats["bgk_nodes"] == 36 and stats["iterations"] == 43
        out.append(D.flow_populations())
        D.close()
    assert np.ptp(out[0]) > 0
    np.testing.assert_array_equal(*out)
