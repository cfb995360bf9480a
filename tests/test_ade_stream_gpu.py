"""The streamed transport step against the staged one: an abiotic law whose rate constant is zero
changes nothing and takes the staged step, so both run the same problem over every law, type and
species split the streamed step accepts."""
import numpy as np
import pytest

from helpers import mixed_geometry

pytestmark = pytest.mark.gpu

STEPS = 21
# Both forms round each of a node's operations alike up to which product a fused multiply-add leaves
# unrounded: half an ulp of a population (at most 1) per step, carried over STEPS steps and summed over
# 7 populations. FP16 storage turns that into one unit of its 11 bits now and then.
TOL = {"F64": STEPS * 7 * 2.0 ** -53, "F32": STEPS * 7 * 2.0 ** -24, "F16S": STEPS * 2.0 ** -11}


def domain(clb, shape, prec, law, mobile, immobile, microbes, staged, seed):
    rng = np.random.default_rng(seed)
    mat = mixed_geometry(*shape, seed=seed, solid_block=min(shape) > 6)
    D = clb.Domain(mat, *shape, 0.8, ade_precision=getattr(clb, prec), bio_codes=(3, 4), perm_ratio=(0.3, 0.3))
    sp = []
    for s in range(mobile + immobile):
        sp.append(dict(omega_pore=float(rng.uniform(0.6, 1.6)), omega_biofilm=float(rng.uniform(0.6, 1.6)),
                       mobile=int(s < mobile), left_type=s % 3, right_type=(s + 1) % 3, left_bc=0.8, right_bc=0.3,
                       c0=float(rng.uniform(0.05, 0.5))))
    if immobile and mobile > 1:
        sp = sp[-1:] + sp[:-1]  # the dual-Monod donor (species 0) is an immobile one
    D.ade_init(sp)
    D.set_velocity(rng.uniform(-0.02, 0.02, (3, D.N)))
    if microbes:
        b = np.where(rng.random((microbes, D.N)) < 0.1, rng.uniform(0.0, 60.0, (microbes, D.N)), 0.0)
        b[:, rng.random(D.N) < 0.05] = 1e-13  # below the threshold
        D.set_biomass(b)
    n = mobile + immobile
    D.set_kinetics(law, {0: [], 1: [2e-2] * n, 2: [3e-2] * n + [0.2] * n, 3: [2e-3, 0.1, 0.4, 1e-4]}[law], 1.0)
    if staged:
        D.set_abiotic_kinetics(clb.LAW_PRECIP, [0.0, 0, min(1, n - 1), 0])
    return D


CASES = [("F64", 1, 1, 0, 0), ("F32", 2, 1, 1, 0), ("F32", 0, 2, 0, 0), ("F64", 2, 3, 1, 0), ("F16S", 1, 5, 0, 0),
         ("F32", 3, 4, 0, 2), ("F64", 3, 2, 0, 2), ("F16S", 3, 4, 0, 2), ("F32", 3, 5, 0, 3), ("F64", 3, 3, 1, 2),
         ("F32", 3, 1, 0, 1), ("F32", 3, 15, 1, 1), ("F32", 1, 16, 0, 0)]


@pytest.mark.parametrize("shape", [(4, 3, 3), (9, 8, 17), (22, 11, 33)])
@pytest.mark.parametrize("prec,law,mobile,immobile,microbes", CASES)
def test_streamed_step_matches_the_staged_step(clb, shape, prec, law, mobile, immobile, microbes):
    out = []
    for staged in (False, True):
        D = domain(clb, shape, prec, law, mobile, immobile, microbes, staged, 11 + mobile)
        D.ade_step(STEPS)
        out.append([D.concentration(s) for s in range(mobile + immobile)] + [D.biomass(m) for m in range(microbes)])
        D.close()
    for a, b in zip(*out):
        np.testing.assert_allclose(a, b, rtol=TOL[prec], atol=TOL[prec])


@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
def test_batch_of_mixed_laws_matches_single_domains(clb, prec):
    """A batch whose domains hold different laws, species counts and sizes (tiles of every streamed
    form, ragged ones among them) against the same domains stepped one by one: the same bits."""
    cases = [(0, 2, 0, 0), (2, 3, 1, 0), (3, 3, 0, 2), (1, 1, 0, 0), (3, 4, 0, 3), (3, 4, 0, 1)]
    shapes = [(9, 8, 17), (22, 11, 33), (14, 13, 12), (4, 3, 3), (18, 9, 21), (30, 16, 16)]
    A, B = ([domain(clb, sh, prec, *c, False, 3 + i) for i, (sh, c) in enumerate(zip(shapes, cases))] for _ in range(2))
    batch = clb.Batch(B)
    batch.schedule(persistent=False)
    for n in (7, 2):
        batch.step(n, flow=False, transport=True)
        for D in A:
            D.ade_step(n)
    for a, b, c in zip(A, B, cases):
        for s in range(c[1] + c[2]):
            np.testing.assert_array_equal(a.concentration(s), b.concentration(s))
        for m in range(c[3]):
            np.testing.assert_array_equal(a.biomass(m), b.biomass(m))
    batch.close()


@pytest.mark.parametrize("shape", [(3, 5, 6), (4, 3, 3), (9, 8, 17), (66, 50, 50), (70, 54, 54)])
@pytest.mark.parametrize("prec,law,mobile,immobile,microbes", CASES[:-2])
def test_many_steps_per_launch_match_single_steps(clb, shape, prec, law, mobile, immobile, microbes):
    """Steps taken many to a launch (a few nodes, ragged blocks, one node per thread, several) against
    the same steps launched one by one: the same bits, from either parity."""
    A, B = (domain(clb, shape, prec, law, mobile, immobile, microbes, False, 5 + mobile) for _ in range(2))
    for n in (4, 3, 1, 8):
        A.ade_step(n)
        for _ in range(n):
            B.ade_step(1)
    for s in range(mobile + immobile):
        np.testing.assert_array_equal(A.concentration(s), B.concentration(s))
    for m in range(microbes):
        np.testing.assert_array_equal(A.biomass(m), B.biomass(m))
    A.close()
    B.close()
