"""Rate laws over immobile species alone (no species of the handle moves): the streamed step against the
staged one (an abiotic law whose rate constant is zero changes nothing and takes the staged step), by
single steps, by many in one call, and in a batch on both schedules."""
import numpy as np
import pytest

from test_ade_stream_gpu import TOL, domain

pytestmark = pytest.mark.gpu

SHAPE, STEPS = (14, 9, 17), 12
CASES = [(1, 2, 0), (2, 3, 0), (3, 2, 1), (3, 3, 2), (3, 4, 3)]  # law, immobile species, microbes


def fields(D, species, microbes):
    return [D.concentration(s) for s in range(species)] + [D.biomass(m) for m in range(microbes)]


def staged(clb, prec, law, n, microbes):
    D = domain(clb, SHAPE, prec, law, 0, n, microbes, True, 21)
    start = fields(D, n, microbes)
    D.ade_step(STEPS)
    end = fields(D, n, microbes)
    D.close()
    assert not any(np.array_equal(a, b) for a, b in zip(start, end))  # the law acts on every field
    return end


@pytest.mark.parametrize("call", [1, STEPS])
@pytest.mark.parametrize("prec", ["F64", "F32", "F16S"])
@pytest.mark.parametrize("law,n,microbes", CASES)
def test_laws_act_on_immobile_species_alone(clb, prec, law, n, microbes, call):
    D = domain(clb, SHAPE, prec, law, 0, n, microbes, False, 21)
    for _ in range(STEPS // call):
        D.ade_step(call)
    for a, b in zip(fields(D, n, microbes), staged(clb, prec, law, n, microbes)):
        np.testing.assert_allclose(a, b, rtol=TOL[prec], atol=TOL[prec])
    D.close()


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("law,n,microbes", CASES)
def test_laws_act_on_immobile_species_in_a_batch(clb, law, n, microbes, persistent):
    D = domain(clb, SHAPE, "F32", law, 0, n, microbes, False, 21)
    batch = clb.Batch([D])
    batch.schedule(persistent=persistent)
    batch.step(STEPS, flow=False, transport=True)
    for a, b in zip(fields(D, n, microbes), staged(clb, "F32", law, n, microbes)):
        np.testing.assert_allclose(a, b, rtol=TOL["F32"], atol=TOL["F32"])
    batch.close()
    D.close()
