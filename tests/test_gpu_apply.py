"""The back-transformation's launches over a batch of several size ranges (GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_wide_columns_beside_a_larger_molecule(engine):
    """1014 AOs (the last sizes with 24 columns a CTA) beside 1202 (8 columns): a molecule's arithmetic
    does not depend on the batch, so it has the bits it has alone (8 columns a CTA)."""
    from axtb_b200 import structures as S

    mols = [S.water_cluster(169, seed=s) for s in range(6)] + [S.alkane(200, seed=3, gauche=0.1)]
    rs = engine.Batch(mols, accuracy=1.0).run(gradient=True)
    for i in (0, 5, 6):
        a = engine.Batch([mols[i]], accuracy=1.0).run(gradient=True)[0]
        assert a.status == rs[i].status == 0 and a.iterations == rs[i].iterations
        assert a.energy == rs[i].energy and np.array_equal(a.gradient, rs[i].gradient)


@pytest.mark.parametrize("size, count", [(129, 5), (129, 70), (170, 66)])
def test_many_large_molecules_have_the_bits_they_have_alone(engine, size, count):
    """Above 768 AOs a molecule is reduced by the whole grid when it is alone and by a team of it in a
    batch (774 and 1020 AOs): the same bits, however many there are."""
    from axtb_b200 import structures as S

    mols = [S.water_cluster(size, seed=i % 3) for i in range(count)]
    rs = engine.Batch(mols, accuracy=1.0).run(gradient=True)
    for i in range(3):
        a = engine.Batch([mols[i]], accuracy=1.0).run(gradient=True)[0]
        for r in rs[i::3]:
            assert a.status == r.status == 0 and a.iterations == r.iterations
            assert a.energy == r.energy and np.array_equal(a.gradient, r.gradient)
