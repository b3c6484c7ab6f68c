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
