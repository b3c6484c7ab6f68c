"""The integrals' two launch forms, a thread per shell pair and a thread per atom pair (GPU).

A molecule alone takes the first form, in a batch of more than 256 atom pairs a multiprocessor the
second: the same operations, so the same bits of the overlap and core Hamiltonian it started from,
for atoms of one, two and three shells.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [[1, 1], [16, 1, 1], [14, 8]])
def test_both_forms_same_bits(engine, extra):
    from axtb_b200 import structures as S

    z, x = S.water_cluster(40, seed=4)
    far = np.array([[0.0, 0.0, 0.0], [2.6, 0.0, 0.0], [-0.1, 2.6, 0.0]])[: len(extra)] + x.max(0) + 6.0
    mol = (np.concatenate([z, extra]), np.concatenate([x, far]))
    alone = engine.Batch([mol], accuracy=1.0)
    full = engine.Batch([mol] * 8, accuracy=1.0)  # 8 x 7400 atom pairs
    a, f = alone.run(gradient=True)[0], full.run(gradient=True)[7]
    for plane in ("overlap", "fock"):
        assert np.array_equal(alone.debug(0, plane), full.debug(7, plane))
    assert a.energy == f.energy and np.array_equal(a.gradient, f.gradient)
