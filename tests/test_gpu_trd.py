"""The tridiagonal reduction on chip (k_trd on a cluster, k_trd_grid on the whole grid; GPU).

Sizes at the edges of the reduction's classes (a class holds 32 rows per row slot of a thread, a
cluster grows by a CTA when its registers and shared memory are full, column slots come in groups), the smallest molecule that takes it and whole-grid sizes with columns in shared memory:
orbital energies from a plain generalized eigensolve of the engine's own Fock and overlap matrices
(scipy, the eigenvalues' absolute error bounded by n eps ||F'||), the density's idempotency
P S P = 2 P and electron count (round-off of n-term sums of elements of order 1), and the same bits
whether a molecule runs alone or in a batch (clusters of another size).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(b, i, r):
    import scipy.linalg

    f, s, p = (b.debug(i, k) for k in ("fock", "overlap", "density"))
    n = len(f)
    eps, _ = scipy.linalg.eigh(0.5 * (f + f.T), s)
    tol = 8.0 * n * np.finfo(float).eps * np.abs(eps).max() * np.linalg.cond(s)
    assert np.abs(np.sort(r.emo) - eps).max() < tol
    assert np.abs(p @ s @ p - 2.0 * p).max() < 4.0 * n * tol
    assert abs(np.trace(p @ s) - r.focc.sum()) < 4.0 * n * tol


# basis functions: 12 and 14 (first), 30/32/36, 62/66, 96/98, 102, 126/128/132/134, 192/194, 252/258,
# 378/390, 510/516, 606/612, 768
@pytest.mark.parametrize("sizes", [[2, -2, 5, -5, 6], [-10, 11, 16, -16], [17, 21, -21, -22], [32, -32, 42, 43], [63, 65], [85, 86, 101], [102, 128]])
def test_cluster_reduction(engine, sizes):
    from axtb_b200 import structures as S

    mols = [S.water_cluster(k, seed=k) if k > 0 else S.alkane(-k, seed=-k, gauche=0.1) for k in sizes]
    b = engine.Batch(mols, accuracy=1.0)
    rs = b.run(gradient=True, levels=True)
    for i, r in enumerate(rs):
        assert r.status == 0
        _check(b, i, r)
    z, x = mols[0]
    alone = engine.Calculator(z, x, accuracy=1.0).singlepoint(x)
    assert alone.energy == rs[0].energy and np.array_equal(alone.gradient, rs[0].gradient)


def test_cluster_reduction_same_bits_in_a_full_batch(engine):
    """Enough molecules that no cluster grows: the bits of each molecule are those it has alone."""
    from axtb_b200 import structures as S

    mols = [S.water_cluster(17 + i % 30, seed=i) for i in range(160)] + [S.water_cluster(90, seed=1)]
    rs = engine.Batch(mols, accuracy=1.0).run(gradient=True)
    for i in (0, 7, 29, 160):
        a = engine.Batch([mols[i]], accuracy=1.0).run(gradient=True)[0]
        assert a.energy == rs[i].energy and np.array_equal(a.gradient, rs[i].gradient)


@pytest.mark.parametrize("size", [130, 171, 215, -200, 300])
def test_grid_reduction(engine, size):
    from axtb_b200 import structures as S

    z, x = S.water_cluster(size, seed=2) if size > 0 else S.alkane(-size, seed=2, gauche=0.1)
    b = engine.Batch([(z, x)], accuracy=1.0)
    r = b.run(gradient=True, levels=True)[0]
    again = b.run(gradient=True, levels=True)[0]
    assert r.status == 0 and r.energy == again.energy and np.array_equal(r.gradient, again.gradient)
    _check(b, 0, r)
