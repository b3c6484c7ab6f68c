"""The tridiagonal reduction on chip at odd sizes (GPU): ammonia clusters, 7 basis functions a molecule.

Among them 32 k + 1 rows, where the reduction's last element is the first of a block of rows that no
reflector has reached: on clusters (161, 385), on the whole grid (161 by its threshold, 833, 1057) and on
teams of it; and remainders of the columns over CTAs, warps and register groups. Checked as the even
sizes are: orbital energies and density from the engine's own matrices.
"""
import numpy as np
import pytest
from test_gpu_trd import _check

pytestmark = pytest.mark.gpu


def ammonia(count, seed):
    """`count` NH3 molecules, turned at random, on a cubic lattice of 6.6 bohr."""
    rng = np.random.default_rng(seed)
    r, side = 1.012 / 0.529177210544, int(np.ceil(count ** (1 / 3)))
    c = np.cos(np.radians(106.7))
    tilt = np.arccos(np.sqrt((1.0 + 2.0 * c) / 3.0))  # of an N-H bond from the axis
    bonds = [[np.sin(tilt) * np.cos(a), np.sin(tilt) * np.sin(a), np.cos(tilt)] for a in 2.0 * np.pi / 3.0 * np.arange(3)]
    shape = np.vstack([np.zeros(3), r * np.array(bonds)])
    z, x = [], []
    for i in range(count):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        z += [7, 1, 1, 1]
        x.append(shape @ q.T + 6.6 * np.array([i // side // side, i // side % side, i % side]))
    return np.array(z), np.vstack(x)


# 21, 35, 63, 77, 161, 259, 385 and 763 AOs on clusters
@pytest.mark.parametrize("sizes", [[3, 5, 9, 11], [23, 37], [55, 109]])
def test_clusters(engine, sizes):
    mols = [ammonia(k, k) for k in sizes]
    b = engine.Batch(mols, accuracy=1.0)
    rs = b.run(gradient=True, levels=True)
    for i, r in enumerate(rs):
        assert r.status == 0 and b.debug(i, "fock").shape[0] == 7 * sizes[i]
        _check(b, i, r)


# 161, 833 and 1057 AOs: one molecule on the whole grid, three on teams
@pytest.mark.parametrize("size, threshold", [(23, 100), (119, 1024), (151, 1024)])
@pytest.mark.parametrize("count", [1, 3])
def test_grid(engine, size, threshold, count):
    mols = [ammonia(size, s) for s in range(count)]
    b = engine.Batch(mols, accuracy=1.0, grid_min_nao=threshold)
    rs = b.run(gradient=True, levels=True)
    for i, r in enumerate(rs):
        assert r.status == 0
        _check(b, i, r)
    alone = engine.Batch(mols[-1:], accuracy=1.0, grid_min_nao=threshold).run(gradient=True)[0]
    assert alone.energy == rs[-1].energy and np.array_equal(alone.gradient, rs[-1].gradient)


def test_small_molecules_on_teams(engine):
    """14 to 42 AOs with the threshold lowered to 12: teams of more CTAs than a molecule has columns."""
    mols = [ammonia(k, k) for k in (2, 2, 3, 3, 4, 5, 6, 6, 6, 2)]
    b = engine.Batch(mols, accuracy=1.0, grid_min_nao=12)
    for i, r in enumerate(b.run(gradient=True, levels=True)):
        assert r.status == 0
        _check(b, i, r)
