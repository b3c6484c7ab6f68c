"""The team kernels at sizes that the stages take by default (GPU).

k_team_grid carries molecules above 2405 AOs and k_team those under 12, or of any size where the stages do
not apply; AXTB_EIGEN_TEAM=1 sends all molecules to them, so that grid-wide barriers, cross-CTA reductions
and the one-CTA algebra are checked at small sizes against the oracle.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

E_TOL, G_TOL = 1e-9, 1e-8  # Eh, Eh/bohr: both sides converged to 1e-6 accuracy


@pytest.mark.parametrize("big", [None, "100", "30"])  # one CTA each; the larger two, then all on the grid
def test_team_kernels_match_the_oracle(engine, monkeypatch, big):
    from axtb_b200 import structures as S

    monkeypatch.setenv("AXTB_EIGEN_TEAM", "1")
    if big:
        monkeypatch.setenv("AXTB_TEAM_BIG_NAO", big)
    mols = [S.water_cluster(20, 3, dims=(5, 2, 2)), S.alkane(8, seed=2), S.alkane(22, seed=4), S.water_cluster(2, 1)]
    b = engine.Batch(mols, accuracy=1e-6)
    res, again = b.run(gradient=True), b.run(gradient=True)
    for (z, x), r, r2 in zip(mols, res, again):
        assert r.energy == r2.energy and np.array_equal(r.gradient, r2.gradient)
        ref = O.singlepoint(z, x, 0.0, None, accuracy=1e-6)
        assert r.status == 0
        assert abs(r.energy - ref["energy"]) < E_TOL
        assert np.abs(r.gradient - ref["gradient"]).max() < G_TOL
    monkeypatch.delenv("AXTB_EIGEN_TEAM")
    for r, s in zip(res, engine.Batch(mols, accuracy=1e-6).run(gradient=True)):  # in stages
        assert abs(r.energy - s.energy) < E_TOL and np.abs(r.gradient - s.gradient).max() < G_TOL
