"""The schedule options choose the reduction they name (GPU; the profiler's cycle shares tell)."""
import pytest

pytestmark = pytest.mark.gpu


def _two_stage(engine, waters, **options):
    from axtb_b200 import structures as S

    b = engine.Batch([S.water_cluster(waters, seed=2)], accuracy=1.0, **options)
    b.set_profiling(True)
    r = b.run(gradient=False)[0]
    parts = b.profile()["two_stage_parts"]
    b.close()
    assert r.status == 0
    return parts["band_reduction"] > 0.0


# 36, 42, 60 and 96 AOs around thresholds below, at and above the default; 780 AOs: above what a cluster holds
@pytest.mark.parametrize("waters, threshold, expected", [
    (6, 40, True), (7, 40, False), (7, 48, True), (10, 48, False), (10, 63, True), (10, 65, True), (16, 65, False),
    (16, 97, True), (130, 1 << 20, True), (6, 33, False), (7, 0, False), (6, 64, False), (10, -1, False)])
def test_band_max_nao(engine, waters, threshold, expected):
    assert _two_stage(engine, waters, band_max_nao=threshold) is expected


def test_cycles_cover_the_whole_eigen_phase(engine):
    """The profiler's shares have every part of a staged molecule's eigen phase, and the molecules' own
    counters (the last iteration) add up to no more than all iterations' parts, the reduction being one of
    them."""
    from axtb_b200 import structures as S

    mols = [S.water_cluster(k, seed=k) for k in (2, 10, 40, 140)]  # 12 to 840 AOs: clusters and the grid
    b = engine.Batch(mols, accuracy=1.0)
    b.run(gradient=False)
    assert all(b.debug(i, "eigen_cycles")[0] == 0.0 for i in range(4))
    b.set_profiling(True)
    assert all(r.status == 0 for r in b.run(gradient=True, levels=True))
    p = b.profile()
    shares = p["team_eigen_phases"]
    assert abs(sum(shares.values()) - 1.0) < 1e-3
    for part in ("transform", "tridiagonal", "bisection", "inverse_iteration", "back_transform", "c_matrix", "density"):
        assert shares[part] > 0.0, shares
    cycles = [float(b.debug(i, "eigen_cycles")[0]) for i in range(4)]
    assert all(x < y for x, y in zip(cycles, cycles[1:])) and cycles[0] > 0.0


@pytest.mark.parametrize("waters, options", [
    ([1], {}), ([2, 10, 40], {}), ([1, 11, 60, 130, 140], {}), ([6, 10, 20], {"band_max_nao": 80}),
    ([3, 5], {"solvation": ("alpb", "water")}), ([12, 30], {"precision": "split", "guess": "sad"}), ([20], {"mixer": "diis"})])
def test_launches_are_those_of_the_run(engine, waters, options):
    """The number of launches of a run is that of its kernels in the profiler's trace (CUPTI)."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    from axtb_b200 import structures as S

    b = engine.Batch([S.water_cluster(k, seed=k) for k in waters], accuracy=1.0, **options)
    for gradient, levels in ((True, True), (False, False)):
        b.run(gradient=gradient, levels=levels)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            b.run(gradient=gradient, levels=levels)
            torch.cuda.synchronize()
        kernels = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA and "axg::" in e.name]
        if not kernels:
            pytest.skip("no kernel in the profiler's trace on this machine")
        assert b.launches == len(kernels)
    b.close()
