"""The engine's launch plans, host arithmetic that needs no device (CPU)."""
import ctypes as C

import numpy as np
import pytest


def _apply_plan(nao, nsm=148):
    from axtb_b200 import _lib

    a = np.asarray(nao, dtype=np.int32)
    width, launches = np.zeros_like(a), np.zeros_like(a)
    ptr = lambda x: x.ctypes.data_as(C.POINTER(C.c_int32))
    assert _lib.load().axtb_gpu_apply_plan(ptr(a), len(a), nsm, ptr(width), ptr(launches)) == 0
    return width, launches


def test_back_transformation_takes_every_molecule_once(engine):
    """All sizes beside every largest size (each remainder of eight), in batches that fill the GPU (24
    columns a CTA as far as they fit) and in small ones (8 columns)."""
    nao = np.arange(12, 2406)
    for nmax in list(range(12, 60)) + list(range(380, 440)) + list(range(980, 1060)) + list(range(1195, 1215)) + [1802, 2399, 2405]:
        sizes = nao[nao <= nmax]
        full = np.concatenate([sizes, np.full(7200, 12), [nmax]])  # 7200 column blocks: more than 148
        width, launches = _apply_plan(full)
        assert (launches == 1).all(), full[launches != 1]
        assert ((width == 24) == (full <= 1016)).all()
    width, launches = _apply_plan([1014] * 5 + [1202])  # the smallest batches that get 24 columns
    assert width.tolist() == [8] * 6 and (launches == 1).all()
    width, launches = _apply_plan([1014] * 6 + [1202])
    assert width.tolist() == [24] * 6 + [8] and (launches == 1).all()


def test_kernels_that_need_the_whole_gpu_share_one_stream(engine):
    """k_team_grid and k_trd_grid (in the stages) wait for all of their own CTAs: never in flight beside
    one another. Everything asked for is launched once, the team kernel's parts in their order."""
    from axtb_b200 import _lib

    TEAM_GRID, TEAM, CHASE, TAIL, STAGES = range(5)
    for bits in range(16):
        grid_mols, team, chase, staged = (bits >> k & 1 for k in range(4))
        if (grid_mols or chase) and not team:  # both are team molecules
            continue
        kernel, side = (C.c_int32 * 5)(), (C.c_int32 * 5)()
        assert _lib.load().axtb_gpu_eigen_order(grid_mols, team, chase, staged, kernel, side) == 0
        steps = [(k, s) for k, s in zip(kernel, side) if k >= 0]
        order = [k for k, _ in steps]
        want = [TEAM_GRID] * grid_mols + [TEAM] * team + [CHASE, TAIL] * chase + [STAGES] * staged
        assert sorted(order) == sorted(want)
        assert all(s == 0 for k, s in steps if k in (TEAM_GRID, STAGES)), steps
        chain = [k for k in order if k in (TEAM, CHASE, TAIL)]
        assert chain == sorted(chain) and len({s for k, s in steps if k in chain}) <= 1
        if grid_mols:  # before the fork: the side stream's kernels start after it
            assert order[0] == TEAM_GRID


def test_autotune_times_distinct_schedules():
    from axtb_b200.autotune import band_candidates

    assert band_candidates(0) == band_candidates(32) == [64]  # no molecule of 34 AOs or more below 32
    assert band_candidates(64) == [64, 65]
    assert band_candidates(160) == [64, 160]


def _cholesky_plan(sizes, eeq):
    from axtb_b200 import _lib

    a = np.ascontiguousarray(sizes, dtype=np.int32)
    out = np.zeros((4096, 5), dtype=np.int32)
    ptr = lambda x: x.ctypes.data_as(C.POINTER(C.c_int32))
    n = _lib.load().axtb_gpu_cholesky_plan(ptr(a), len(a), eeq, ptr(out), len(out))
    assert 0 <= n <= len(out)
    return out[:n]


def _tiles(kernel, p, n):
    rt = (n + 63) // 64
    left = np.maximum(rt - 1 - p, 0)
    return [rt * rt, np.where((rt > 1) & (p < rt), rt - 1, 0), left * (left + 1) // 2, (n + 31) // 32, (n + 7) // 8,
            np.ones_like(n)][kernel]


@pytest.mark.parametrize("eeq", [0, 1])
@pytest.mark.parametrize("case", ["one", "small", "edges", "mixed", "small and one large", "many", "none"])
def test_cholesky_steps_cover_every_tile_with_few_empty_ctas(engine, case, eeq):
    rng = np.random.default_rng(1)
    sizes = {"one": [1202], "small": [12] * 300, "edges": [129, 128, 127, 65, 64, 63, 1], "mixed": rng.integers(12, 603, 1024),
             "small and one large": [2400] + [18] * 20000, "many": rng.integers(12, 130, 140000), "none": []}[case]
    n = np.sort(np.asarray(sizes, dtype=np.int64))[::-1]
    plan = _cholesky_plan(n, eeq)
    steps = int((n.max() + 63) // 64) if len(n) else 0
    order = [(0, 0)] + [(k, p) for p in range(steps) for k in (1, 2)] + [(k, 0) for k in (3, 4, 5)] * eeq
    at = 0
    for kernel, p in order:  # in this order, each molecule with tiles in exactly one launch that has them all
        need, got = _tiles(kernel, p, n), np.zeros(len(n), dtype=int)
        while at < len(plan) and tuple(plan[at][:2]) == (kernel, p):
            x, first, count = plan[at][2:]
            assert count <= 65535 and (need[first:first + count] <= x).all()
            assert (x - need[first:first + count]).sum() <= 16384
            got[first:first + count] += 1
            at += 1
        assert ((got == 1) == (need > 0)).all()
    assert at == len(plan)
    assert len(plan) <= 3 * len(order) + 16  # no launch for each size
