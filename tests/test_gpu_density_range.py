"""The allocation-free density over the range of a Fock matrix's magnitude (GPU).

A Fock matrix of zeros, and random ones scaled towards the end of the range: the solutions of the inverse
iteration grow as the inverse of the levels' spacing, above what can be squared. Every level is filled
alike (300 K), so the density is (electrons per level) times the identity. Equal levels are filled in one
step, so the tolerance is round-off.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KT = 300.0 * 3.1668115634564e-6


def _call(f, nocc):
    import torch

    from axtb_b200 import _lib

    n = len(f)
    new = lambda *shape: torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
    fock, overlap = torch.tensor(f, device="cuda"), torch.eye(n, dtype=torch.float64, device="cuda")
    emo, focc, p = new(n), new(n), new(n, n)
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    rc = _lib.load().axtb_gpu_density_static(ptr(fock), ptr(overlap), n, nocc, nocc, KT, ptr(emo), ptr(focc), ptr(p),
                                             ptr(status), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    return emo.cpu().numpy(), focc.cpu().numpy(), p.cpu().numpy(), int(status.item())


@pytest.mark.parametrize("n", [12, 33, 100, 256])
@pytest.mark.parametrize("scale", [0.0, 1e-140, 1e-155])
def test_density_of_tiny_matrices(engine, n, scale):
    a = np.random.default_rng(n).normal(size=(n, n))
    f = scale * (a + a.T)
    emo, focc, p, status = _call(f, n / 4.0)
    assert status == 0
    assert np.abs(np.sort(emo) - np.linalg.eigvalsh(f)).max() <= 1e-13 * scale * n + 1e-300
    assert np.abs(focc - 0.5).max() < 1e-11
    assert np.abs(p - 0.5 * np.eye(n)).max() < 1e-11
