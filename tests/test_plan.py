"""The engine's launch plans, host arithmetic that needs no device (CPU)."""
import ctypes as C

import numpy as np


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
