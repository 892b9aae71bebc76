"""Sizes that the C ABI refuses before it touches the device. The pointers
here are no memory: with a GPU present nothing of this is called."""
from __future__ import annotations

import ctypes

import pytest
import torch

from kernelkit import _native


@pytest.mark.skipif(torch.cuda.is_available(), reason="no device wanted")
@pytest.mark.parametrize("shape", [(16383, 16383, 16383),
                                   (16383, 8001, 16383)])
def test_adjoint_refuses_more_tiles_than_blocks(shape):
    L = _native.load()
    vol = _native.kk_volume()
    vol.data = 0x1000
    vol.shape[:] = shape
    vol.stride[:] = (shape[1] * shape[2], shape[2], 1)
    proj = _native.kk_projections()
    proj.data = 0x2000
    proj.n_angles = proj.rows = proj.cols = 1
    proj.stride[:] = (1, 1, 1)
    rc = L.kk_cone_fp_adjoint(
        proj, vol, ctypes.c_void_p(0x3000), (ctypes.c_float * 9)(),
        _native.KK_INTERP_TEX8, 16, 0, ctypes.c_void_p(0x4000), 5, None)
    assert rc == _native.KK_ERR_UNSUPPORTED
    assert b"too large" in L.kk_last_error()
