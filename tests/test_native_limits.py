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


F32, BF16, F16 = _native.KK_F32, _native.KK_BF16, _native.KK_F16


@pytest.mark.skipif(torch.cuda.is_available(), reason="no device wanted")
@pytest.mark.parametrize("as_float", [False, True])
@pytest.mark.parametrize("volume,projections,residual", [
    (F16, BF16, False), (F32, F16, True), (F32, BF16, True),
    (BF16, F32, True), (F16, F32, True), (BF16, BF16, True),
    (F16, BF16, True)])
def test_storage_types_stay_refused(volume, projections, residual, as_float):
    """Also when the volume is traced from a float32 copy, whose kernels
    exist for more combinations."""
    L = _native.load()
    vol = _native.kk_volume()
    vol.data = 0x1000
    vol.shape[:] = (4, 4, 4)
    vol.stride[:] = (16, 4, 1)
    vol.dtype = volume
    proj = _native.kk_projections()
    proj.data = 0x2000
    proj.n_angles, proj.rows, proj.cols = 1, 4, 4
    proj.stride[:] = (16, 4, 1)
    proj.dtype = projections
    o = _native.kk_fp_options()
    res = _native.kk_fp_residual(0x5000, 0x6000)
    if residual:
        o.residual = ctypes.addressof(res)
    if as_float:
        o.padded, o.padded_elems = 0x7000, 512
        o.flags = _native.KK_FP_OPT_PADDED_FLOAT
    rc = L.kk_cone_fp_ex(vol, proj, ctypes.c_void_p(0x3000),
                         (ctypes.c_float * 9)(), o, None)
    assert rc == _native.KK_ERR_UNSUPPORTED
    assert b"dtype combination" in L.kk_last_error()


@pytest.mark.skipif(torch.cuda.is_available(), reason="no device wanted")
def test_a_failed_texture_keeps_its_reason():
    """Giving back the kept textures, of which there are none, does not
    replace the error that asked for it."""
    import kernelkit.kernels  # registers what is given back

    assert kernelkit.kernels and _native.RECLAIM
    with pytest.raises(_native.KernelKitError, match="kk_layered_create"):
        _native.Layered(1, 1, 1, F32)
    with pytest.raises(_native.KernelKitError, match="kk_gather_create"):
        _native.Gather(1, 1, 1)
