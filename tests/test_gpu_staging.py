"""Staging textures of the backprojection when something else goes on: no
memory for a texture."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import kernelkit as kk
from kernelkit import _native
from kernelkit.kernels import VoxelDrivenConeBP, cone_bp
from kernelkit.kernels.cone_fp import interp_code

pytestmark = pytest.mark.gpu

SHAPE = (33, 30, 37)


def _case(n, interp="texture", rows=41, cols=45):
    """(kernel, volume geometry, projections)."""
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.4, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, roll=0.01, pitch=0.02, yaw=2 * math.pi * k / n)
           for k in range(n)]
    vg = kk.resolve_volume_geometry(shape=SHAPE, voxel_size=1.0)
    K = VoxelDrivenConeBP(interpolation=interp)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    g = torch.Generator(device="cuda").manual_seed(n)
    return K, vg, torch.rand((n, rows, cols), generator=g, device="cuda")


def _direct(K, y, vg):
    """The device-memory path of the C ABI."""
    out = torch.empty(SHAPE, device="cuda")
    _native.check(_native.load().kk_cone_bp(
        _native.projections_desc(y), _native.volume_desc(out),
        K._params_dev.data_ptr(), float(np.float32(vg.voxel_volume())),
        interp_code(K.interpolation), 0, None, _native.current_stream()))
    return out


class _NoMemory:
    """A texture that no GPU has the memory for (2.2 TB): the allocation
    itself fails, with the runtime's own error."""

    def __new__(cls, *shape_and_dtype):
        return _native.Layered(2048, 16383, 16383, _native.KK_F32)


def test_failed_creation_leaves_no_error_behind():
    K, vg, y = _case(5)
    with pytest.raises(_native.KernelKitError):
        _NoMemory()
    out = torch.empty(SHAPE, device="cuda")
    _native.check(_native.load().kk_cone_bp(
        _native.projections_desc(y), _native.volume_desc(out),
        K._params_dev.data_ptr(), 1.0, _native.KK_INTERP_TEX8, 0, None,
        _native.current_stream()))


@pytest.mark.parametrize("interp", ["texture", "exact"])
def test_no_memory_for_a_texture(interp, monkeypatch):
    """The projections are then read from device memory."""
    K, vg, y = _case(40, interp)
    cone_bp.release_staging_textures()

    class Native:
        def __getattr__(self, name):
            return _NoMemory if name == "Layered" else getattr(_native, name)

    monkeypatch.setattr(cone_bp, "_native", Native())
    out = torch.empty(SHAPE, device="cuda")
    K([f.clone() for f in y], out, vg, additive=False)
    assert cone_bp._STAGES.items == []
    assert torch.equal(out, _direct(K, y, vg))
