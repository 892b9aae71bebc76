"""Textures that a SIRT solver makes."""
from __future__ import annotations

import math

import pytest
import torch

import kernelkit as kk
from kernelkit import _native
from kernelkit.kernels import VoxelDrivenConeBP, cone_bp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angles", [9, 130])
def test_one_texture_of_the_projections(angles, monkeypatch):
    """C = 1 / A^T 1 comes through the solver's own texture, with the bits
    of a staged backprojection."""
    det = kk.Detector(rows=41, cols=45, pixel_height=1.4, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, yaw=2 * math.pi * k / angles) for k in range(angles)]
    vg = kk.resolve_volume_geometry(shape=(33, 30, 37), voxel_size=1.0)
    made = []
    init = _native.Layered.__init__

    def count(self, *args):
        made.append(args[:3])
        init(self, *args)

    cone_bp.release_staging_textures()
    monkeypatch.setattr(_native.Layered, "__init__", count)
    s = kk.SIRT(torch.rand((angles, 41, 45), device="cuda"), pgs, vg)
    monkeypatch.undo()
    assert cone_bp._STAGES.items == []
    assert sorted(made) == sorted([(33, 30, 37), (angles, 41, 45)])
    K = VoxelDrivenConeBP()
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    C = torch.empty((33, 30, 37), device="cuda")
    K([torch.ones((41, 45), device="cuda") for _ in pgs], C, vg,
      additive=False)
    assert len(cone_bp._STAGES.items) == 1
    C = torch.where(C == 0, torch.zeros_like(C), 1 / C)
    assert torch.equal(s.C, C)
