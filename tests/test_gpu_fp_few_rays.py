"""Exact weights: the zero-padded volume copy is made where the rays take
enough samples to pay for it, and both ways give the same projections up to
the rounding of a product that only one of them fuses."""
from __future__ import annotations

import math

import pytest
import torch

import kernelkit as kk
from conftest import rel_l2
from kernelkit.kernels import RayDrivenConeFP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angles,rows,cols,padded", [
    (1, 3, 5, False),  # one angle of a few pixels
    (2, 40, 78, False), (2, 40, 82, True),  # 7.8 and 8.2 samples per voxel
    (12, 41, 43, True)])
def test_padded_where_it_pays(angles, rows, cols, padded):
    shape = (20, 40, 40)
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.1, pixel_width=0.7)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, yaw=0.3 + 2 * math.pi * k / angles)
           for k in range(angles)]
    vg = kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)
    x = torch.rand(shape, device="cuda")
    outs = []
    for copy in (True, False):
        K = RayDrivenConeFP(interpolation="exact")
        K.padded_copy = copy
        K.compile()
        K.set_params(K.geoms2params(pgs, vg))
        out = torch.empty((angles, rows, cols), device="cuda")
        K(x, pgs, vg, out, additive=False)
        outs.append(out.cpu().numpy())
        assert hasattr(K, "_pad_buf") == (copy and padded)
    # a fused product differs by half an ulp of a weight, 2^-24
    assert rel_l2(*outs) <= 2e-7
    # texture weights keep the copy in every case
    K = RayDrivenConeFP()
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    K(x, pgs, vg, out, additive=False)
    assert hasattr(K, "_pad_buf")
