"""Paired rays of the padded forward projector: exact weights, and detectors
whose rows do not share their in-slice coordinate (tilted), against the
unpadded projector, over ray directions, layouts, storage types, slice
spans and extents that leave partial slabs, rows and columns. Texture-
compatible weights agree bit for bit; exact weights up to the rounding of
a product that only one of the two fuses."""
from __future__ import annotations

import math

import pytest
import torch

import kernelkit as kk
from conftest import rel_l2
from kernelkit.kernels import RayDrivenConeFP

pytestmark = pytest.mark.gpu

#: a fused product differs by half an ulp of a weight, 2^-24
EXACT_TOL = 2e-7


def _scan(kind, n=14, rows=70, cols=41):
    tilt = 0.01 if kind == "tilted" else 0.0
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.2, pixel_width=1.4)
    g0 = kk.ProjectionGeometry(
        [-70.0, 0.5, -0.3], [60.0, 0.0, 0.2], det,
        u=(0.0, math.cos(tilt), math.sin(tilt)),
        v=(0.0, -math.sin(tilt), math.cos(tilt)))
    pitch = (lambda k: -1.2 + 2.4 * k / n) if kind == "alldirs" else \
        (lambda k: 0.02 if kind == "tilted" else 0.0)
    return [kk.rotate(g0, pitch=pitch(k), yaw=0.05 + 2 * math.pi * k / n)
            for k in range(n)]


def _project(kind, interp, padded, vol, axes, span=None, tex=True):
    pgs = _scan(kind)
    shape = [0, 0, 0]
    for k in range(3):
        shape[axes[k]] = vol.shape[k]
    vg = kk.resolve_volume_geometry(shape=tuple(shape), voxel_size=1.0)
    K = RayDrivenConeFP(interpolation=interp, volume_axes=axes,
                        use_texture_unit=tex)
    K.padded_copy = padded
    K.slices_per_launch = span
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    assert K._general == (kind != "circular")
    det = pgs[0].detector
    out = torch.zeros((len(pgs), det.rows, det.cols), device="cuda")
    K(vol, pgs, vg, out, additive=False)
    assert float(out.abs().sum()) > 0
    return out


def _same(kind, interp, vol, axes=(0, 1, 2), **kw):
    got = _project(kind, interp, True, vol, axes, **kw)
    ref = _project(kind, interp, False, vol, axes, **kw)
    if interp == "texture":
        assert torch.equal(got, ref)
    else:
        assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) <= EXACT_TOL


def _volume(shape, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(5)
    return torch.rand(shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("kind", ["circular", "tilted", "alldirs"])
@pytest.mark.parametrize("shape", [(33, 47, 38), (16, 16, 16), (5, 70, 3)])
def test_padded_pairs(shape, kind, interp):
    _same(kind, interp, _volume(shape))


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("kind", ["circular", "tilted"])
def test_padded_pairs_options(kind, interp):
    vol = _volume((37, 33, 40))
    _same(kind, interp, vol, span=16)
    _same(kind, interp, vol, tex=False)
    _same(kind, interp, vol, axes=(2, 1, 0))
    _same(kind, interp, vol, axes=(0, 2, 1))
    _same(kind, interp, vol[:, 1:, 2:37])
    _same(kind, interp, vol.to(torch.bfloat16))
    _same(kind, interp, vol.to(torch.float16))
