"""The column pass of the exact adjoint (circular scans), at the sizes and
scans where it can go wrong: volumes around its 31 x 32 texel tiles,
detectors of one row or column, coarse rows (more than a texel apart) and
fine ones (many rays per texel, down to the ray-by-ray path below 1/16
texel), an upside-down detector, a source inside the volume, other slab
lengths and permuted volumes. Checked by the FP64 dot-product identity
<A x, y> = <x, A^T y>, relative to |A x| |y|."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import kernelkit as kk
from kernelkit.kernels import RayDrivenConeFP

pytestmark = pytest.mark.gpu

#: float32 sums of up to a few hundred terms per voxel and ray: the adjoint's
#: own bound. A lost or doubled sample of these scans (up to 4e4 rays) moves
#: the identity by more than 5e-6
DOT_TOL = 1e-6


def _circle(n, rows, cols, ph=1.3, pw=1.3, source=-80.0, v=(0.0, 0.0, 1.0)):
    det = kk.Detector(rows=rows, cols=cols, pixel_height=ph, pixel_width=pw)
    g0 = kk.ProjectionGeometry([source, 0.0, 0.0], [80.0, 0.0, 0.0], det, v=v)
    return [kk.rotate(g0, yaw=0.1 + 2 * math.pi * k / n) for k in range(n)]


SCANS = {
    "one_tile": (_circle(9, 50, 50), (31, 31, 32)),
    "over_one_tile": (_circle(9, 52, 52), (32, 33, 33)),
    "thin": (_circle(7, 9, 60), (40, 37, 1)),
    "one_row": (_circle(9, 1, 60), (33, 34, 5)),
    "one_column": (_circle(9, 40, 1), (17, 16, 30)),
    "two_rows": (_circle(40, 2, 40, ph=9.0), (20, 20, 21)),
    "coarse": (_circle(12, 12, 14, ph=5.0, pw=5.0), (33, 30, 34)),
    "fine": (_circle(6, 200, 90, ph=0.35, pw=0.5), (20, 21, 34)),
    "very_fine": (_circle(3, 300, 24, ph=0.08, pw=1.3), (12, 12, 10)),
    "upside_down": (_circle(10, 50, 40, v=(0.0, 0.0, -1.0)), (24, 25, 35)),
    "source_inside": (_circle(8, 40, 40, source=-6.3), (20, 22, 24)),
}


def _mismatch(pgs, shape, volume_axes=(0, 1, 2), **kw):
    vg = kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)
    K = RayDrivenConeFP(volume_axes=volume_axes, **kw)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    det = pgs[0].detector
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn([shape[i] for i in volume_axes], generator=g,
                    device="cuda")
    y = torch.randn((len(pgs), det.rows, det.cols), generator=g,
                    device="cuda")
    ax, aty = torch.empty_like(y), torch.empty_like(x)
    K(x, pgs, vg, ax, additive=False)
    K.transpose(y, pgs, vg, aty)
    scale = float(ax.double().norm() * y.double().norm())
    assert scale > 0
    return abs(float((ax.double() * y.double()).sum())
               - float((x.double() * aty.double()).sum())) / scale


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("name", sorted(SCANS))
def test_dot_product_identity(name, interp):
    pgs, shape = SCANS[name]
    assert _mismatch(pgs, shape, interpolation=interp) <= DOT_TOL


@pytest.mark.parametrize("volume_axes", [(2, 1, 0), (1, 0, 2), (0, 2, 1)])
@pytest.mark.parametrize("name", ["over_one_tile", "upside_down"])
def test_permuted_volumes(name, volume_axes):
    pgs, shape = SCANS[name]
    assert _mismatch(pgs, shape, volume_axes) <= DOT_TOL


@pytest.mark.parametrize("slab", [1, 7, 40])
def test_slab_lengths(slab):
    pgs, shape = SCANS["over_one_tile"]
    assert _mismatch(pgs, shape, slices_per_block=slab) <= DOT_TOL


def test_more_tiles_than_one_round():
    """Enough (slice, tile) pairs for the four-way split of the records."""
    assert _mismatch(_circle(5, 380, 260), (230, 160, 250)) <= DOT_TOL
