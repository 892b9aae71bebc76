"""The exact adjoint where few samples could be lost unseen: slabs of many
hundred slices on long axes, whose rounded slice coordinates leave the
straight line by more than the candidate boxes' own margin, and volumes with
enough tiles for the four-warp column kernel, with so few rays that every
sample counts. Checked by <A x, y> = <x, A^T y>."""
from __future__ import annotations

import math

import pytest
import torch

import kernelkit as kk
from kernelkit.kernels import RayDrivenConeFP

pytestmark = pytest.mark.gpu


def _mismatch(pgs, shape, y_of=None, **kw):
    vg = kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)
    K = RayDrivenConeFP(**kw)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    det = pgs[0].detector
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(shape, generator=g, device="cuda")
    y = torch.randn((len(pgs), det.rows, det.cols), generator=g,
                    device="cuda")
    if y_of is not None:
        y = y_of(y, g)
    ax, aty = torch.empty_like(y), torch.empty_like(x)
    K(x, pgs, vg, ax, additive=False)
    K.transpose(y, pgs, vg, aty)
    ax = torch.where(y != 0, ax, torch.zeros_like(ax))
    scale = float(ax.double().norm() * y.double().norm())
    assert scale > 0
    return abs(float((ax.double() * y.double()).sum())
               - float((x.double() * aty.double()).sum())) / scale


#: long axis (source, detector, their height), detector, volume
LONG = {
    # narrow rows at the far end of a long axis (the column walk's start)
    "rows": (-5000.0, 1500.0, 1900.0, 600, 8, 0.09, 1.3, (1200, 6, 4000)),
    # a source inside the slab: rows in both orders
    "behind": (-20.0, 1500.0, 1900.0, 600, 8, 0.09, 1.3, (1200, 6, 4000)),
    # narrow columns across a long axis (the candidate columns)
    "columns": (-2600.0, 1500.0, 0.0, 8, 6000, 1.3, 0.9, (1200, 4000, 6)),
}


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("slab", [16, 300, 1200])
@pytest.mark.parametrize("tilt", [0.0, 1e-3])
@pytest.mark.parametrize("name", sorted(LONG))
def test_long_slabs(name, tilt, slab, interp):
    """Float32 sums of up to 1200 terms (2^-24 sqrt(1200), 2e-6) of at least
    14400 rays agree to 2e-6 / sqrt(14400), 2e-8, of |A x| |y|; five times
    that is allowed. One lost sample moves the identity by about 1e-6."""
    sx, dx, z, rows, cols, ph, pw, shape = LONG[name]
    det = kk.Detector(rows=rows, cols=cols, pixel_height=ph, pixel_width=pw)
    g0 = kk.ProjectionGeometry([sx, 0.0, z], [dx, 0.0, z], det,
                               v=(0.0, math.sin(tilt), math.cos(tilt)))
    pgs = [kk.rotate(g0, yaw=0.0007 * k) for k in range(3)]
    assert _mismatch(pgs, shape, interpolation=interp,
                     slices_per_block=slab) <= 1e-7


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("flip", [1.0, -1.0])
def test_single_rays_of_many_tiles(flip, interp):
    """300 rays that cross some 60000 samples, 2000 of them at the edges of
    the tiles' rows and as many at their texels': one lost or doubled moves
    the identity by about 1 / (300 sqrt(230)), 2e-4. Rounding: sums of up to
    230 terms, 2^-24 sqrt(230) / sqrt(300), 5e-8; 1e-6 is allowed."""
    det = kk.Detector(rows=380, cols=260, pixel_height=1.3, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-400.0, 0.0, 0.0], [80.0, 0.0, 0.0], det,
                               v=(0.0, 0.0, flip))
    pgs = [kk.rotate(g0, yaw=0.1 + 2 * math.pi * k / 5) for k in range(5)]

    def few(y, g):
        keep = torch.randperm(y.numel(), generator=g, device="cuda")[:300]
        out = torch.zeros_like(y)
        out.view(-1)[keep] = y.view(-1)[keep]
        return out

    shape = (230, 160, 250)
    for axis, across in ((0, 1), (1, 0)):  # the four-warp kernel's volumes
        assert shape[axis] * -(-shape[across] // 31) * -(-shape[2] // 32) \
            >= 148 * 40
    assert _mismatch(pgs, shape, few, interpolation=interp) <= 1e-6
