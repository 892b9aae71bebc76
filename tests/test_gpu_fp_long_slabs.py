"""Projections with slabs of more than a thousand slices along the ends of a
long axis: the rounded slice coordinates drift by more than the 0.028 texel
between the half texel and the margin of the usual slabs, so rays whose first
and last sample are inside (or outside) the volume leave (or enter) it in
between. Checked by <A x, y> = <x, A^T y> with the adjoint, which tests every
sample."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import kernelkit as kk
from kernelkit.kernels import RayDrivenConeFP

SHAPE = (1100, 7, 2048)


def test_sequences_leave_the_line():
    """What the kernels are up against, on the CPU: a float32 sequence that
    ends 0.53 texel inside the axis by its line, and outside by its sums."""
    rng = np.random.default_rng(0)
    n, steps, outside = SHAPE[2], SHAPE[0] - 1, 0
    for _ in range(300):
        a = np.float32(rng.uniform(-1e-3, 1e-3))
        z = z0 = np.float32(n - 0.531 - float(a) * steps)
        line = np.float32(float(z0) + float(a) * steps)
        for _ in range(steps):
            z = np.float32(z + a)
        assert line <= n - 0.53 + 1e-3
        outside += z >= n - 0.502
    assert outside > 0


@pytest.mark.gpu
@pytest.mark.parametrize("interp,padded,tex", [
    ("texture", True, True), ("texture", True, False),
    ("texture", False, False), ("exact", True, False),
    ("exact", False, False)])
@pytest.mark.parametrize("end", [1023.0, -1023.0])
@pytest.mark.parametrize("tilt", [0.0, 1e-4])
def test_ends_of_a_long_axis(tilt, end, interp, padded, tex):
    """4800 rays of up to 1100 samples: rounding moves the identity by
    2^-24 sqrt(1100) / sqrt(4800), 3e-8, of |A x| |y|; 2e-7 is allowed. A
    slab left out where its samples' weights reach 0.04 moves it by
    0.04 / sqrt(4800) / 33 and more, and many are at a time."""
    det = kk.Detector(rows=600, cols=8, pixel_height=0.012, pixel_width=0.9)
    g0 = kk.ProjectionGeometry([-4000.0, 0.0, end], [1500.0, 0.0, end], det,
                               v=(0.0, np.sin(tilt), np.cos(tilt)))
    pgs = [g0]
    vg = kk.resolve_volume_geometry(shape=SHAPE, voxel_size=1.0)
    K = RayDrivenConeFP(interpolation=interp, slices_per_block=SHAPE[0],
                        use_texture_unit=tex)
    K.padded_copy = padded
    if interp == "exact" and padded:
        K._pads = lambda *a: True
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(SHAPE, generator=g, device="cuda")
    y = torch.randn((1, 600, 8), generator=g, device="cuda")
    ax, aty = torch.empty_like(y), torch.empty_like(x)
    K(x, pgs, vg, ax, additive=False)
    K.transpose(y, pgs, vg, aty)
    scale = float(ax.double().norm() * y.double().norm())
    assert scale > 0
    assert abs(float((ax.double() * y.double()).sum())
               - float((x.double() * aty.double()).sum())) / scale <= 2e-7
