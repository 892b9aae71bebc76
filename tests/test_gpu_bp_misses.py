"""Backprojection of scans whose cone misses part of the volume: thread
blocks skip the angles that cannot reach them, which must not change a
voxel. Cones narrower than the volume, volumes beside the axis and a source
plane that cuts the volume (voxels behind the source are sampled too, as in
the reference) against the float64-accumulating oracle, through the texture
and from device memory, with the extents that leave partial blocks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import kernelkit as kk
from kernelkit.kernels import VoxelDrivenConeBP
from oracle import cone

pytestmark = pytest.mark.gpu

#: The oracle's own float32 and float64 sample positions give volumes up to
#: 1.6e-4 apart on these scans (positions on a step of the 1/256 weights);
#: the kernel's approximate reciprocal may take either side: twice that. A
#: block that misses one angle's contributions is off by more than 5e-3.
TOL = 3.2e-4

SCANS = {
    # (source x, detector x, rows, cols, volume shape, volume shift)
    "narrow": (-90.0, 60.0, 10, 12, (40, 37, 70), (0.0, 0.0, 0.0)),
    "beside": (-120.0, 80.0, 30, 22, (31, 33, 65), (25.0, -14.0, 20.0)),
    "far_beside": (-150.0, 70.0, 24, 24, (13, 9, 33), (60.0, 10.0, 0.0)),
    "source_inside": (-14.25, 60.0, 40, 48, (36, 34, 34), (0.0, 0.0, 0.0)),
    "one_block": (-60.0, 60.0, 12, 14, (6, 8, 32), (3.0, 0.0, 0.0)),
}


@pytest.mark.parametrize("fetch", ["texture", "global"])
@pytest.mark.parametrize("n_angles", [33, 5])
@pytest.mark.parametrize("name", sorted(SCANS))
def test_skipped_angles_leave_the_volume_unchanged(name, n_angles, fetch):
    sx, dx, rows, cols, shape, shift = SCANS[name]
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.1, pixel_width=1.0)
    g0 = kk.ProjectionGeometry([sx, 0.0, 0.0], [dx, 0.0, 0.0], det)
    pgs = [kk.rotate(g0, yaw=0.013 + 2 * np.pi * k / n_angles)
           for k in range(n_angles)]
    half = np.asarray(shape) / 2
    vg = kk.VolumeGeometry(shape, (1.0,) * 3, np.asarray(shift) - half,
                           np.asarray(shift) + half)
    rng = np.random.default_rng(3)
    sino = rng.uniform(0.0, 1.0, (n_angles, rows, cols)).astype(np.float32)
    K = VoxelDrivenConeBP()
    K.compile()
    params = K.geoms2params(pgs, vg)
    K.set_params(params)
    src = torch.as_tensor(sino, device="cuda")
    if fetch == "texture":
        src = kk.kernel.copy_to_texture(src, layered=True)
    vol = torch.zeros(shape, device="cuda")
    K(src, vol, vg)
    ref = cone.cone_bp(sino, params, shape, 1.0)
    got = vol.cpu().numpy()
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)
