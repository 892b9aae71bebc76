"""Backprojection launches split by 32-angle chunk (volumes of few blocks):
bit for bit the one-chunk-per-launch batched kernel's volumes, for angle
counts that leave one to four chunks and partial ones, extents with partial
blocks, the additive and update epilogues and 16-bit volumes."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

import kernelkit as kk
from conftest import rel_l2
from kernelkit import _native
from kernelkit.kernels import VoxelDrivenConeBP

pytestmark = pytest.mark.gpu


def _setup(n, shape):
    det = kk.Detector(rows=40, cols=44, pixel_height=1.4, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, yaw=2 * math.pi * k / n) for k in range(n)]
    vg = kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)
    K = VoxelDrivenConeBP()
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    g = torch.Generator(device="cuda").manual_seed(n)
    y = torch.rand((n, 40, 44), generator=g, device="cuda")
    lay = _native.Layered(n, 40, 44, _native.KK_F32)
    lay.copy_from(y)
    return K, vg, y, lay, g


def _batched(K, vg, lay, vol, update, work, additive):
    pr = (_native.kk_bp_problem * 1)(_native.kk_bp_problem(
        lay.handle, _native.volume_desc(vol), K._params_dev.data_ptr(),
        float(np.float32(vg.voxel_volume())), update, work.data_ptr(),
        int(additive), 0, 0))
    _native.check(_native.load().kk_cone_bp_layered_batched(
        pr, 1, _native.current_stream()))
    return vol


@pytest.mark.parametrize("shape", [(7, 5, 3), (33, 17, 40), (6, 2, 32),
                                   (64, 61, 66)])
@pytest.mark.parametrize("n", [32, 33, 64, 96, 128, 129, 200])
def test_split_equals_one_chunk_per_launch(n, shape):
    K, vg, _, lay, g = _setup(n, shape)
    start = torch.rand(shape, generator=g, device="cuda")
    work = torch.empty(shape, device="cuda")
    none = _native.kk_bp_update(None, None, 0.0, 0.0, 0, 0)
    for additive in (False, True):
        got = start.clone()
        K(lay, got, vg, additive=additive)
        ref = _batched(K, vg, lay, start.clone(), none, work, additive)
        assert torch.equal(got, ref)
    scale = torch.rand(shape, generator=g, device="cuda")
    upd = _native.kk_bp_update(scale.data_ptr(), None, 0.1, 0.0, 1, 0)
    got = start.clone()
    K.update(lay, got, vg, scale, min_value=0.1)
    ref = _batched(K, vg, lay, start.clone(), upd, work, False)
    assert torch.equal(got, ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [64, 130])
def test_split_16bit_volumes(n, dtype):
    """float32 sums, rounded once: the float32 volume's values rounded."""
    K, vg, _, lay, _ = _setup(n, (33, 17, 40))
    ref = torch.empty((33, 17, 40), device="cuda")
    K(lay, ref, vg, additive=False)
    got = torch.empty((33, 17, 40), dtype=dtype, device="cuda")
    K(lay, got, vg, additive=False)
    assert torch.equal(got, ref.to(dtype))
    assert rel_l2(got.float().cpu().numpy(), ref.cpu().numpy()) > 0
