"""Backprojection of projections that are staged through a texture (lists
of arrays, permuted and strided arrays, exact weights) against the
device-memory path of the C ABI, at angle counts around the 128-angle
stages; two streams sharing one kernel; calls recorded into a CUDA graph,
which keep the device-memory path."""
from __future__ import annotations

import gc
import math

import numpy as np
import pytest
import torch

import kernelkit as kk
from conftest import rel_l2
from kernelkit import _native
from kernelkit.kernels import VoxelDrivenConeBP, cone_bp
from kernelkit.kernels.cone_fp import interp_code

pytestmark = pytest.mark.gpu

#: float32 rounding of the same samples: the texture unit's and the emulated
#: filter agree to a few ulp of the largest texel
TOL = 1e-6


def _scan(n, shape=(33, 30, 37), rows=41, cols=45):
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.4, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, roll=0.01, pitch=0.02, yaw=2 * math.pi * k / n)
           for k in range(n)]
    return pgs, kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)


def _kernel(pgs, vg, interp, **kw):
    K = VoxelDrivenConeBP(interpolation=interp, **kw)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    return K


def _direct(K, y, vg, start, additive):
    out = start.clone()
    _native.check(_native.load().kk_cone_bp(
        _native.projections_desc(y), _native.volume_desc(out),
        K._params_dev.data_ptr(), float(np.float32(vg.voxel_volume())),
        interp_code(K.interpolation), int(additive), None,
        _native.current_stream()))
    return out


def _layouts(y):
    big = torch.zeros((y.shape[0], y.shape[1] + 3, 2 * y.shape[2]),
                      device="cuda")
    strided = big[:, 2:-1, ::2]
    strided.copy_(y)
    return {"array": (y, (0, 1, 2)),
            "list": ([f.clone() for f in y], (0, 1, 2)),
            "strided": (strided, (0, 1, 2)),
            "columns_first": (y.permute(0, 2, 1).contiguous(), (0, 2, 1)),
            "rows_first": (y.permute(1, 0, 2).contiguous(), (1, 0, 2))}


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("n", [1, 128, 131])
@pytest.mark.parametrize("additive", [False, True])
@pytest.mark.parametrize("layout", ["array", "list", "strided",
                                    "columns_first", "rows_first"])
def test_staged_equals_device_memory(layout, additive, n, interp):
    pgs, vg = _scan(n)
    det = pgs[0].detector
    g = torch.Generator(device="cuda").manual_seed(n)
    y = torch.rand((n, det.rows, det.cols), generator=g, device="cuda")
    start = torch.rand(tuple(int(s) for s in vg.shape), generator=g,
                       device="cuda")
    src, axes = _layouts(y)[layout]
    K = _kernel(pgs, vg, interp, projection_axes=axes)
    got = start.clone()
    K(src, got, vg, additive=additive)
    assert K._stages(_native.projections_desc(y), got)
    ref = _direct(K, y, vg, start, additive)
    assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) <= TOL


@pytest.mark.parametrize("interp", ["texture", "exact"])
def test_border_and_non_finite_texels(interp):
    """Texels at the border and non-finite ones reach the voxels they reach
    from device memory, and no others."""
    pgs, vg = _scan(9, shape=(40, 40, 48), rows=24, cols=20)
    y = torch.zeros((9, 24, 20), device="cuda")
    y[:, 0], y[:, :, -1] = 1.0, 2.0
    y[3, 5, 7] = math.inf
    y[4, 0, 0] = math.nan
    K = _kernel(pgs, vg, interp)
    got = torch.empty((40, 40, 48), device="cuda")
    K([f.clone() for f in y], got, vg, additive=False)
    ref = _direct(K, y, vg, got, False)
    if interp == "exact":  # the same operations on the same four texels
        assert torch.equal(torch.isfinite(got), torch.isfinite(ref))
    fine = torch.isfinite(got) & torch.isfinite(ref)
    assert int(fine.sum()) > 0.9 * fine.numel()
    assert rel_l2(got[fine].cpu().numpy(), ref[fine].cpu().numpy()) <= TOL


def test_two_streams_share_a_kernel():
    pgs, vg = _scan(131)
    det = pgs[0].detector
    K = _kernel(pgs, vg, "texture")
    ys = [torch.rand((131, det.rows, det.cols), device="cuda")
          for _ in range(2)]
    lists = [[f.clone() for f in y] for y in ys]
    outs = [torch.empty((33, 30, 37), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        for s, f, o in zip(streams, lists, outs):
            with torch.cuda.stream(s):
                K(f, o, vg, additive=False)
    torch.cuda.synchronize()
    for y, o in zip(ys, outs):
        ref = _direct(K, y, vg, o, False)
        assert rel_l2(o.cpu().numpy(), ref.cpu().numpy()) <= TOL


def test_textures_are_bounded_and_given_back():
    def go(n, rows):
        pgs, vg = _scan(n, rows=rows)
        K = _kernel(pgs, vg, "texture")
        y = torch.rand((n, rows, 45), device="cuda")
        out = torch.empty((33, 30, 37), device="cuda")
        K(list(y), out, vg, additive=False)
        ref = _direct(K, y, vg, out, False)
        assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= TOL
        return K

    pool = cone_bp._STAGES
    keep = [go(3, 30 + i) for i in range(6)]
    assert len(pool.items) == pool.LIMIT
    keep.append(go(2, 35))  # fewer layers of the last shape
    assert len(pool.items) == pool.LIMIT
    cone_bp.release_staging_textures()
    assert pool.items == []
    keep.append(go(2, 35))
    assert len(pool.items) == 1
    del keep
    gc.collect()
    if not list(pool.users):  # no kernel of another test is alive
        assert pool.items == []


def test_captured_calls_take_the_device_memory_path():
    pgs, vg = _scan(20)
    det = pgs[0].detector
    K = _kernel(pgs, vg, "texture")
    cone_bp.release_staging_textures()
    y = torch.rand((20, det.rows, det.cols), device="cuda")
    out = torch.zeros((33, 30, 37), device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        K(y, out, vg, additive=False)
    assert cone_bp._STAGES.items == []
    g.replay()
    assert torch.equal(out, _direct(K, y, vg, out, False))


def test_small_volumes_keep_the_device_memory_path():
    pgs, vg = _scan(5, shape=(4, 5, 6), rows=60, cols=80)
    K = _kernel(pgs, vg, "exact")
    cone_bp.release_staging_textures()
    y = torch.rand((5, 60, 80), device="cuda")
    out = torch.empty((4, 5, 6), device="cuda")
    K(y, out, vg, additive=False)
    assert cone_bp._STAGES.items == []
    assert torch.equal(out, _direct(K, y, vg, out, False))
