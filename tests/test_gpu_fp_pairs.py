"""Paired rays of the padded forward projector: exact weights, detectors
whose rows do not share their in-slice coordinate (tilted), and last row
tiles of at most 32 rows (two columns per thread), against the unpadded
projector, over ray directions, layouts, storage types, slice
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


def _project(kind, interp, padded, vol, axes, span=None, tex=True, rows=70,
             cols=41, residual=None):
    pgs = _scan(kind, rows=rows, cols=cols)
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
    if residual is None:
        K(vol, pgs, vg, out, additive=False)
    else:
        K.residual(vol, pgs, vg, out, *residual)
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


@pytest.mark.parametrize("kind", ["circular", "tilted", "alldirs"])
@pytest.mark.parametrize("rows,cols", [(1, 9), (32, 8), (33, 12), (64, 5),
                                       (65, 4), (96, 13), (961, 7),
                                       (1025, 7)])
def test_last_row_tiles(rows, cols, kind):
    vol = _volume((24, 26, 40))
    for interp in ("texture", "exact"):
        _same(kind, interp, vol, rows=rows, cols=cols)
    y, w = (torch.rand((14, rows, cols), device="cuda") for _ in range(2))
    _same(kind, "texture", vol, rows=rows, cols=cols, residual=(y, w),
          span=16)


def test_batched_padded_copies():
    """kk_cone_fp_batched_ex from padded copies gives the unpadded launches'
    projections bit for bit, and keeps to the volumes when one problem has
    no copy."""
    import ctypes

    from kernelkit import _native

    L = _native.load()
    jobs = []
    for n, rows, cols in ((21, 40, 30), (40, 70, 61), (33, 64, 9)):
        pgs = _scan("circular", n=9, rows=rows, cols=cols)
        vg = kk.resolve_volume_geometry(shape=n, voxel_size=1.0)
        K = RayDrivenConeFP()
        K.compile()
        K.set_params(K.geoms2params(pgs, vg))
        jobs.append((K, _volume((n, n, n)), (9, rows, cols), vg))

    def run(options):
        outs = [torch.zeros(s, device="cuda") for _, _, s, _ in jobs]
        pr = (_native.kk_fp_problem * len(jobs))()
        keep = []
        for q, (K, vol, _, vg), out in zip(pr, jobs, outs):
            q.vol = _native.volume_desc(vol)
            q.proj = _native.projections_desc(out)
            q.angles = K._params_dev.data_ptr()
            q.out_scale[:] = [float(v) for r in K._output_scale(vg.voxel_size)
                              for v in r]
            lay = _native.Layered(*vol.shape, _native.KK_F32)
            lay.copy_from(vol)
            keep.append(lay)
            q.vtex = lay.handle
            q.span = 16
        _native.check(L.kk_cone_fp_batched_ex(
            pr, len(jobs), _native.KK_INTERP_TEX8, 16, options,
            _native.current_stream()))
        torch.cuda.synchronize()
        return outs

    def options(skip=None):
        pads = [K._padded(_native.volume_desc(v)) for K, v, _, _ in jobs]
        ptr = (ctypes.c_void_p * 3)(*[None if i == skip else p
                                      for i, (p, _) in enumerate(pads)])
        return _native.kk_fp_batch_options(
            ptr, (ctypes.c_int64 * 3)(*[e for _, e in pads]))

    ref = run(None)
    assert all(float(r.abs().sum()) > 0 for r in ref)
    for o in (options(), options(skip=1)):
        for a, b in zip(run(o), ref):
            assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["circular", "tilted"])
@pytest.mark.parametrize("shape,floats", [((33, 47, 38), True),
                                          ((257, 20, 18), False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_float_copies_of_16bit_volumes(dtype, shape, floats, kind):
    """16-bit storage runs (half_texture): a float32 padded copy up to 256
    slices, the volume's type beyond, and the unpadded projections bit for
    bit, plain and with the residual epilogue."""
    vol = _volume(shape, dtype)
    vg = kk.resolve_volume_geometry(shape=shape, voxel_size=1.0)
    pgs = _scan(kind, rows=44, cols=23)
    y, w = (torch.rand((14, 44, 23), device="cuda").half() for _ in range(2))
    outs = []
    for padded in (True, False):
        K = RayDrivenConeFP()
        K.half_texture, K.padded_copy = True, padded
        K.compile()
        K.set_params(K.geoms2params(pgs, vg))
        out = torch.zeros_like(y)
        K(vol, pgs, vg, out, additive=False)
        res = torch.zeros_like(y)
        K.residual(vol, pgs, vg, res, y, w)
        outs.append((out, res))
        if padded:
            want = torch.float32 if floats else dtype
            assert K._pad_buf.dtype == want
    assert float(outs[0][0].abs().sum()) > 0
    assert torch.equal(outs[0][0], outs[1][0])
    assert torch.equal(outs[0][1], outs[1][1])
