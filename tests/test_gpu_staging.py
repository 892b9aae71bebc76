"""Staging textures of the backprojection: the tiles that exact weights
gather from, no memory for a texture, a graph being recorded on another
stream, textures that have to go while they are in use, copied kernels."""
from __future__ import annotations

import copy
import gc
import math

import numpy as np
import pytest
import torch

import kernelkit as kk
from kernelkit import _native
from kernelkit.algo import capture_graph
from kernelkit.kernels import VoxelDrivenConeBP, cone_bp
from kernelkit.kernels.cone_fp import interp_code

pytestmark = pytest.mark.gpu

SHAPE = (33, 30, 37)


def _case(n, interp="texture", rows=41, cols=45):
    """(kernel, volume geometry, projections)."""
    det = kk.Detector(rows=rows, cols=cols, pixel_height=1.4, pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-90.0, 0.0, 0.0], [70.0, 1.0, 2.0], det)
    pgs = [kk.rotate(g0, roll=0.01, pitch=0.02, yaw=2 * math.pi * k / n)
           for k in range(n)]
    vg = kk.resolve_volume_geometry(shape=SHAPE, voxel_size=1.0)
    K = VoxelDrivenConeBP(interpolation=interp)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    g = torch.Generator(device="cuda").manual_seed(n)
    return K, vg, torch.rand((n, rows, cols), generator=g, device="cuda")


def _direct(K, y, vg):
    """The device-memory path of the C ABI."""
    out = torch.empty(SHAPE, device="cuda")
    _native.check(_native.load().kk_cone_bp(
        _native.projections_desc(y), _native.volume_desc(out),
        K._params_dev.data_ptr(), float(np.float32(vg.voxel_volume())),
        interp_code(K.interpolation), 0, None, _native.current_stream()))
    return out


class _NoMemory:
    """A texture that no GPU has the memory for (2.2 TB): the allocation
    itself fails, with the runtime's own error."""

    def __new__(cls, *shape_and_dtype):
        return _native.Layered(2048, 16383, 16383, _native.KK_F32)


def test_failed_creation_leaves_no_error_behind():
    K, vg, y = _case(5)
    with pytest.raises(_native.KernelKitError):
        _NoMemory()
    out = torch.empty(SHAPE, device="cuda")
    _native.check(_native.load().kk_cone_bp(
        _native.projections_desc(y), _native.volume_desc(out),
        K._params_dev.data_ptr(), 1.0, _native.KK_INTERP_TEX8, 0, None,
        _native.current_stream()))


@pytest.mark.parametrize("interp", ["texture", "exact"])
def test_no_memory_for_a_texture(interp, monkeypatch):
    """The projections are then read from device memory."""
    K, vg, y = _case(40, interp)
    cone_bp.release_staging_textures()

    class Native:
        def __getattr__(self, name):
            return (_NoMemory if name in ("Layered", "Gather")
                    else getattr(_native, name))

    monkeypatch.setattr(cone_bp, "_native", Native())
    out = torch.empty(SHAPE, device="cuda")
    K([f.clone() for f in y], out, vg, additive=False)
    assert cone_bp._STAGES.items == []
    assert torch.equal(out, _direct(K, y, vg))


def _same(a, b):
    nan = torch.isnan(a)
    return (torch.equal(nan, torch.isnan(b))
            and torch.equal(a[~nan], b[~nan]))


@pytest.mark.parametrize("n,rows,cols", [
    (1, 1, 1), (33, 2, 45), (131, 400, 23),  # 2 tiles to a row of the array
    (40, 41, 1500), (97, 700, 301)])
def test_gather_tiles(n, rows, cols):
    """The same operations on the same texels as from device memory, bit for
    bit; frames of infinities, NaNs and the largest values next to each
    other stay where they are."""
    K, vg, y = _case(n, "exact", rows, cols)
    y[1::5], y[2::7], y[3::11] = math.inf, math.nan, 3e38
    y[0, 0], y[0, -1], y[0, :, 0], y[0, :, -1] = 1.0, 2.0, 3.0, 4.0
    K._stages = lambda *a: True  # also where the copy does not pay
    out = torch.empty(SHAPE, device="cuda")
    cone_bp.release_staging_textures()
    K(y, out, vg, additive=False)
    assert [type(i["texture"]) for i in cone_bp._STAGES.items] == [
        _native.Gather]
    assert _same(out, _direct(K, y, vg))


@pytest.mark.parametrize("n", [20, 131])
def test_frames_too_large_for_gathers(n, monkeypatch):
    """Staged in a layered texture, whose texels are read one by one."""
    with pytest.raises(NotImplementedError):
        _native.Gather(1000, 16000, 16000)
    K, vg, y = _case(n, "exact")
    y[1::5], y[0, 0], y[0, :, -1] = math.inf, 1.0, 4.0

    class Native:
        class Gather:
            def __init__(self, *shape):
                raise NotImplementedError

        def __getattr__(self, name):
            return getattr(_native, name)

    cone_bp.release_staging_textures()
    monkeypatch.setattr(cone_bp, "_native", Native())
    out = torch.empty(SHAPE, device="cuda")
    K(y, out, vg, additive=False)
    assert len(cone_bp._STAGES.items) == 1
    assert _same(out, _direct(K, y, vg))


def test_other_streams_while_a_graph_is_recorded():
    """Textures are made, looked for, evicted and given back on one stream
    while another one is recorded; the recording goes on."""
    cases = [_case(9, "exact", rows=20 + r) for r in range(6)]
    outs = [torch.empty(SHAPE, device="cuda") for _ in cases]
    x = torch.zeros(1000, device="cuda")
    side = [torch.cuda.Stream() for _ in range(2)]
    cone_bp.release_staging_textures()
    torch.cuda.synchronize()

    def work():
        x.add_(1.0)
        for s in side:
            with torch.cuda.stream(s):
                for (K, vg, y), o in zip(cases, outs):
                    K(y, o, vg, additive=False)
        cone_bp.release_staging_textures()
        x.mul_(2.0)

    g = capture_graph(work)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, torch.full_like(x, 6.0))
    for (K, vg, y), o in zip(cases, outs):
        assert torch.equal(o, _direct(K, y, vg))


def test_textures_collected_while_a_graph_is_recorded():
    """An operator's texture that the garbage collector frees in the middle
    of a recording does not end it."""
    x = torch.zeros(1000, device="cuda")
    gc.collect()

    class Owner:
        def __init__(self):
            self.texture = _native.Layered(64, 64, 64, _native.KK_F32)
            self.gather = _native.Gather(64, 64, 64)
            self.cycle = self

    def work():
        x.add_(1.0)
        assert gc.collect() > 0
        x.mul_(2.0)

    Owner()
    torch.cuda.synchronize()
    g = capture_graph(work)
    g.replay()
    assert torch.equal(x, torch.full_like(x, 2.0))


@pytest.mark.parametrize("way", ["evicted", "released", "last kernel gone"])
def test_textures_in_use_are_waited_for(way, monkeypatch):
    """No texture is freed before the kernels that sample it are done."""
    pool = cone_bp._StagePool()
    monkeypatch.setattr(cone_bp, "_STAGES", pool)
    ended, busy = [], torch.cuda.Stream()
    destroy = _native.Layered.__del__

    def log(texture):
        if id(texture) in events:
            ended.append(events[id(texture)].query())
        destroy(texture)

    cases = [_case(3, rows=20 + r) for r in range(pool.LIMIT)]
    extra = _case(3, rows=40)
    out = torch.empty(SHAPE, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        for K, vg, y in cases:
            torch.cuda._sleep(10_000_000)  # some milliseconds
            K(y.permute(0, 2, 1).contiguous().permute(0, 2, 1), out, vg)
    events = {id(i["texture"]): i["used"] for i in pool.items}
    assert len(events) == pool.LIMIT
    monkeypatch.setattr(_native.Layered, "__del__", log)
    if way == "evicted":
        K, vg, y = extra
        K(y, torch.empty(SHAPE, device="cuda"), vg)
    elif way == "released":
        cone_bp.release_staging_textures()
    else:
        # (the pool is told of the kernels it has seen in use)
        del K, y, extra
        cases.clear()
        gc.collect()
        assert pool.items == []
    assert ended == [True] * (1 if way == "evicted" else pool.LIMIT)
    monkeypatch.setattr(_native.Layered, "__del__", destroy)
    torch.cuda.synchronize()


def test_copied_kernels_keep_the_textures(monkeypatch):
    pool = cone_bp._StagePool()
    monkeypatch.setattr(cone_bp, "_STAGES", pool)
    K, vg, y = _case(7, "exact")
    out = torch.empty(SHAPE, device="cuda")
    twin = copy.copy(K)
    K(y, out, vg, additive=False)
    twin(y, out, vg, additive=False)
    del K
    gc.collect()
    assert len(pool.items) == 1  # the copy is a user of its own
    assert torch.equal(out, _direct(twin, y, vg))
    del twin
    gc.collect()
    assert pool.items == []


def test_an_error_in_between_is_no_lost_use(monkeypatch):
    """A call that fails after it has filled the texture still counts as
    its use."""
    pool = cone_bp._StagePool()
    monkeypatch.setattr(cone_bp, "_STAGES", pool)
    K, vg, y = _case(5)
    frames = [f.clone() for f in y]
    out = torch.empty(SHAPE, device="cuda")
    K(frames, out, vg)
    item, = pool.items
    torch.cuda.synchronize()

    class Library:
        def __getattr__(self, name):
            if name == "kk_cone_bp_layered_ex":
                return lambda *args: _native.KK_ERR_UNSUPPORTED
            return getattr(_native.load(), name)

    class Native:
        load = Library

        def __getattr__(self, name):
            return getattr(_native, name)

    monkeypatch.setattr(cone_bp, "_native", Native())
    torch.cuda._sleep(100_000_000)
    with pytest.raises(NotImplementedError):
        K(frames, out, vg)
    assert not item["used"].query()
    torch.cuda.synchronize()


def test_given_back_when_there_is_no_memory_for_another_texture():
    K, vg, y = _case(5, "exact")
    out = torch.empty(SHAPE, device="cuda")
    K(y, out, vg)
    assert cone_bp._STAGES.items
    made = []

    def create(handle):  # fails as long as the pool keeps something
        made.append(len(cone_bp._STAGES.items))
        return _native.KK_ERR_CUDA if made[-1] else _native.KK_OK

    _native._create(create)
    assert len(made) == 2 and made[-1] == 0
    K(y, out, vg, additive=False)
    assert torch.equal(out, _direct(K, y, vg))


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("strides", [(41, 1, 1), (41 * 3, 3, 1), (7, 2, 1),
                                     (2, 1, 3)])
def test_overlapping_frames(strides, interp):
    """Sliding windows over one row, whose rows overlap, are projections
    like any others."""
    K, vg, y = _case(9, interp)
    y = y.reshape(-1).as_strided((9, 41, 45), strides)
    K._layered_source = lambda textures: None
    out = torch.empty(SHAPE, device="cuda")
    K(y, out, vg, additive=False)
    ref = _direct(K, y, vg)
    assert (out - ref).norm() <= 1e-6 * ref.norm()
