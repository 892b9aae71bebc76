"""One projector used from several streams and threads: its workspaces (the
volume texture, the padded copy, the adjoint's ray set-ups) belong to one
call at a time. Calls recorded into CUDA graphs."""
from __future__ import annotations

import copy
import math
import threading

import pytest
import torch

import kernelkit as kk
from kernelkit.kernels import RayDrivenConeFP

pytestmark = pytest.mark.gpu

N, ANGLES, PIXELS = 96, 20, 140


def _projector(interp, n=N):
    det = kk.Detector(rows=PIXELS, cols=PIXELS, pixel_height=1.3,
                      pixel_width=1.3)
    g0 = kk.ProjectionGeometry([-200.0, 0.0, 0.0], [200.0, 0.0, 0.0], det)
    pgs = [kk.rotate(g0, yaw=0.1 + 2 * math.pi * k / ANGLES)
           for k in range(ANGLES)]
    vg = kk.resolve_volume_geometry(shape=n, voxel_size=1.0)
    K = RayDrivenConeFP(interpolation=interp)
    K.compile()
    K.set_params(K.geoms2params(pgs, vg))
    return K, pgs, vg


def _volumes(count):
    g = torch.Generator(device="cuda").manual_seed(3)
    return [torch.rand((N, N, N), generator=g, device="cuda") * (i + 1)
            for i in range(count)]


def _out():
    return torch.empty((ANGLES, PIXELS, PIXELS), device="cuda")


@pytest.mark.parametrize("interp", ["texture", "exact"])
@pytest.mark.parametrize("threads", [False, True])
def test_streams_and_threads_share_a_projector(interp, threads):
    K, pgs, vg = _projector(interp)
    volumes = _volumes(3)
    expect = []
    for x in volumes:
        y = _out()
        K(x, pgs, vg, y, additive=False)
        v = torch.empty_like(x)
        K.transpose(y, pgs, vg, v)
        expect.append((y, v))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in volumes]
    got = [[] for _ in volumes]

    def work(i, rounds):
        with torch.cuda.stream(streams[i]):
            for _ in range(rounds):
                y, v = _out(), torch.empty_like(volumes[i])
                K(volumes[i], pgs, vg, y, additive=False)
                K.transpose(expect[i][0], pgs, vg, v)
                got[i].append((y, v))

    if threads:
        pool = [threading.Thread(target=work, args=(i, 6)) for i in range(3)]
        for p in pool:
            p.start()
        for p in pool:
            p.join()
    else:
        for _ in range(6):
            for i in range(3):
                work(i, 1)
    torch.cuda.synchronize()
    for pairs, (y0, v0) in zip(got, expect):
        assert len(pairs) == 6
        for y, v in pairs:
            assert torch.equal(y, y0)
            assert torch.equal(v, v0)


@pytest.mark.parametrize("interp", ["texture", "exact"])
def test_threads_on_one_stream(interp):
    K, pgs, vg = _projector(interp)
    volumes = _volumes(3)
    expect = []
    for x in volumes:
        expect.append(_out())
        K(x, pgs, vg, expect[-1], additive=False)
    got = [[_out() for _ in range(8)] for _ in volumes]

    def work(i):
        for y in got[i]:
            K(volumes[i], pgs, vg, y, additive=False)

    pool = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    torch.cuda.synchronize()
    for ys, y0 in zip(got, expect):
        for y in ys:
            assert torch.equal(y, y0)


def test_recorded_exact_calls_keep_no_workspace():
    """The graph owns all that it uses: other calls of the projector do not
    reach it, nor does the projector's end."""
    K, pgs, vg = _projector("exact")
    (x, other), y, z = _volumes(2), _out(), _out()
    K(other, pgs, vg, z, additive=False)  # the padded copy exists
    K.padded_copy = False
    expect = _out()
    K(x, pgs, vg, expect, additive=False)
    K.padded_copy = True
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        K(x, pgs, vg, y, additive=False)
    K._pad_buf.fill_(float("nan"))
    g.replay()
    assert torch.equal(y, expect)


def test_solver_graphs_keep_the_padded_copy():
    K, pgs, vg = _projector("exact")
    x, = _volumes(1)
    y = _out()
    K(x, pgs, vg, y, additive=False)
    s = kk.SIRT(y, pgs, vg, interpolation="exact")
    assert s.fp.single_owner
    s.run(2)
    twin = kk.SIRT(y, pgs, vg, interpolation="exact")
    twin.run(2, use_graph=False)
    assert torch.equal(s.x, twin.x)


def test_copies_and_lifetime():
    """Copies share the workspaces and the turns; a projector is freed with
    its last reference."""
    import weakref

    K, pgs, vg = _projector("exact")
    x, = _volumes(1)
    y, z = _out(), _out()
    K(x, pgs, vg, y, additive=False)
    twin = copy.copy(K)
    assert twin._turns is K._turns
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        twin(x, pgs, vg, z, additive=False)
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    deep = copy.deepcopy(K)
    assert deep._turns is not K._turns
    deep(x, pgs, vg, z, additive=False)
    assert torch.equal(y, z)
    gone = weakref.ref(K)
    del K, twin
    assert gone() is None
