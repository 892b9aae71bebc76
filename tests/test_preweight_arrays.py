"""Pre-weighting parameters of a whole list of geometries at once: bit for
bit those of one geometry after the other, for float32 and float64 vectors,
and only for plain lists of one detector."""
from __future__ import annotations

import numpy as np
import pytest

import kernelkit as kk
from cases import CASES
from helpers import build_case
from kernelkit import processing


def _one_by_one(geoms, monkeypatch):
    with monkeypatch.context() as m:
        m.setattr(processing, "_preweight_arrays", lambda g: None)
        return processing.preweight_params(geoms)


@pytest.mark.parametrize("case", sorted(CASES))
def test_arrays_equal_one_by_one(case, monkeypatch):
    pgs, _ = build_case(case)
    f32 = [kk.ProjectionGeometry(g.source_position, g.detector_position,
                                 g.detector, u=g.u, v=g.v) for g in pgs]
    for geoms in (pgs, f32, tuple(pgs), pgs[:1]):
        got = processing._preweight_arrays(geoms)
        assert got is not None
        assert np.array_equal(got, _one_by_one(geoms, monkeypatch))


def test_other_forms_go_one_by_one(monkeypatch):
    pgs, _ = build_case("small")
    det = pgs[0].detector
    assert processing._preweight_arrays([]) is None
    assert processing._preweight_arrays(
        kk.ProjectionGeometrySequence.fromList(pgs)) is None
    mixed = list(pgs)
    mixed[1] = kk.ProjectionGeometry(
        pgs[1].source_position, pgs[1].detector_position, det, u=pgs[1].u,
        v=pgs[1].v)  # float32 among float64
    other = list(pgs)
    other[2] = kk.ProjectionGeometry(
        pgs[2].source_position, pgs[2].detector_position,
        kk.Detector(det.rows, det.cols, 2.0 * det.pixel_height,
                    det.pixel_width))
    scalar = [kk.ProjectionGeometry(
        g.source_position, g.detector_position,
        kk.Detector(det.rows, det.cols, np.float64(1.1), 1.1)) for g in pgs]
    for geoms in (mixed, other, scalar):
        assert processing._preweight_arrays(geoms) is None
        assert np.array_equal(processing.preweight_params(geoms),
                              _one_by_one(geoms, monkeypatch))
