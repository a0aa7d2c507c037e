"""Geometries whose projections take the column walk, the whole and the subset
(the dispatch's estimate, csrc/capi.cu, project_cols; tests/test_host_calls.py
checks that they do): name -> image, sinogram, subset, subsets."""
from apirl_b200.geometry import ImageGeom, Sino3DGeom

PROJECTED = {
    "16 sinograms": (ImageGeom(160, 160, 31, 2.0, 2.0, 2.0), Sino3DGeom.span1(24, 200, 16, 200.0, 16 * 4.0, 400.0, 0), 1, 2),
    "33 sinograms, not square": (ImageGeom(96, 64, 66, 2.0, 2.0, 2.0), Sino3DGeom.span1(50, 80, 33, 80.0, 33 * 4.0, 250.0, 0), 1, 2),
    "97 sinograms, subset of 3": (ImageGeom(72, 90, 41, 2.0, 2.0, 2.0), Sino3DGeom.span1(30, 70, 21, 70.0, 21 * 4.0, 250.0, 2), 2, 3),
    "rays past the image": (ImageGeom(64, 48, 128, 2.0, 2.0, 2.0), Sino3DGeom.span1(40, 160, 64, 160.0, 64 * 4.0, 250.0, 0), 0, 2),
    "steep": (ImageGeom(48, 48, 160, 4.0, 4.0, 0.5), Sino3DGeom.span1(64, 60, 8, 120.0, 80.0, 150.0, 7), 1, 2),
}
