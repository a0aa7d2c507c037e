"""The bounds-tested projection (fewer than 16 sinograms), which takes eight
steps at a time, on walks of a few steps to many and on both sides of its
dispatch by bins (the walk's step selects or branches): bit-identical to the
oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import apirl_b200 as ap  # noqa: E402
from apirl_b200.geometry import ImageGeom, Sino3DGeom  # noqa: E402

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n,nz,n_proj,n_r,rings,max_rd", [
    (1, 1, 7, 5, 1, 0), (2, 3, 9, 8, 2, 1), (5, 2, 11, 9, 3, 2), (9, 1, 33, 21, 1, 0), (40, 5, 30, 61, 4, 1),
    (24, 1, 300, 252, 1, 0), (24, 1, 300, 253, 1, 0), (31, 3, 180, 200, 4, 1)])
def test_project_few_sinograms(oracle, n, nz, n_proj, n_r, rings, max_rd):
    ig = ImageGeom(n, n, nz, 2.0, 2.0, 2.0)
    sg = Sino3DGeom.span1(n_proj, n_r, rings, 1.2 * n, rings * 2.0 * nz / rings, 300.0, max_rd)
    img = np.random.default_rng(n).random(ig.n_voxels, dtype=np.float32) - np.float32(0.3)
    P = ap.SiddonProjector(ig, sg)
    out = P.project(torch.from_numpy(img).to(DEV), torch.empty(P.num_bins(), dtype=torch.float32, device=DEV))
    want = oracle.project_3d(sg, ig, img)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
