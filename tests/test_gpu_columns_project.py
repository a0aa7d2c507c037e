"""Projections on the column walk (csrc/columns.cu, k_project_cols), whole and
subset, bit-identical to the oracle: a half-empty warp, a remainder of one lane,
nx != ny, rays that miss the image, z crossings closer than a batch of steps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import apirl_b200 as ap  # noqa: E402
from column_cases import PROJECTED  # noqa: E402

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("name", sorted(PROJECTED))
def test_projection_against_oracle(oracle, name):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ig, sg, sub, nsub = PROJECTED[name]
    img = (np.random.default_rng(7).random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    x = torch.from_numpy(img).to(DEV)
    P = ap.SiddonProjector(ig, sg)
    for s, n in ((-1, 1), (sub, nsub)):
        want = oracle.project_3d(sg, ig, img, s, n)
        out = torch.full((want.size,), float("nan"), dtype=torch.float32, device=DEV)
        P.project(x, out, s, n)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
