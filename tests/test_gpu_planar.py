"""The 2D pass on its padded layouts (csrc/planar.cu) at the sizes where it
can go wrong, against the oracle: sides around a tile's 32 and 8 and a batch's
8 segments, slices of one row or column (rays outside the image: the
bounds-tested walk), a bin count that leaves a part warp, one bin, subsets.
Updated image rel L2 <= 1e-5 (fp32 atomics in another order), FP64 likelihood
against the FP64 sum of the oracle's float estimates 1e-9."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import apirl_b200 as ap  # noqa: E402
from apirl_b200.geometry import ImageGeom, Sino2DGeom  # noqa: E402

DEV = torch.device("cuda:0")


def t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ap.load_library()


@pytest.mark.parametrize("nx,ny,n_proj,n_r", [(32, 32, 20, 33), (33, 31, 7, 64), (9, 8, 5, 31), (65, 7, 11, 40),
                                              (1, 24, 9, 16), (40, 1, 9, 16), (4, 4, 1, 1), (130, 130, 6, 190)])
@pytest.mark.parametrize("dtype", [np.float32, np.uint16])
def test_pass_against_oracle(oracle, nx, ny, n_proj, n_r, dtype):
    ig = ImageGeom(nx, ny, 1, 2.0, 2.0, 1.0)
    sg = Sino2DGeom(n_proj, n_r, 1.1 * max(nx, ny), 400.0)
    rng = np.random.default_rng(nx * 1000 + ny)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    est = oracle.project_2d(sg, ig, x0)
    meas = rng.poisson(est * 2 + 0.3).astype(dtype)
    sens = (rng.random(ig.n_voxels, dtype=np.float32) + 1).astype(np.float32)
    P = ap.SiddonProjector(ig, sg)
    m = meas.astype(np.float32)
    want = oracle.update(x0, oracle.backproject_2d(sg, ig, oracle.inverse_divide(m, est)), sens, np.float32(0), False)
    pos = est > 0
    e64 = est[pos].astype(np.float64)
    want_lik = float(np.sum(m[pos] * np.log(e64) - e64))
    for _ in range(2):  # the sums are zero again after a pass
        x, bp = t(x0), torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV)
        lik = torch.zeros(1, dtype=torch.float64, device=DEV)
        P.em_pass(t(meas), x, bp, t(sens), ge=False, lik=lik)
        assert rel(x.cpu().numpy(), want) <= 1e-5
        assert abs(lik.item() - want_lik) <= 1e-9 * abs(want_lik) + 1e-12
        assert not bp.any()
    # the backprojected ratio alone, added to what bp holds, and over subsets
    ratio = oracle.backproject_2d(sg, ig, oracle.inverse_divide(m, est))
    bp = t(x0)
    for s in range(min(2, n_proj)):
        P.em_project_backproject(t(meas), t(x0), bp, s, min(2, n_proj))
    assert rel(bp.cpu().numpy(), x0 + ratio) <= 1e-5


def test_image_of_several_slices(oracle):
    """A 2D pass over a two-slice image: the rays cross the first slice; the
    other has no backprojection, so its update is x * 0 / sens = 0."""
    ig, sg = ImageGeom(33, 31, 2, 2.0, 2.0, 1.0), Sino2DGeom(16, 40, 40.0, 400.0)
    one = ImageGeom(33, 31, 1, 2.0, 2.0, 1.0)
    n = one.n_voxels
    rng = np.random.default_rng(3)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    sens = (rng.random(ig.n_voxels, dtype=np.float32) + 1).astype(np.float32)
    est = oracle.project_2d(sg, one, x0[:n])
    meas = rng.poisson(est * 2 + 0.3).astype(np.float32)
    want = oracle.update(x0[:n], oracle.backproject_2d(sg, one, oracle.inverse_divide(meas, est)), sens[:n],
                         np.float32(0), False)
    P = ap.SiddonProjector(ig, sg)
    x = t(x0)
    P.em_pass(t(meas), x, torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV), t(sens), ge=False)
    got = x.cpu().numpy()
    assert rel(got[:n], want) <= 1e-5
    assert not got[n:].any()


def test_pass_with_additive_term(oracle):
    """An additive term in the counts' layout, whole and packed to a subset."""
    ig, sg = ImageGeom(33, 40, 1, 2.0, 2.0, 1.0), Sino2DGeom(21, 47, 44.0, 400.0)
    rng = np.random.default_rng(4)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    sens = (rng.random(ig.n_voxels, dtype=np.float32) + 1).astype(np.float32)
    whole = rng.poisson(4.0, 21 * 47).astype(np.float32)
    add = (rng.random(21 * 47, dtype=np.float32) + 0.1).astype(np.float32)
    P = ap.SiddonProjector(ig, sg)
    for sub, nsub, packed in ((-1, 1, False), (1, 3, False), (1, 3, True)):
        pick = lambda v: v.reshape(21, 47)[max(sub, 0)::nsub].reshape(-1)
        est = pick((oracle.project_2d(sg, ig, x0) + add).astype(np.float32))
        m = pick(whole)
        ratio = np.zeros((21, 47), np.float32)  # the other subsets' bins add nothing
        ratio[max(sub, 0)::nsub] = oracle.inverse_divide(m, est).reshape(-1, 47)
        bp = oracle.backproject_2d(sg, ig, ratio.reshape(-1))
        want = oracle.update(x0, bp, sens, np.float32(0), False)
        e64 = est[est > 0].astype(np.float64)
        want_lik = float(np.sum(m[est > 0] * np.log(e64) - e64))
        x, lik = t(x0), torch.zeros(1, dtype=torch.float64, device=DEV)
        a, c = (pick(add), m) if packed else (add, whole)
        P.em_pass(t(c), x, torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV), t(sens), sub, nsub, add=t(a),
                  ge=False, counts_packed=packed, lik=lik)
        assert rel(x.cpu().numpy(), want) <= 1e-5
        assert abs(lik.item() - want_lik) <= 1e-9 * abs(want_lik)
