"""The listed pass's three ways to walk a LOR's bins with counts (csrc/columns.cu:
the block that lists the crossings, the small blocks of LORs with few counts,
a lane a bin) against the oracle: sinogram counts around a warp and the window
in which a block looks for counts, LORs past the image and with their corners
outside it, every count type, an additive term, subsets.  Updated image rel L2
<= 1e-5 (fp32 atomics in another order), likelihood 1e-6 (the rounding of the
image dot product)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import apirl_b200 as ap  # noqa: E402
from apirl_b200 import _lib  # noqa: E402
from apirl_b200.geometry import ImageGeom, Sino3DGeom  # noqa: E402

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


# rings, largest ring difference, angles, r, subsets, and the share of bins with counts
LANES = [(16, 0, 100, 90, 1), (33, 0, 170, 100, 2), (17, 8, 102, 90, 1), (33, 4, 100, 90, 1)]
SMALL = [(33, 4, 40, 50, 1), (45, 44, 33, 50, 1)]
WINDOWS = [(46, 45, 6, 24, 1), (64, 63, 5, 24, 1)]


@pytest.mark.parametrize("rings,max_rd,n_proj,n_r,nsub", LANES + SMALL + WINDOWS)
@pytest.mark.parametrize("share,dtype,with_add", [(0.004, np.uint16, False), (0.1, np.uint32, True), (0.6, np.float32, False)])
def test_listed_pass(oracle, rings, max_rd, n_proj, n_r, nsub, share, dtype, with_add):
    ig = ImageGeom(27, 24, 2 * rings - 1, 2.5, 2.5, 2.0)
    sg = Sino3DGeom.span1(n_proj, n_r, rings, 45.0, rings * 4.0, 120.0, max_rd)
    rng = np.random.default_rng(rings * 100 + int(share * 100))
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    sub = nsub - 1 if nsub > 1 else -1
    counts = (rng.random(sg.n_bins) < share) * (1 + rng.poisson(2.0, sg.n_bins))
    meas = counts.astype(dtype)
    pick = lambda v: v.reshape(sg.n_sinos, n_proj, n_r)[:, max(sub, 0)::nsub, :].reshape(-1)
    m = pick(meas).astype(np.float32)
    est = oracle.project_3d(sg, ig, x0, sub, nsub)
    add = (rng.random(sg.n_bins, dtype=np.float32) + 0.5).astype(np.float32) if with_add else None
    if with_add:
        est = (est + pick(add)).astype(np.float32)
    sens = (rng.random(ig.n_voxels, dtype=np.float32) + 1).astype(np.float32)
    bp = oracle.backproject_3d(sg, ig, oracle.inverse_divide(m, est), sub, nsub, threads=1)
    want = oracle.update(x0, bp, sens, np.float32(0), True)
    nz = est != 0
    e64 = est[nz].astype(np.float64)
    want_lik = float(np.sum(m[nz] * np.log(e64) - e64))
    P = ap.SiddonProjector(ig, sg)
    P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
    zeros = lambda: torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV)
    G = P.backproject_ones(zeros(), sub, nsub)
    less = torch.tensor([float(np.sum(pick(add), dtype=np.float64))], dtype=torch.float64, device=DEV) if with_add else None
    for _ in range(2):  # the sums and the queue are empty again after a pass
        x, lik = t(x0), torch.zeros(1, dtype=torch.float64, device=DEV)
        P.em_pass_sparse(t(meas), x, zeros(), t(sens), G, sub, nsub, lik=lik, add=t(add) if with_add else None, zero_add=less)
        assert rel(x.cpu().numpy(), want) <= 1e-5
        assert abs(lik.item() - want_lik) <= 1e-6 * max(abs(want_lik), float(np.sum(e64)))


@pytest.mark.parametrize("rings,max_rd,n_proj,n_r,nsub", LANES + [(16, 7, 100, 90, 1), (33, 4, 40, 50, 1)])
@pytest.mark.parametrize("share", [0.0, 0.01, 0.3, 1.0])
def test_backprojection_of_few_values(oracle, rings, max_rd, n_proj, n_r, nsub, share):
    """A backprojection leaves LORs without values: empty, sparse and full
    sinograms (256 of them and more), twice, added to what the image holds."""
    ig = ImageGeom(27, 24, 2 * rings - 1, 2.5, 2.5, 2.0)
    sg = Sino3DGeom.span1(n_proj, n_r, rings, 45.0, rings * 4.0, 120.0, max_rd)
    rng = np.random.default_rng(rings)
    sub = nsub - 1 if nsub > 1 else -1
    P = ap.SiddonProjector(ig, sg)
    n = P.num_bins(sub, nsub)
    v = ((rng.random(n, dtype=np.float32) + 0.5) * (rng.random(n) < share)).astype(np.float32)
    want = oracle.backproject_3d(sg, ig, v, sub, nsub, threads=1)
    x0 = rng.random(ig.n_voxels, dtype=np.float32)
    for _ in range(2):
        got = P.backproject(t(v), t(x0), sub, nsub).cpu().numpy().astype(np.float64)
        if not v.any():
            assert np.array_equal(got, x0)
        else:
            assert np.linalg.norm(got - (x0.astype(np.float64) + want)) <= 1e-5 * np.linalg.norm(want) + 1e-6


@pytest.mark.parametrize("rings", [16, 33])
@pytest.mark.parametrize("share", [0.01, 0.3, 1.0])
def test_long_backprojection_of_few_values(oracle, rings, share):
    """Calls so long that the bins of LORs with up to 8 values are queued, some
    of them past the image, beside LORs with more; twice."""
    ig = ImageGeom(200, 190, 5, 2.0, 2.0, 2.0)
    sg = Sino3DGeom.span1(116, 230, rings, 230.0, rings * 0.7, 400.0, 0)
    rng = np.random.default_rng(rings)
    v = ((rng.random(sg.n_bins, dtype=np.float32) + 0.5) * (rng.random(sg.n_bins) < share)).astype(np.float32)
    want = oracle.backproject_3d(sg, ig, v, threads=1)
    P = ap.SiddonProjector(ig, sg)
    for _ in range(2):
        got = P.backproject(t(v), torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV)).cpu().numpy()
        assert rel(got, want) <= 1e-5


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("rings,max_rd,n_proj,n_r,nsub", [LANES[1], LANES[3], SMALL[0]])
def test_zero_count_image_and_packed_counts(oracle, rings, max_rd, n_proj, n_r, nsub, packed):
    """The same with the zero-count image's likelihood, counts and additive term
    packed to the subset, and the backprojection alone added to what bp holds."""
    ig = ImageGeom(27, 24, 2 * rings - 1, 2.5, 2.5, 2.0)
    sg = Sino3DGeom.span1(n_proj, n_r, rings, 45.0, rings * 4.0, 120.0, max_rd)
    rng = np.random.default_rng(rings + packed)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    sub = nsub - 1 if nsub > 1 else -1
    meas = ((rng.random(sg.n_bins) < 0.05) * (1 + rng.poisson(2.0, sg.n_bins))).astype(np.float32)
    add = (rng.random(sg.n_bins, dtype=np.float32) + 0.5).astype(np.float32)
    pick = lambda v: np.ascontiguousarray(v.reshape(sg.n_sinos, n_proj, n_r)[:, max(sub, 0)::nsub, :]).reshape(-1)
    m, est = pick(meas), (oracle.project_3d(sg, ig, x0, sub, nsub) + pick(add)).astype(np.float32)
    ratio = oracle.backproject_3d(sg, ig, oracle.inverse_divide(m, est), sub, nsub, threads=1)
    e64 = est.astype(np.float64)
    want_lik = float(np.sum(m * np.log(e64) - e64))
    P = ap.SiddonProjector(ig, sg)
    zeros = lambda: torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV)
    c, a = (t(m), t(pick(add))) if packed else (t(meas), t(add))
    zimg, zadd = zeros(), torch.zeros(1, dtype=torch.float64, device=DEV)
    P.zero_count_image(c, zimg, sub, nsub, add=a, zero_add=zadd, counts_packed=packed)
    x, lik = t(x0), torch.zeros(1, dtype=torch.float64, device=DEV)
    sens = np.ones(ig.n_voxels, np.float32)
    P.em_pass_sparse(c, x, zeros(), t(sens), zimg, sub, nsub, add=a, zero_add=zadd, counts_packed=packed, lik=lik)
    assert rel(x.cpu().numpy(), oracle.update(x0, ratio, sens, np.float32(0), True)) <= 1e-5
    assert abs(lik.item() - want_lik) <= 1e-6 * max(abs(want_lik), float(np.sum(e64)))
    bp = P.em_project_backproject(c, t(x0), t(x0), sub, nsub, add=a, counts_packed=packed, zimg=zimg, zero_add=zadd)
    assert rel(bp.cpu().numpy(), x0.astype(np.float64) + ratio) <= 1e-5


@pytest.mark.parametrize("first,n", [(0, 40), (8, 33), (20, 21), (0, 41)])
def test_shards_with_nearly_every_bin(oracle, first, n):
    """Shards whose LORs go to the queue whole, of a projector that would queue fewer bins a LOR itself."""
    ig = ImageGeom(27, 24, 41, 2.5, 2.5, 2.0)
    sg = Sino3DGeom.span1(100, 90, 41, 45.0, 82.0, 120.0, 0)
    rng = np.random.default_rng(n)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    est = oracle.project_3d(sg, ig, x0)
    meas = (1 + rng.poisson(2.0, sg.n_bins)).astype(np.float32).reshape(41, -1)
    inside = np.zeros_like(meas)
    inside[first:first + n] = meas[first:first + n]
    want = oracle.backproject_3d(sg, ig, oracle.inverse_divide(inside.reshape(-1), est), threads=1)
    P = ap.SiddonProjector(ig, sg)
    P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
    P.set_shard(first, n)
    zeros = lambda: torch.zeros(ig.n_voxels, dtype=torch.float32, device=DEV)
    G = P.backproject_ones(zeros())
    for _ in range(2):
        bp = P.em_project_backproject(t(meas.reshape(-1)), t(x0), zeros(), zimg=G)
        assert rel(bp.cpu().numpy(), want) <= 1e-5
