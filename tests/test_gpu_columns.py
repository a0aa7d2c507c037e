"""The column walk (csrc/columns.cuh) at the sizes where it can go wrong,
against the oracle: sinogram counts around a warp's 32 and a block's 256, odd
and even slices, z crossings closer than a batch of steps, an image much
shorter than the scanner, rays outside the image in x / y (the bounds-tested
walk), compressed sinograms.  Projection bit-identical; backprojections and
one fused pass rel L2 <= 1e-5 (fp32 atomics in another order), likelihoods to
1e-6 (listed: the rounding of the image dot product) and 1e-9."""
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


def zeros(n):
    return torch.zeros(n, dtype=torch.float32, device=DEV)


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    m = np.isfinite(a) & np.isfinite(b)
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    return float(np.linalg.norm(a[m] - b[m]) / max(np.linalg.norm(b[m]), 1e-300))


def bits_equal(a, b):
    return np.array_equal(np.ascontiguousarray(a, np.float32).view(np.uint32),
                          np.ascontiguousarray(b, np.float32).view(np.uint32))


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ap.load_library()


# image, sinogram (their passes and backprojections take the columns; the
# projections that do are in column_cases.py)
CASES = {
    "16 sinograms": (ImageGeom(96, 96, 31, 2.08, 2.08, 2.03), Sino3DGeom.span1(40, 90, 16, 99.84, 16 * 4.06, 200.0, 0)),
    "31 sinograms": (ImageGeom(64, 64, 21, 2.08, 2.08, 2.03), Sino3DGeom.span1(36, 80, 11, 66.56, 11 * 4.054, 200.0, 1)),
    "33 sinograms": (ImageGeom(64, 64, 66, 2.08, 2.08, 2.03), Sino3DGeom.span1(36, 80, 33, 66.56, 33 * 4.06, 200.0, 0)),
    "257 sinograms": (ImageGeom(24, 24, 514, 5.0, 5.0, 1.0), Sino3DGeom.span1(21, 41, 257, 60.0, 257 * 2.0, 200.0, 0)),
    "steep": (ImageGeom(48, 48, 160, 4.0, 4.0, 0.5), Sino3DGeom.span1(32, 60, 8, 96.0, 80.0, 150.0, 7)),
    "short image": (ImageGeom(64, 64, 5, 2.08, 2.08, 2.03), Sino3DGeom.span1(20, 60, 9, 66.56, 9 * 4.06, 150.0, 8)),
    "not square": (ImageGeom(64, 40, 9, 2.5, 3.1, 2.0), Sino3DGeom.span1(40, 90, 5, 80.0, 5 * 4.0, 150.0, 4)),
    "span 3": (ImageGeom(72, 72, 17, 2.0, 2.0, 2.0), Sino3DGeom.span(30, 72, 9, 72.0, 36.0, 150.0, 3, 8)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_against_oracle(oracle, name):
    ig, sg = CASES[name]
    rng = np.random.default_rng(len(name))
    img = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    P = ap.SiddonProjector(ig, sg)
    nsub = 3
    for sub, ns in ((-1, 1), (1, nsub)):
        want = oracle.project_3d(sg, ig, img, sub, ns)
        assert bits_equal(P.project(t(img), zeros(want.size), sub, ns).cpu().numpy(), want)
        v = rng.random(want.size, dtype=np.float32)
        v[rng.random(want.size) < 0.3] = 0.0
        e = rng.random(want.size, dtype=np.float32)
        e[rng.random(want.size) < 0.1] = 0.0
        assert rel(P.backproject(t(v), zeros(ig.n_voxels), sub, ns).cpu().numpy(),
                   oracle.backproject_3d(sg, ig, v, sub, ns)) <= 1e-5
        assert rel(P.divide_and_backproject(t(v), t(e), zeros(ig.n_voxels), sub, ns).cpu().numpy(),
                   oracle.divide_and_backproject_3d(sg, ig, v, e, sub, ns)) <= 1e-5
        a, b = P.backproject_and_ones(t(v), zeros(ig.n_voxels), zeros(ig.n_voxels), sub, ns)
        assert rel(a.cpu().numpy(), oracle.backproject_3d(sg, ig, v, sub, ns)) <= 1e-5
        assert rel(b.cpu().numpy(), oracle.backproject_3d(sg, ig, np.ones_like(v), sub, ns)) <= 1e-5
    s = 1
    est = oracle.project_3d(sg, ig, img, s, nsub)
    sens = (rng.random(ig.n_voxels, dtype=np.float32) + 1).astype(np.float32)
    G = P.backproject_ones(zeros(ig.n_voxels), s, nsub)
    P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
    # all bins with counts, most, and so few that a LOR has one or none
    for level, dtype in ((3.0, np.uint32), (0.05, np.uint16), (1e-4, np.float32)):
        meas = rng.poisson(oracle.project_3d(sg, ig, img) * level).astype(dtype)
        m_sub = meas.reshape(sg.n_sinos, sg.n_proj, sg.n_r)[:, s::nsub, :].reshape(-1).astype(np.float32)
        ratio = oracle.inverse_divide(m_sub, est)
        want_x = oracle.update(img, oracle.backproject_3d(sg, ig, ratio, s, nsub, threads=1), sens, np.float32(0), True)
        nz = est != 0
        e64 = est[nz].astype(np.float64)
        want_lik = float(np.sum(m_sub[nz] * np.log(e64) - e64))
        for listed in (False, True):
            x, lik = t(img), torch.zeros(1, dtype=torch.float64, device=DEV)
            if listed:
                P.em_pass_sparse(t(meas), x, zeros(ig.n_voxels), t(sens), G, s, nsub, lik=lik)
            else:
                P.em_pass(t(meas), x, zeros(ig.n_voxels), t(sens), s, nsub, lik=lik)
            assert rel(x.cpu().numpy(), want_x) <= 1e-5
            assert abs(lik.item() - want_lik) <= (1e-6 if listed else 1e-9) * abs(want_lik)


@pytest.mark.parametrize("n", [1016, 1024, 1160, 1230])
def test_widest_lists(oracle, n):
    """Images around the widest whose crossing list fits a block's shared
    memory (and wider: the padded pair): the listed pass and a projection."""
    ig, sg = ImageGeom(n, n, 2, 0.4, 0.4, 4.0), Sino3DGeom.span1(3, 200, 16, 0.2 * n, 16 * 0.5, 400.0, 0)
    rng = np.random.default_rng(n)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    est = oracle.project_3d(sg, ig, x0)
    P = ap.SiddonProjector(ig, sg)
    assert bits_equal(P.project(t(x0), zeros(est.size)).cpu().numpy(), est)
    P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
    meas = rng.poisson(est * 0.05).astype(np.float32)
    G = P.backproject_ones(zeros(ig.n_voxels))
    sens = np.ones(ig.n_voxels, np.float32)
    x = P.em_pass_sparse(t(meas), t(x0), zeros(ig.n_voxels), t(sens), G)
    bp = oracle.backproject_3d(sg, ig, oracle.inverse_divide(meas, est), threads=1)
    assert rel(x.cpu().numpy(), oracle.update(x0, bp, sens, np.float32(0), True)) <= 1e-5


def test_divide_at_the_ends_of_the_float_range(oracle):
    """Values and estimates whose ratio, or whose products with a segment,
    leave the float range: the same finite, infinite and NaN voxels as the
    reference's (seg * v) / e."""
    ig, sg = CASES["31 sinograms"]
    rng = np.random.default_rng(5)
    n = sg.n_bins
    v = rng.random(n, dtype=np.float32)
    e = (rng.random(n, dtype=np.float32) + 0.5).astype(np.float32)
    at = rng.choice(n, 60, replace=False)
    for k, (vv, ee) in enumerate([(1e-35, 1.0), (1e35, 1e3), (3.0, 1e-38), (2.0, np.inf), (1e-20, 1e20), (0.0, 1e-40)]):
        v[at[10 * k:10 * k + 10]] = vv
        e[at[10 * k:10 * k + 10]] = ee
    P = ap.SiddonProjector(ig, sg)
    got = P.divide_and_backproject(t(v), t(e), zeros(ig.n_voxels)).cpu().numpy()
    want = oracle.divide_and_backproject_3d(sg, ig, v, e, threads=1)
    assert rel(got, want) <= 1e-5


def test_project_on_streams_and_in_a_graph(oracle):
    """Projections of other images queued on three streams at once (two column
    slots), and one captured into a graph and replayed: all bit-identical."""
    ig, sg = CASES["31 sinograms"]
    rng = np.random.default_rng(8)
    imgs = [rng.random(ig.n_voxels, dtype=np.float32) for _ in range(6)]
    want = [oracle.project_3d(sg, ig, i) for i in imgs]
    P = ap.SiddonProjector(ig, sg)
    dev, outs = [t(i) for i in imgs], [zeros(sg.n_bins) for _ in imgs]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for k in range(6):
        P.project(dev[k], outs[k], stream=streams[k % 3])
    torch.cuda.synchronize()
    for k in range(6):
        assert bits_equal(outs[k].cpu().numpy(), want[k])
    out = zeros(sg.n_bins)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        P.project(dev[0], out)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert bits_equal(out.cpu().numpy(), want[0])


@pytest.mark.parametrize("rings,max_rd", [(1, 0), (15, 0), (17, 0), (5, 2)])
@pytest.mark.parametrize("ring", [70.0, 200.0])
def test_rays_past_the_image(oracle, rings, max_rd, ring):
    """Half of the radial bins past the image's corners and sides, angles along
    the axes and diagonals among them, from a near and a far ring: rays that
    miss the image record nothing, whichever walk serves them (one sinogram and
    15: bin by bin; 17 and 19: columns), and those that just touch it all their
    segments."""
    ig = ImageGeom(33, 33, 5, 2.0, 2.0, 4.0)
    sg = Sino3DGeom.span1(16, 131, rings, 66.0, rings * 4.0, ring, max_rd)
    rng = np.random.default_rng(rings)
    x0 = (rng.random(ig.n_voxels, dtype=np.float32) + 0.5).astype(np.float32)
    P = ap.SiddonProjector(ig, sg)
    est = oracle.project_3d(sg, ig, x0)
    assert (est.reshape(-1, 131)[:, [0, -1]] == 0).all()
    assert bits_equal(P.project(t(x0), zeros(est.size)).cpu().numpy(), est)
    v = rng.random(est.size, dtype=np.float32)
    want = oracle.backproject_3d(sg, ig, v, threads=1)
    assert rel(P.backproject(t(v), zeros(ig.n_voxels)).cpu().numpy(), want) <= 1e-5
    m = rng.poisson(3.0, est.size).astype(np.uint16)
    add = (rng.random(est.size, dtype=np.float32) + 0.5).astype(np.float32)
    bp = P.em_project_backproject(t(m), t(x0), zeros(ig.n_voxels), add=t(add))
    want = oracle.backproject_3d(sg, ig, oracle.inverse_divide(m.astype(np.float32), est + add), threads=1)
    assert rel(bp.cpu().numpy(), want) <= 1e-5
