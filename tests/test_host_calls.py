"""The calls that the library's host code makes, on a runtime without a GPU
(fake_gpu.py): what a projector writes is in place before a stream reads it."""
import os
import subprocess

import pytest

import fake_gpu


@pytest.fixture(scope="module")
def gpu(tmp_path_factory):
    so = fake_gpu.build(tmp_path_factory.mktemp("fake"))
    return lambda script: fake_gpu.run(so, script)


GEOMS = '''
G3 = (ImageGeom(32, 32, 21, 2.0, 2.0, 2.0), Sino3DGeom.span1(16, 40, 11, 33.0, 22.0, 100.0, 1))
G2 = (ImageGeom(32, 32, 1, 2.0, 2.0, 2.0), Sino2DGeom(16, 40, 33.0, 100.0))
'''


def waited(log):
    """The legacy stream was waited for after the last write on it."""
    writes = [i for i, l in enumerate(log) if l.split()[:2] in (["memset", "legacy"], ["memcpy", "legacy"])]
    waits = [i for i, l in enumerate(log) if l.split()[:2] == ["sync", "legacy"]]
    return bool(writes) and bool(waits) and waits[-1] > writes[-1]


@pytest.mark.parametrize("step", ["ap.SiddonProjector(*G3)", "ap.SiddonProjector(*G2)", "P.set_sampling(2, 2)",
                                  "P.set_alpha_precision(True)",
                                  "P.set_option(_lib.APIRL_OPT_ACCUMULATE, _lib.APIRL_ACC_COMPENSATED)"])
def test_tables_and_zeros_are_waited_for(gpu, step):
    """Non-blocking streams do not wait for the legacy stream, on which tables are copied and buffers cleared."""
    log = gpu(GEOMS + f"P = ap.SiddonProjector(*G3)\nfake.clear()\n{step}\ndone(fake.log())")
    assert waited(log), log


def test_second_pair_is_cleared_on_the_callers_stream(gpu):
    log = gpu(GEOMS + '''
P = ap.SiddonProjector(*G3)
fake.clear()
_lib.check(lib.apirl_backproject_and_ones(P.h, D, D, ctypes.c_void_p(1 << 42), -1, 1, S))
done(fake.log())''')
    assert any(l.startswith("memset 0x9990") for l in log)
    assert not any(l.split()[:2] == ["memset", "legacy"] for l in log), log


@pytest.mark.parametrize("nz", [1, 2])
def test_2d_passes_update_every_slice(gpu, nz):
    """The padded 2D layouts hold one slice; an image of several takes the pass that updates all its voxels."""
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom(32, 32, {nz}, 2.0, 2.0, 2.0), Sino2DGeom(16, 40, 33.0, 100.0))
fake.clear()
_lib.check(lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, None, S))
done(fake.launches())''')
    assert any("k_planar_update" in n for n in names) == (nz == 1)
    assert any("k_update" in n for n in names) == (nz == 2)


@pytest.mark.parametrize("ny", [65534 * 8, 65534 * 8 + 1, 65535 * 8 - 1])
def test_tall_2d_images_stay_within_the_grid(gpu, ny):
    """The update's grid has one row of blocks a tile row of 8 and one for the likelihood, 65535 at most."""
    log = gpu(f'''
P = ap.SiddonProjector(ImageGeom(4, {ny}, 1, 2.0, 2.0, 2.0), Sino2DGeom(3, 4, 33.0, 100.0))
fake.clear()
st = lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, D, S)
done([st] + fake.log())''')
    assert log[0] == 0 and not any(l.startswith("refused") for l in log[1:]), log


@pytest.mark.parametrize("nz", [65534 * 32, 65534 * 32 + 1])
def test_long_images_stay_within_the_grid(gpu, nz):
    """As above for the column layout's update, whose grid has a layer more than 32 slices each (images of
    more than 65535 slices that keep to the padded pair have no pass, and had none)."""
    log = gpu(f'''
P = ap.SiddonProjector(ImageGeom(8, 8, {nz}, 2.0, 2.0, 0.01), Sino3DGeom.span1(3, 4, 16, 16.0, 500.0, 100.0, 0))
fake.clear()
st = lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, D, S)
done([st] + fake.log())''')
    cols = any("k_em_cols" in l for l in log[1:])
    assert cols == (nz == 65534 * 32) and not any(l.startswith("refused") and "k_col" in l for l in log[1:]), log


ROOM = GEOMS + '''
G = Sino3DGeom.span1(64, 90, 20, 140.0, 40.0, 200.0, 1)   # enough bins for a projection on the columns
def em(P):
    fake.clear()
    _lib.check(lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, None, S))
    return [k for k in ("k_em_cols_rays", "k_em_cols", "k_em_pass_rays", "k_em_pass_persist", "k_planar_pass",
                        "k_em_pass") if any(k in n for n in fake.launches())][0]
def project(P):
    fake.clear()
    _lib.check(lib.apirl_project(P.h, D, D, -1, 1, S))
    return [k for k in ("k_project_cols", "k_project") if any(k in n for n in fake.launches())][0]
def under_limits(make, look):
    P = make(); full = fake.used(); seen = [look(P)]; P.close()
    for k in range(1, 60):
        fake.limit(full - full * k // 60)
        try:
            P = make()
        except _lib.ApirlError as e:
            state = ["oom" if e.code == _lib.APIRL_ERR_OOM else str(e)]
            assert fake.used() == 0
            lib.apirl_projector_num_bins(None, 0, 1)
            _g.cudaGetLastError()
        else:
            state = look(P)
            P.close()
        assert fake.used() == 0
        if state != seen[-1]: seen.append(state)
    return seen
'''


def test_projectors_without_room_for_the_columns(gpu):
    """Creation takes what fits: all column images, those of the passes, none; each serves every call."""
    seen = gpu(ROOM + '''
done(under_limits(lambda: ap.SiddonProjector(ImageGeom(64, 64, 39, 2.0, 2.0, 1.0), G), lambda P: [em(P), project(P)]))''')
    assert seen == [["k_em_cols", "k_project_cols"], ["k_em_cols", "k_project"], ["k_em_pass_persist", "k_project"], ["oom"]]


def test_sampled_projectors_without_room_for_the_columns(gpu):
    """set_sampling makes its tables first: what fitted without a column layout still does."""
    seen = gpu(ROOM + '''
def make():
    P = ap.SiddonProjector(ImageGeom(64, 64, 39, 2.0, 2.0, 1.0), G)
    try:
        P.set_sampling(4, 4)
    except Exception:
        P.close()
        raise
    return P
done(under_limits(make, lambda P: [em(P)]))''')
    assert [s[0] for s in seen if s[0] != "oom"][0] == "k_em_cols_rays"
    assert ["k_em_pass_rays"] in seen and seen[-1] == ["oom"]


def test_2d_projectors_without_room_for_the_padded_layouts(gpu):
    seen = gpu(ROOM + '''
done(under_limits(lambda: ap.SiddonProjector(ImageGeom(256, 256, 1, 2.0, 2.0, 1.0), Sino2DGeom(16, 40, 256.0, 400.0)),
                  lambda P: [em(P)]))''')
    assert seen == [["k_planar_pass"], ["k_em_pass"], ["oom"]]


@pytest.mark.parametrize("iters", [1, 4])
def test_reconstructions_without_room_for_the_columns(gpu, iters):
    """A whole reconstruction whose buffers do not fit beside the columns runs on the padded pair."""
    seen = gpu(ROOM + f'''
ig, sg = ImageGeom(64, 64, 39, 2.0, 2.0, 1.0), G
m, x = np.ones(sg.n_bins, np.float32), np.ones(ig.n_voxels, np.float32)
a = np.full(sg.n_bins, 0.5, np.float32)
peak = 1 << 40
def run(limit):
    fake.limit(limit); fake.clear()
    try:
        ap.osem_3d(ig, sg, m, x, {iters}, 4, add=a)
    except _lib.ApirlError as e:
        _g.cudaGetLastError()
        return "oom" if e.code == _lib.APIRL_ERR_OOM else str(e)
    finally:
        assert fake.used() == 0
    return "cols" if any("k_em_cols" in n for n in fake.launches()) else "pair"
# device bytes by bisection: the least room the run takes on the columns, on the pair
def least(ok):
    lo, hi = 0, 1 << 32
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if run(mid) in ok else (mid, hi)
    return hi
cols, pair = least(["cols"]), least(["cols", "pair"])
done([run(1 << 40), cols, pair, run(cols - 2048), run(pair - 2048)])''')
    assert seen[0] == "cols" and seen[3:] == ["pair", "oom"]
    # the difference is the three column images (and the queue), no more
    assert seen[1] > seen[2]


def test_2d_reconstructions_keep_no_layouts_they_do_not_walk(gpu):
    log = gpu('''
ig, sg = ImageGeom(128, 128, 1, 2.0, 2.0, 1.0), Sino2DGeom(16, 40, 128.0, 400.0)
ap.mlem_2d(ig, sg, np.ones(sg.n_bins, np.float32), np.ones(ig.n_voxels, np.float32), 2)
done(fake.log())''')
    assert not any("k_planar" in l for l in log)
    assert not any(l == f"malloc legacy {6 * 132 * 132 * 4}" for l in log) and "memset legacy " not in log, log


def test_creation_takes_one_block(gpu):
    """A fresh device mapping costs more than all else in creation: one for a projector, one for its sampled rays."""
    counts = gpu(GEOMS + '''
n = []
def mallocs(make):
    fake.clear()
    P = make()
    n.append(sum(l.startswith("malloc") for l in fake.log()))
    return P
P = mallocs(lambda: ap.SiddonProjector(*G3)); mallocs(lambda: P.set_sampling(2, 2)); mallocs(lambda: ap.SiddonProjector(*G2))
done(n)''')
    assert counts == [1, 1, 1]


@pytest.mark.parametrize("rings,max_rd,n_proj,want", [(16, 0, 100, "k_em_cols_direct"), (33, 4, 100, "k_em_cols_direct"),
                                                      (33, 4, 40, "k_em_cols_few"), (16, 0, 40, ""), (46, 45, 100, "")])
def test_listed_passes_defer_lors_with_few_counts(gpu, rings, max_rd, n_proj, want):
    """Where a LOR's crossings are listed for few rays, the pass leaves them to a second kernel."""
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom(27, 24, 31, 2.5, 2.5, 2.0), Sino3DGeom.span1({n_proj}, 90, {rings}, 45.0, 64.0, 120.0, {max_rd}))
P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
fake.clear()
_lib.check(lib.apirl_em_pass_sparse(P.h, D, 0, 0, None, D, D, D, D, None, None, 0.0, 0, -1, 1, None, S))
done(fake.launches())''')
    assert any("k_em_cols_listed" in n for n in names)
    second = [k for k in ("k_em_cols_direct", "k_em_cols_few") if any(k in n for n in names)]
    assert second == ([want] if want else [])


def test_batched_jobs_with_few_counts_take_lists(gpu):
    """A block a LOR pays from some tens of counts in it on: jobs with fewer (here none) walk lists of their bins."""
    names = gpu('''
from apirl_b200.batch import Batch, Job
ig, sg = ImageGeom(128, 128, 31, 2.0, 2.0, 2.0), Sino3DGeom.span1(160, 160, 16, 160.0, 64.0, 443.0, 0)
b = Batch(0, 8 << 30)
b.run_all([Job(ig, sg, np.zeros(sg.n_bins, np.uint16), 10, 8)])
done(sorted(set(fake.launches())))''')
    assert any("k_lor_counts" in n for n in names) and any("k_nz_write" in n for n in names)
    assert not any("k_em_multi_cols" in n for n in names)


@pytest.mark.parametrize("n,nsub,cols", [(32, 8, False), (32, 1, True), (64, 8, True)])
def test_small_divisions_take_one_launch(gpu, n, nsub, cols):
    nr = int(1.3 * n + 0.5)
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom({n}, {n}, 33, 2.0, 2.0, 2.0), Sino3DGeom.span1({nr}, {nr}, 17, {nr}.0, 68.0, 443.0, 0))
fake.clear()
_lib.check(lib.apirl_divide_and_backproject(P.h, D, D, D, 0, {nsub}, S))
done(fake.launches())''')
    assert any("k_scatter_cols" in x for x in names) == cols and any("k_backproject3" in x for x in names) != cols


@pytest.mark.parametrize("rings,ns,nsub,cols", [(16, 12, 1, False), (16, 12, 8, True), (40, 12, 1, True), (16, 3, 1, True)])
def test_sampled_passes_with_few_rays_in_flight_walk_bin_by_bin(gpu, rings, ns, nsub, cols):
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom(64, 64, 31, 2.0, 2.0, 2.0), Sino3DGeom.span1(83, 83, {rings}, 83.0, 64.0, 443.0, 0))
P.set_sampling({ns}, 1)
fake.clear()
for bp in (0, 1):
    if bp: _lib.check(lib.apirl_em_project_backproject(P.h, D, 0, 0, None, D, D, 0, {nsub}, None, S))
    else: _lib.check(lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, 0, {nsub}, D, S))
done(fake.launches())''')
    assert sum("k_em_cols_rays" in n for n in names) == (2 if cols else 0)
    assert sum("k_em_pass_rays" in n for n in names) == (0 if cols else 2)
    assert any("k_col_" in n for n in names) == cols


@pytest.mark.parametrize("n,rings,cols", [(320, 16, False), (320, 24, True), (256, 18, False), (128, 16, True)])
def test_full_passes_of_few_sinograms_on_wide_images_take_the_pair(gpu, n, rings, cols):
    names = gpu(f'''
P = ap.SiddonProjector(ImageGeom({n}, {n}, 31, 2.0, 2.0, 2.0), Sino3DGeom.span1(20, 83, {rings}, {n}.0, 64.0, 900.0, 0))
P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
fake.clear()
_lib.check(lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, -1, 1, D, S))
full = fake.launches()
fake.clear()
_lib.check(lib.apirl_em_pass_sparse(P.h, D, 0, 0, None, D, D, D, D, None, None, 0.0, 0, -1, 1, D, S))
done([full, fake.launches()])''')
    assert any("k_em_cols" in x for x in names[0]) == cols and any("k_em_pass_persist" in x for x in names[0]) != cols
    assert any("k_col_" in x for x in names[0]) == cols
    assert any("k_em_cols_listed" in x for x in names[1])


def test_autotuner_reports_the_shape_in_force_where_there_is_one(gpu):
    """Passes on the columns ignore block size and gather segments: neither is chosen from the noise of equal passes."""
    got = gpu(GEOMS + '''
G = Sino3DGeom.span1(16, 40, 11, 33.0, 22.0, 100.0, 0)   # 11 sinograms: the padded pair
out = []
for sg in (G3[1], G):
    P = ap.SiddonProjector(G3[0], sg)
    P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
    for z in (D, None):
        fake.clear()
        tune, block = _lib.TuneC(), ctypes.c_int()
        _lib.check(lib.apirl_projector_autotune_ex(P.h, D, 0, D, z, -1, 1, 2, ctypes.byref(tune), S))
        passes = sum("k_em" in n for n in fake.launches())
        fake.clear()
        _lib.check(lib.apirl_projector_autotune(P.h, D, 0, D, -1, 1, 2, ctypes.byref(block), S))
        out.append([tune.block, tune.unroll, passes, block.value, sum("k_em" in n for n in fake.launches())])
done(out)''')
    assert got[:2] == [[128, 6, 3, 128, 0], [128, 4, 3, 128, 0]]
    assert got[2][2] == got[3][2] == 45 and got[2][4] == got[3][4] == 15


def test_projections_of_the_column_cases_take_the_columns(gpu):
    got = gpu(f'''
sys.path.insert(0, {fake_gpu.HERE!r})
from column_cases import PROJECTED
out = {{}}
for name, (ig, sg, sub, nsub) in PROJECTED.items():
    P = ap.SiddonProjector(ig, sg)
    fake.clear()
    _lib.check(lib.apirl_project(P.h, D, D, -1, 1, S))
    _lib.check(lib.apirl_project(P.h, D, D, sub, nsub, S))
    out[name] = sum("k_project_cols" in n for n in fake.launches())
done(out)''')
    assert got and all(n == 2 for n in got.values()), got


def _few_on_wide(n, rings, max_rd, nsub, call):
    nr = int(1.3 * n + 0.5)
    return f'''
P = ap.SiddonProjector(ImageGeom({n}, {n}, 9, 2.0, 2.0, 2.0), Sino3DGeom.span1({nr}, {nr}, {rings}, {nr}.0, 20.0, 443.0, {max_rd}))
fake.clear()
_lib.check({call.format(sub=0 if nsub > 1 else -1, nsub=nsub)})
done(fake.launches())'''


@pytest.mark.parametrize("n,rings,max_rd,nsub,cols", [(256, 16, 0, 1, False), (230, 5, 2, 1, False), (256, 24, 0, 1, True),
                                                      (128, 18, 0, 1, True), (256, 40, 0, 4, True)])
def test_projections_of_few_sinograms_on_wide_images(gpu, n, rings, max_rd, nsub, cols):
    names = gpu(_few_on_wide(n, rings, max_rd, nsub, "lib.apirl_project(P.h, D, D, {sub}, {nsub}, S)"))
    assert any("k_project_cols" in x for x in names) == cols


@pytest.mark.parametrize("n,rings,max_rd,nsub,cols", [(230, 5, 2, 1, False), (230, 5, 2, 8, True), (256, 28, 0, 1, True)])
def test_long_full_passes_of_few_sinograms(gpu, n, rings, max_rd, nsub, cols):
    names = gpu(_few_on_wide(n, rings, max_rd, nsub,
                             "lib.apirl_em_pass(P.h, D, 0, 0, None, D, D, D, None, 0.0, 0, {sub}, {nsub}, D, S)"))
    assert any("k_em_cols" in x for x in names) == cols


@pytest.mark.parametrize("n,rings,n_proj,n_r,want", [(200, 16, 116, 230, True), (200, 257, 116, 230, False), (64, 16, 116, 230, False)])
def test_long_backprojections_queue_lors_with_few_values(gpu, n, rings, n_proj, n_r, want):
    log = gpu(f'''
P = ap.SiddonProjector(ImageGeom({n}, 190, 5, 2.0, 2.0, 2.0), Sino3DGeom.span1({n_proj}, {n_r}, {rings}, 230.0, 11.0, 400.0, 0))
fake.clear()
_lib.check(lib.apirl_backproject(P.h, D, D, -1, 1, S))
done(fake.log())''')
    assert any("k_scatter_cols_direct" in l for l in log) == want
    assert any(l.startswith("memset 0x9990") for l in log) == want  # the queue is emptied on the caller's stream


def test_queue_has_room_for_every_shard(tmp_path):
    exe = str(tmp_path / "queue_room_check")
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include", "-I" + os.path.join(fake_gpu.ROOT, "apirl_b200", "csrc"),
                    os.path.join(fake_gpu.HERE, "queue_room_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_queue_is_sized_by_its_room(gpu):
    """41 sinograms over 9000 LORs: 40 bins a LOR (a shard of 40), 4 bytes each, beyond what 8000 LORs' block has."""
    sizes = gpu('''
out = []
for n_proj in (80, 100):    # 7200 and 9000 LORs: without and with the queue of bins
    fake.clear()
    P = ap.SiddonProjector(ImageGeom(27, 24, 31, 2.5, 2.5, 2.0), Sino3DGeom.span1(n_proj, 90, 41, 45.0, 64.0, 120.0, 0))
    out.append([int(l.split()[2]) for l in fake.log() if l.startswith("malloc")][0])
done(out)''')
    assert sizes[1] - sizes[0] >= 9000 * 40 * 4
